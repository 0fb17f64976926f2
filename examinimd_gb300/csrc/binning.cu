// BinningKKSort on the device (binning_kksort.cpp:71-140).
//
// Bin of a particle: per-dimension int((x_d - min_d) * nbin_d/(max_d - min_d)),
// flattened with x slowest (the decode of binning_kksort.cpp:61-63).  The
// permutation is a stable counting sort: each bin lists its particles in
// ascending index, which is what a serial BinSort produces.  Four kernels:
// bin + histogram (whose counts number a bin's members), scan, scatter, and a
// per-bin rank pass that restores ascending order inside each bin.  With sort=true
// a gather reorders x, v, f, type, id, q of the binned range.
#include <algorithm>
#include <cmath>

#include "emd_device.cuh"
#include "emd_internal.h"

namespace emd {
namespace {

// Bin centre coordinates, min_d + (i + 0.5) w_d for every bin index i of
// each dimension (nbx | nby | nbz entries): the per-particle FP32 offsets and
// the mixed form's FP64 centres both read them, so neither repeats the
// conversion, multiply and adds per particle on the FP64 pipe.
__global__ void k_bin_ctab(int nbx, int nby, int nbz, double minx, double miny, double minz, double wx, double wy,
                           double wz, double* __restrict__ tab) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < nbx) tab[t] = minx + (t + 0.5) * wx;
  else if (t < nbx + nby) tab[t] = miny + (t - nbx + 0.5) * wy;
  else if (t < nbx + nby + nbz) tab[t] = minz + (t - nbx - nby + 0.5) * wz;
}

struct BinGrid {
  int nbx, nby, nbz;
  double minx, miny, minz, mulx, muly, mulz;
  const double* ctab;
  float min32[3], mul32[3], off32[3];  // off32: 2 |min| mul + 2
};

// int((x - min) mul) as the reference rounds it (binning_kksort.cpp:61-63), in FP64 only
// where FP32 leaves it open: t is within 3e-7 (|t| + 2 |min| mul) of the FP64 value, so
// away from integers by more than three times that both truncate alike.  Nine FP64
// instructions a particle less (4.4 million: 0.127 -> 0.066 ms).
__device__ __noinline__ int bin_fp64(double x, double min, double mul) { return int((x - min) * mul); }
__device__ __forceinline__ int bin_of(const BinGrid& G, int d, double x, double min, double mul) {
  const float t = (f32_bits(x) - G.min32[d]) * G.mul32[d];
  const float b = floorf(t), r = t - b, e = 1e-6f * (t + G.off32[d]);
  return t > e && t < 1e6f && r > e && r < 1.f - e ? int(b) : bin_fp64(x, min, mul);
}

// bin of a particle, and its FP32 position relative to the bin's centre, for the
// neighbour candidate tests
__device__ __forceinline__ int bin_particle(const BinGrid& G, const double4_32a& p, float4* xl, unsigned* status) {
  int ix = bin_of(G, 0, p.x, G.minx, G.mulx);
  int iy = bin_of(G, 1, p.y, G.miny, G.muly);
  int iz = bin_of(G, 2, p.z, G.minz, G.mulz);
  if (ix < 0 || ix >= G.nbx || iy < 0 || iy >= G.nby || iz < 0 || iz >= G.nbz) {
    // outside the binned box: the reference would index out of bounds; keep
    // the particle in the nearest bin and report it
    latch_status(status, ST_BOUNDS);
    ix = min(max(ix, 0), G.nbx - 1);
    iy = min(max(iy, 0), G.nby - 1);
    iz = min(max(iz, 0), G.nbz - 1);
  }
  *xl = make_float4(float(p.x - G.ctab[ix]), float(p.y - G.ctab[G.nbx + iy]),
                    float(p.z - G.ctab[G.nbx + G.nby + iz]), __int_as_float(int(f32_bits(p.w))));
  return (ix * G.nby + iy) * G.nbz + iz;
}

__global__ void __launch_bounds__(256) k_bin_index(BinGrid G, const double4_32a* __restrict__ x4, int first, int n,
                                                   int* __restrict__ binof, int* __restrict__ slot,
                                                   int* __restrict__ bincount, float4* __restrict__ xl,
                                                   unsigned* status) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= n) return;
  const int b = bin_particle(G, x4[first + r], xl + first + r, status);
  binof[r] = b;
  slot[r] = atomicAdd(&bincount[b], 1);
}

__global__ void __launch_bounds__(256) k_bin_scatter(const int* __restrict__ binof, int n,
                                                     const int* __restrict__ binoffsets,
                                                     const int* __restrict__ slot, int* __restrict__ perm_tmp) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= n) return;
  perm_tmp[binoffsets[binof[r]] + slot[r]] = r;
}

// One warp per bin: each member's rank = number of members with a smaller
// index, which puts the bin in ascending order (members are distinct).
__global__ void __launch_bounds__(256) k_bin_rank(const int* __restrict__ bincount,
                                                  const int* __restrict__ binoffsets, int nbins,
                                                  const int* __restrict__ perm_tmp, int* __restrict__ permute) {
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (warp >= nbins) return;
  const int n = bincount[warp];
  const int off = binoffsets[warp];
  for (int e = lane; e < n; e += 32) {
    const int val = perm_tmp[off + e];
    int rank = 0;
    for (int k = 0; k < n; ++k) rank += perm_tmp[off + k] < val ? 1 : 0;
    permute[off + rank] = val;
  }
}

// The whole binning of a small system by one CTA: its passes take less than the
// launches (64 atoms: five operations, 27 us, 9 in one; 864 atoms, then with their
// 2,200 ghosts: 28 and 19).
constexpr int BIN_SMALL = 4096, BIN_SMALL_BINS = 2048, BIN_SMALL_THREADS = 1024;
__global__ void __launch_bounds__(BIN_SMALL_THREADS) k_bin_small(BinGrid G, const double4_32a* __restrict__ x4,
                                                                 int first, int n, int* __restrict__ binof,
                                                                 int* __restrict__ bincount,
                                                                 int* __restrict__ binoffsets, int* perm_tmp,
                                                                 int* __restrict__ permute,
                                                                 float4* __restrict__ xl, unsigned* status) {
  constexpr int PER = BIN_SMALL / BIN_SMALL_THREADS;
  __shared__ int cnt[BIN_SMALL_BINS], off[BIN_SMALL_BINS];
  __shared__ int wsum[32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nbins = G.nbx * G.nby * G.nbz;
  cnt[tid] = cnt[tid + BIN_SMALL_THREADS] = 0;
  __syncthreads();
  int bin[PER], slot[PER];
#pragma unroll
  for (int k = 0; k < PER; ++k) {
    const int r = tid + k * BIN_SMALL_THREADS;
    if (r >= n) continue;
    bin[k] = bin_particle(G, x4[first + r], xl + first + r, status);
    binof[r] = bin[k];
    slot[k] = atomicAdd(&cnt[bin[k]], 1);
  }
  __syncthreads();
  const int c0 = cnt[2 * tid], c1 = cnt[2 * tid + 1];
  int x = c0 + c1;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(FULL_MASK, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) wsum[warp] = x;
  __syncthreads();
  int base = x - c0 - c1;
  for (int k = 0; k < warp; ++k) base += wsum[k];
  off[2 * tid] = base;
  off[2 * tid + 1] = base + c0;
  __syncthreads();
  for (int b = tid; b < nbins; b += BIN_SMALL_THREADS) {
    bincount[b] = cnt[b];
    binoffsets[b] = off[b];
  }
#pragma unroll
  for (int k = 0; k < PER; ++k) {
    const int r = tid + k * BIN_SMALL_THREADS;
    if (r < n) perm_tmp[off[bin[k]] + slot[k]] = r;
  }
  __syncthreads();
  // each particle's rank in its bin: members with a smaller index
#pragma unroll
  for (int k = 0; k < PER; ++k) {
    const int r = tid + k * BIN_SMALL_THREADS;
    if (r >= n) continue;
    const int o = off[bin[k]], m = cnt[bin[k]];
    int rank = 0;
    for (int e = 0; e < m; ++e) rank += perm_tmp[o + e] < r ? 1 : 0;
    permute[o + rank] = r;
  }
}

// BinSort::sort of every particle field at once: dst(r) = src(perm(r))
__global__ void __launch_bounds__(256) k_sort_gather(const int* __restrict__ perm, int n,
                                                     const double4_32a* __restrict__ x4, const double* __restrict__ v,
                                                     const double* __restrict__ f, const double* __restrict__ q,
                                                     const int* __restrict__ type, const int* __restrict__ id,
                                                     double4_32a* __restrict__ ox4, double* __restrict__ ov,
                                                     double* __restrict__ of, double* __restrict__ oq,
                                                     int* __restrict__ otype, int* __restrict__ oid) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= n) return;
  const int s = perm[r];
  ox4[r] = x4[s];
  for (int d = 0; d < 3; ++d) {
    ov[3 * r + d] = v[3 * s + d];
    of[3 * r + d] = f[3 * s + d];
  }
  oq[r] = q[s];
  otype[r] = type[s];
  oid[r] = id[s];
}

// the sorted fields back in place, in one launch
__global__ void __launch_bounds__(256) k_sort_copy(int n, const double4_32a* __restrict__ x4,
                                                   const double* __restrict__ d, const int* __restrict__ t,
                                                   double4_32a* __restrict__ ox4, double* __restrict__ ov,
                                                   double* __restrict__ of, double* __restrict__ oq,
                                                   int* __restrict__ otype, int* __restrict__ oid) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= n) return;
  ox4[r] = x4[r];
  const size_t m = size_t(n);
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const size_t e = r + k * m;
    ov[e] = d[e];
    of[e] = d[3 * m + e];
  }
  oq[r] = d[6 * m + r];
  otype[r] = t[r];
  oid[r] = t[m + r];
}

}  // namespace
}  // namespace emd

using namespace emd;

extern "C" {

emd_status emd_binning_create(emd_ctx* ctx, double dx_in, double dy_in, double dz_in, int halo_depth, int do_local,
                              int do_ghost, int sort, int nbin_out[3]) {
  EMD_API_BEGIN
  require(dx_in > 0 && dy_in > 0 && dz_in > 0 && halo_depth >= 0, EMD_ERR_ARG, "emd_binning_create: bad bin size");
  if (!(do_local || do_ghost)) return EMD_OK;
  const int first = do_local ? 0 : c.N_local;
  const int last = do_ghost ? c.N_local + c.N_ghost : c.N_local;
  const int n = last - first;
  // host-side geometry, same expressions and order as binning_kksort.cpp:76-99
  const double sub[3] = {c.sub_hi[0] - c.sub_lo[0], c.sub_hi[1] - c.sub_lo[1], c.sub_hi[2] - c.sub_lo[2]};
  int nb[3] = {int(sub[0] / dx_in), int(sub[1] / dy_in), int(sub[2] / dz_in)};
  for (int d = 0; d < 3; ++d)
    if (nb[d] == 0) nb[d] = 1;
  const double dxyz[3] = {sub[0] / nb[0], sub[1] / nb[1], sub[2] / nb[2]};
  for (int d = 0; d < 3; ++d) nb[d] += 2 * halo_depth;
  const double eps = dxyz[0] / 1000;
  for (int d = 0; d < 3; ++d) {
    c.bmin[d] = -dxyz[d] * halo_depth - eps + c.sub_lo[d];
    c.bmax[d] = dxyz[d] * halo_depth + eps + c.sub_hi[d];
    c.bmul[d] = double(nb[d]) / (c.bmax[d] - c.bmin[d]);
    c.nbin[d] = nb[d];
  }
  c.nhalo = halo_depth;
  c.bin_first = first;
  c.bin_count_n = n;
  const long long nbins_ll = (long long)nb[0] * nb[1] * nb[2];
  require(nbins_ll < 0x7fffffffLL, EMD_ERR_ARG, "emd_binning_create: too many bins");
  const int nbins = int(nbins_ll);
  c.bincount.reserve(size_t(nbins) + 1, c.stream);
  c.binoffsets.reserve(size_t(nbins) + 1, c.stream);
  c.binof.reserve(size_t(n) + 1, c.stream);
  c.permute.reserve(size_t(n) + 1, c.stream);
  c.perm_tmp.reserve(size_t(n) + 1, c.stream);
  c.bin_slot.reserve(size_t(n) + 1, c.stream);
  c.xl_bin.reserve(size_t(first + n) + 1, c.stream, true);
  const int ntab = nb[0] + nb[1] + nb[2];
  // a box binned as before keeps its table
  const double key[9] = {double(nb[0]), double(nb[1]), double(nb[2]), c.bmin[0], c.bmin[1],
                         c.bmin[2],     c.bmax[0],     c.bmax[1],     c.bmax[2]};
  if (size_t(ntab) > c.bin_ctab.cap || !std::equal(key, key + 9, c.bin_ctab_key)) {
    c.bin_ctab_key[0] = 0;  // no box's, should the launch fail
    c.bin_ctab.reserve(size_t(ntab), c.stream);
    TimedLaunch t(c, "bin_ctab");
    k_bin_ctab<<<blocks_for(ntab, 256), 256, 0, c.stream>>>(
        nb[0], nb[1], nb[2], c.bmin[0], c.bmin[1], c.bmin[2], (c.bmax[0] - c.bmin[0]) / nb[0],
        (c.bmax[1] - c.bmin[1]) / nb[1], (c.bmax[2] - c.bmin[2]) / nb[2], c.bin_ctab.p);
    EMD_CHECK_LAUNCH();
    std::copy(key, key + 9, c.bin_ctab_key);
  }
  BinGrid G{nb[0], nb[1], nb[2], c.bmin[0], c.bmin[1], c.bmin[2], c.bmul[0], c.bmul[1], c.bmul[2], c.bin_ctab.p, {}, {}, {}};
  for (int d = 0; d < 3; ++d) {
    G.min32[d] = float(c.bmin[d]);
    G.mul32[d] = float(c.bmul[d]);
    G.off32[d] = float(2.0 * std::fabs(c.bmin[d]) * c.bmul[d] + 2.0);
  }
  c.xl_bin_valid = true;
  c.bin_sorted = false;
  if (n > 0 && n <= BIN_SMALL && nbins <= BIN_SMALL_BINS) {
    TimedLaunch t(c, "bin_small");
    k_bin_small<<<1, BIN_SMALL_THREADS, 0, c.stream>>>(G, c.x4.p, first, n, c.binof.p, c.bincount.p, c.binoffsets.p,
                                                       c.perm_tmp.p, c.permute.p, c.xl_bin.p, c.d_status);
    EMD_CHECK_LAUNCH();
  } else {
    EMD_CUDA(cudaMemsetAsync(c.bincount.p, 0, sizeof(int) * nbins, c.stream));
    if (n > 0) {
      TimedLaunch t(c, "bin_index");
      k_bin_index<<<blocks_for(n, 256), 256, 0, c.stream>>>(G, c.x4.p, first, n, c.binof.p, c.bin_slot.p,
                                                            c.bincount.p, c.xl_bin.p, c.d_status);
      EMD_CHECK_LAUNCH();
    }
    exclusive_scan_int(c, c.bincount.p, c.binoffsets.p, nbins);
    if (n > 0) {
      {
        TimedLaunch t(c, "bin_scatter");
        k_bin_scatter<<<blocks_for(n, 256), 256, 0, c.stream>>>(c.binof.p, n, c.binoffsets.p, c.bin_slot.p,
                                                                c.perm_tmp.p);
        EMD_CHECK_LAUNCH();
      }
      TimedLaunch t(c, "bin_rank");
      k_bin_rank<<<blocks_for((long long)nbins * 32, 256), 256, 0, c.stream>>>(c.bincount.p, c.binoffsets.p, nbins,
                                                                               c.perm_tmp.p, c.permute.p);
      EMD_CHECK_LAUNCH();
    }
  }
  if (sort && n > 0) {
    c.x_version++;
    // BinSort::sort of x, v, f, type, id, q over the binned range: one
    // fused gather kernel into staging buffers, then one copy back
    materialize_zero(c, true, false);
    c.xl_ok = 0;
    const int* perm = c.permute.p;
    c.stage_x4.reserve(size_t(n), c.stream);
    c.stage_d.reserve(7 * size_t(n), c.stream);
    c.stage_i.reserve(2 * size_t(n), c.stream);
    {
      TimedLaunch t(c, "bin_sort_gather");
      k_sort_gather<<<blocks_for(n, 256), 256, 0, c.stream>>>(
          perm, n, c.x4.p + first, c.v.p + 3 * size_t(first), c.f.p + 3 * size_t(first), c.q.p + first,
          c.type.p + first, c.id.p + first, c.stage_x4.p, c.stage_d.p, c.stage_d.p + 3 * size_t(n),
          c.stage_d.p + 6 * size_t(n), c.stage_i.p, c.stage_i.p + n);
      EMD_CHECK_LAUNCH();
    }
    {
      TimedLaunch t(c, "bin_sort_copy");
      k_sort_copy<<<blocks_for(n, 256), 256, 0, c.stream>>>(n, c.stage_x4.p, c.stage_d.p, c.stage_i.p, c.x4.p + first,
                                                            c.v.p + 3 * size_t(first), c.f.p + 3 * size_t(first),
                                                            c.q.p + first, c.type.p + first, c.id.p + first);
      EMD_CHECK_LAUNCH();
    }
    c.neigh_ready = false;
    // the bin indices, FP32 offsets and permutation of this binning refer to
    // the order before the sort: no neighbour list is built from it
    c.bin_sorted = true;
    c.xl_bin_valid = false;
  }
  c.binning_ready = true;
  if (nbin_out)
    for (int d = 0; d < 3; ++d) nbin_out[d] = nb[d];
  EMD_API_END
}

emd_status emd_binning_get(emd_ctx* ctx, int* bincount, int* binoffsets, int* permute, double bounds[6]) {
  EMD_API_BEGIN
  require(c.binning_ready, EMD_ERR_STATE, "emd_binning_get: no binning");
  const size_t nbins = size_t(c.nbin[0]) * c.nbin[1] * c.nbin[2];
  if (bincount) EMD_CUDA(cudaMemcpyAsync(bincount, c.bincount.p, sizeof(int) * nbins, cudaMemcpyDeviceToHost, c.stream));
  if (binoffsets)
    EMD_CUDA(cudaMemcpyAsync(binoffsets, c.binoffsets.p, sizeof(int) * nbins, cudaMemcpyDeviceToHost, c.stream));
  if (permute && c.bin_count_n > 0)
    EMD_CUDA(cudaMemcpyAsync(permute, c.permute.p, sizeof(int) * c.bin_count_n, cudaMemcpyDeviceToHost, c.stream));
  if (bounds)
    for (int d = 0; d < 3; ++d) {
      bounds[2 * d] = c.bmin[d];
      bounds[2 * d + 1] = c.bmax[d];
    }
  // the bounds are host values: no wait unless a device array was copied
  if (bincount || binoffsets || permute) EMD_CUDA(cudaStreamSynchronize(c.stream));
  EMD_API_END
}

}  // extern "C"
