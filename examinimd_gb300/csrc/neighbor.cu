// NeighborCSR / Neighbor2D on the device (neighbor_csr.h:176-435,
// neighbor_2d.h:175-331).
//
// One warp per interior bin (rows_of_bin, neigh_bin.cuh).
//
// One pass writes rows column-major in 16-byte granules (neigh_rows.cuh:
// the LayoutLeft of the reference's Neighbor2D view on a GPU, four entries
// per granule) with capacity K; the host grows K like
// Neighbor2D's regrow loop (x1.2) when a row overflows.
// NeighborCSR rows are compacted behind an exclusive scan of the counts when
// they are read (emd_neigh_get): the force kernels take column-major rows as fast
// (905,728 atoms: 2.66 ms either way), and compacting them took 0.54 ms a build.  Rows built for the mixed-precision force carry packed entries
// (j << 6) | (kx << 4) | (ky << 2) | kz with k = (bin_j - bin_i) + 1 per
// dimension, which the force kernel uses to difference FP32 bin-relative
// coordinates; the FP64 drop-in stores plain j.
#include <algorithm>

#include "emd_device.cuh"
#include "emd_internal.h"
#include "neigh_bin.cuh"

namespace emd {
namespace {

constexpr int NB_WARPS = 4;     // warps per CTA, one interior bin each (independent)
constexpr int NB_THREADS = 32 * NB_WARPS;
constexpr int NB_SLOTS = 64;  // spread slots for the longest-row reduction
static_assert(1 + NB_SLOTS <= kHostInts, "read-back of the row-length slots exceeds the pinned scratch");

struct NeighArgs {
  RowArgs r;
  const int* bincount;
  const int* binoffsets;
  int nbx, nhalo;
  int* flags;  // [0] overflow, [1] longest row
  int ibins;   // interior bins
};

// FP32 offsets of the binned particles from their bin centres, exactly as
// the binning writes them (k_bin_index), for a list built again from the
// same binning after the mixed force took the binning's copy over
__global__ void __launch_bounds__(256) k_xl_from_bins(const double4_32a* __restrict__ x4,
                                                      const int* __restrict__ binof, int n, int nbx, int nby, int nbz,
                                                      const double* __restrict__ ctab, float4* __restrict__ xl) {
  const int a = blockIdx.x * blockDim.x + threadIdx.x;
  if (a >= n) return;
  const int b = binof[a];
  const int bx = b / (nby * nbz), by = (b / nbz) % nby, bz = b % nbz;
  const double4_32a p = x4[a];
  xl[a] = make_float4(float(p.x - ctab[bx]), float(p.y - ctab[nbx + by]), float(p.z - ctab[nbx + nby + bz]),
                      __int_as_float(int(p.w)));
}

template <bool HALF, bool PACKED>
__global__ void __launch_bounds__(NB_THREADS) k_neigh_bin(NeighArgs a) {
  // each warp of the CTA builds the rows of its own bin with its own staging
  // arrays; the warps never wait for each other (more resident warps than one
  // warp per CTA allows, at the same shared memory per warp)
  __shared__ __align__(16) RowStage st[NB_WARPS];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int bin = blockIdx.x * NB_WARPS + warp;
  if (bin >= a.ibins) return;
  const int iy = a.r.nby - 2 * a.nhalo, iz = a.r.nbz - 2 * a.nhalo;
  const int mx = rows_of_bin<HALF, PACKED>(a.r, st[warp], bin / (iy * iz) + a.nhalo, (bin / iz) % iy + a.nhalo,
                                           bin % iz + a.nhalo, [&](int b, int& off) {
                                             off = a.binoffsets[b];
                                             return a.bincount[b];
                                           });
  // overflow flag and longest row: one atomic per warp into one of 64 slots
  // (a single shared address would serialise millions of atomics in L2)
  if (lane == 0) {
    if (mx > 0) atomicMax(&a.flags[1 + (bin & (NB_SLOTS - 1))], mx);
    if (mx > a.r.K) a.flags[0] = 1;
  }
}

// owned atoms outside every interior bin get an empty row (the reference
// never visits them)
__global__ void k_zero_rows(int* num, int n, int* flags) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) num[i] = 0;
  if (i < 1 + NB_SLOTS) flags[i] = 0;
}

// Row starts (NeighListCSR::row_map) in 64 bits: a list of 28 million liquid atoms has
// more than 2^31 entries.  Each tile of rows is scanned by one CTA, then the tiles'
// totals by one, which leaves the number of entries behind the last.
constexpr int RS_TILE = 1024;
__device__ __forceinline__ long long row_scan(long long v, long long& total) {
  __shared__ long long sh[RS_TILE / 32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  long long x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const long long y = __shfl_up_sync(FULL_MASK, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) sh[w] = x;
  __syncthreads();
  long long before = 0;
  total = 0;
  for (int k = 0; k < RS_TILE / 32; ++k) {
    before += k < w ? sh[k] : 0;
    total += sh[k];
  }
  __syncthreads();
  return before + x - v;
}
__global__ void __launch_bounds__(RS_TILE) k_row_starts(const int* __restrict__ num, int n,
                                                        long long* __restrict__ starts,
                                                        long long* __restrict__ tiles) {
  const int i = blockIdx.x * RS_TILE + threadIdx.x;
  long long total;
  const long long s = row_scan(i < n ? num[i] : 0, total);
  if (i < n) starts[i] = s;
  if (threadIdx.x == 0) tiles[blockIdx.x] = total;
}
__global__ void __launch_bounds__(RS_TILE) k_row_tiles(long long* tiles, int nt) {
  long long run = 0;
  for (int t0 = 0; t0 < nt; t0 += RS_TILE) {
    const int t = t0 + threadIdx.x;
    long long total;
    const long long s = row_scan(t < nt ? tiles[t] : 0, total);
    if (t < nt) tiles[t] = run + s;
    run += total;
  }
  if (threadIdx.x == 0) tiles[nt] = run;
}

// column-major rows -> CSR rows
__global__ void __launch_bounds__(256) k_rows_to_csr(const int* __restrict__ rows, int stride,
                                                     const int* __restrict__ num, const long long* __restrict__ starts,
                                                     const long long* __restrict__ tiles, int n,
                                                     int* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int m = num[i];
  out += starts[i] + tiles[i / RS_TILE];
  for (int k = 0; k < m; ++k) out[k] = rows[quad_index(i, k, stride)];
}

// packed entries -> plain j (for emd_neigh_get)
__global__ void k_unpack(int* __restrict__ e, long long n) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t < n) e[t] = e[t] >> 6;
}

}  // namespace
}  // namespace emd

using namespace emd;

// number of entries of the current list; forms the row starts
static long long neigh_total(Ctx& c) {
  if (c.neigh_total >= 0) return c.neigh_total;
  const int n = c.neigh_rows, nt = (n + RS_TILE - 1) / RS_TILE;
  if (n == 0) return c.neigh_total = 0;
  c.neigh_starts.reserve(size_t(n), c.stream);
  c.neigh_tiles.reserve(size_t(nt) + 1, c.stream);
  {
    TimedLaunch t(c, "neigh_row_starts");
    k_row_starts<<<nt, RS_TILE, 0, c.stream>>>(c.num_neighs.p, n, c.neigh_starts.p, c.neigh_tiles.p);
    EMD_CHECK_LAUNCH();
    k_row_tiles<<<1, RS_TILE, 0, c.stream>>>(c.neigh_tiles.p, nt);
    EMD_CHECK_LAUNCH();
  }
  EMD_CUDA(cudaMemcpyAsync(c.h_ll, c.neigh_tiles.p + nt, sizeof(long long), cudaMemcpyDeviceToHost, c.stream));
  EMD_CUDA(cudaStreamSynchronize(c.stream));
  return c.neigh_total = c.h_ll[0];
}

extern "C" {

emd_status emd_neigh_init(emd_ctx* ctx, int kind, double neigh_cut, int comm_newton) {
  EMD_API_BEGIN
  require(kind == EMD_NEIGH_CSR || kind == EMD_NEIGH_2D, EMD_ERR_ARG, "emd_neigh_init: kind");
  require(neigh_cut > 0, EMD_ERR_ARG, "emd_neigh_init: neigh_cut must be positive");
  c.neigh_kind = kind;
  c.neigh_cut = neigh_cut;
  c.comm_newton = comm_newton ? 1 : 0;
  c.maxneighs = 16;  // NeighList2D() initial capacity (neighbor_2d.h:101-104)
  c.neigh_scratch_k = 16;
  c.neigh_ready = false;
  EMD_API_END
}

emd_status emd_neigh_create(emd_ctx* ctx, int half_neigh, long long* total_out) {
  EMD_API_BEGIN
  require(c.neigh_cut > 0, EMD_ERR_STATE, "emd_neigh_init not called");
  require(c.binning_ready && c.bin_first == 0 && c.bin_count_n == c.N_local + c.N_ghost, EMD_ERR_STATE,
          "emd_neigh_create: needs a binning of owned and ghost particles");
  require(!c.bin_sorted, EMD_ERR_STATE,
          "emd_neigh_create: the last binning re-sorted the particles, so its permutation no longer refers to "
          "them; bin owned and ghost particles again without sorting first (as ExaMiniMD does)");
  require(c.nhalo >= 1, EMD_ERR_STATE,
          "emd_neigh_create: the binning has no halo bins; rows read the 27 bins around each interior one");
  const int n = c.N_local;
  c.half_neigh = half_neigh ? 1 : 0;
  const int packed = (c.lj_ready && c.lj_prec == EMD_PREC_MIXED) ? 1 : 0;
  require(!packed || (long long)(c.N_local + c.N_ghost) < (1LL << 25), EMD_ERR_ARG,
          "emd_neigh_create: packed rows need fewer than 2^25 particles");
  c.num_neighs.reserve(size_t(n) + 1, c.stream);
  c.resize_flag.reserve(1 + NB_SLOTS, c.stream);
  if (!c.xl_bin_valid) {  // a second build from one binning in the mixed form
    const int n_all = c.N_local + c.N_ghost;
    c.xl_bin.reserve(size_t(n_all) + 1, c.stream);
    if (n_all > 0) {
      TimedLaunch t(c, "neigh_xl_from_bins");
      k_xl_from_bins<<<blocks_for(n_all, 256), 256, 0, c.stream>>>(c.x4.p, c.binof.p, n_all, c.nbin[0], c.nbin[1],
                                                                   c.nbin[2], c.bin_ctab.p, c.xl_bin.p);
      EMD_CHECK_LAUNCH();
    }
    c.xl_bin_valid = true;
  }
  NeighArgs a;
  a.r.x4 = c.x4.p;
  a.r.xl = c.xl_bin.p;
  a.bincount = c.bincount.p;
  a.binoffsets = c.binoffsets.p;
  a.r.permute = c.permute.p;
  a.nbx = c.nbin[0];
  a.r.nby = c.nbin[1];
  a.r.nbz = c.nbin[2];
  a.nhalo = c.nhalo;
  a.r.wx = float((c.bmax[0] - c.bmin[0]) / c.nbin[0]);
  a.r.wy = float((c.bmax[1] - c.bmin[1]) / c.nbin[1]);
  a.r.wz = float((c.bmax[2] - c.bmin[2]) / c.nbin[2]);
  a.r.n_local = n;
  a.r.cutsq = c.neigh_cut * c.neigh_cut;
  const double band = row_band(std::max({double(a.r.wx), double(a.r.wy), double(a.r.wz)}), c.neigh_cut);
  a.r.cut_lo = float(a.r.cutsq * (1.0 - band));
  a.r.cut_hi = float(a.r.cutsq * (1.0 + band));
  a.r.newton = c.comm_newton;
  a.r.num_neighs = c.num_neighs.p;
  a.r.stride = n + 1;
  a.flags = c.resize_flag.p;
  const int ibins = (c.nbin[0] - 2 * c.nhalo) * (c.nbin[1] - 2 * c.nhalo) * (c.nbin[2] - 2 * c.nhalo);
  a.ibins = ibins;
  const bool two_d = c.neigh_kind == EMD_NEIGH_2D;
  int& K = two_d ? c.maxneighs : c.neigh_scratch_k;
  DevBuf<int>& rows = two_d ? c.neighs : c.neigh_rows2d;
  // row starts and total are read when asked for (emd_neigh_get): the force
  // kernels take the column-major rows of either kind of list as they are
  while (true) {
    rows.reserve(size_t(n + 1) * size_t((K + 3) & ~3) + 4, c.stream);
    a.r.rows = rows.p;
    a.r.K = K;
    {
      TimedLaunch t(c, "neigh_zero_rows");
      k_zero_rows<<<blocks_for(std::max(n, 1 + NB_SLOTS), 256), 256, 0, c.stream>>>(c.num_neighs.p, n,
                                                                                  c.resize_flag.p);
      EMD_CHECK_LAUNCH();
    }
    if (n > 0) {
      if (ibins > 0) {
        TimedLaunch t(c, "neigh_build");
        auto k = c.half_neigh ? (packed ? k_neigh_bin<true, true> : k_neigh_bin<true, false>)
                        : (packed ? k_neigh_bin<false, true> : k_neigh_bin<false, false>);
        k<<<(ibins + NB_WARPS - 1) / NB_WARPS, NB_THREADS, 0, c.stream>>>(a);
        EMD_CHECK_LAUNCH();
      }
    }
    EMD_CUDA(cudaMemcpyAsync(c.h_int, c.resize_flag.p, (1 + NB_SLOTS) * sizeof(int), cudaMemcpyDeviceToHost,
                             c.stream));
    EMD_CUDA(cudaStreamSynchronize(c.stream));
    int longest = 0;
    for (int k = 1; k <= NB_SLOTS; ++k) longest = std::max(longest, c.h_int[k]);
    c.h_int[1] = longest;
    c.neigh_maxrow = n > 0 ? longest : 0;
    if (!c.h_int[0]) break;
    // neighbor_2d.h:325-327: grow to 1.2x the longest row and redo
    K = int(c.h_int[1] * 1.2);
  }
  if (packed) {
    const int n_all = c.N_local + c.N_ghost;
    c.abin.reserve(size_t(n_all) + 1, c.stream);
    EMD_CUDA(cudaMemcpyAsync(c.abin.p, c.binof.p, sizeof(int) * n_all, cudaMemcpyDeviceToDevice, c.stream));
  }
  c.neigh_stride = n + 1;
  c.neigh_rows = n;
  c.neigh_total = -1;
  c.neigh_ready = true;
  c.neigh_packed = packed;
  c.neigh_builds++;
  if (packed) lj_mixed_after_build(c);
  if (total_out) *total_out = neigh_total(c);
  EMD_API_END
}

emd_status emd_neigh_get(emd_ctx* ctx, int* num_neighs, int* entries) {
  EMD_API_BEGIN
  require(c.neigh_ready, EMD_ERR_STATE, "emd_neigh_get: no neighbour list");
  const DeviceGuard device(c.device);
  const int n = c.neigh_rows;
  neigh_total(c);
  if (num_neighs && n > 0)
    EMD_CUDA(cudaMemcpyAsync(num_neighs, c.num_neighs.p, sizeof(int) * n, cudaMemcpyDeviceToHost, c.stream));
  if (entries && c.neigh_total > 0) {
    DevBuf<int> tmp;
    tmp.reserve(size_t(c.neigh_total), c.stream);
    k_rows_to_csr<<<blocks_for(n, 256), 256, 0, c.stream>>>(neigh_rows(c), c.neigh_stride, c.num_neighs.p,
                                                            c.neigh_starts.p, c.neigh_tiles.p, n, tmp.p);
    EMD_CHECK_LAUNCH();
    if (c.neigh_packed) {
      k_unpack<<<blocks_for(c.neigh_total, 256), 256, 0, c.stream>>>(tmp.p, c.neigh_total);
      EMD_CHECK_LAUNCH();
    }
    EMD_CUDA(cudaMemcpyAsync(entries, tmp.p, sizeof(int) * c.neigh_total, cudaMemcpyDeviceToHost, c.stream));
    EMD_CUDA(cudaStreamSynchronize(c.stream));
    tmp.release();
  }
  EMD_CUDA(cudaStreamSynchronize(c.stream));
  EMD_API_END
}

emd_status emd_neigh_maxneighs(emd_ctx* ctx, int* maxneighs) {
  EMD_API_BEGIN
  if (maxneighs) *maxneighs = c.neigh_kind == EMD_NEIGH_2D ? c.maxneighs : 0;
  EMD_API_END
}

}  // extern "C"
