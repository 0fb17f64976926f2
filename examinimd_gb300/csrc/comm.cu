// CommSerial on the device (comm_serial.h:95-213, comm_serial.cpp:47-127):
// periodic wrap, six-phase ghost creation with stable (count + place)
// compaction so ghosts land at exactly the indices the serial reference
// gives them, one-launch ghost position refresh, and the phase-ordered
// reverse force accumulation.  -fmad=false (pure add/sub anyway).
#include <cooperative_groups.h>

#include <algorithm>
#include <cstring>

#include "emd_device.cuh"
#include "emd_internal.h"

namespace emd {
namespace {

// TagExchangeSelf (comm_serial.h:95-108): each condition tests the
// coordinate as it was before the call.
__global__ void k_exchange(double4_32a* __restrict__ x4, int n, double lx, double ly, double lz) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double4_32a p = x4[i];
  // compared as integers (a double comparison takes the FP64 pipe, six of them most
  // of this kernel: 0.098 -> 0.053 ms for 4,000,000); bits of x > 0 order as integers,
  // those of x < 0 have the sign and are not minus zero's
  auto wrap = [](double& v, double l) {
    const long long b = __double_as_longlong(v);
    if (b > __double_as_longlong(l)) v -= l;
    else if (b < 0 && b != (-0x7fffffffffffffffLL - 1)) v += l;
  };
  wrap(p.x, lx);
  wrap(p.y, ly);
  wrap(p.z, lz);
  x4[i] = p;
}

__device__ __forceinline__ double comp(const double4_32a& p, int d) { return d == 0 ? p.x : (d == 1 ? p.y : p.z); }

// TagHaloSelf (comm_serial.h:112-181) for both phases of one dimension: the
// upper face's particles (x >= hi - depth, imaged at x - L) in index order, then
// the lower face's (x <= lo + depth).  The odd phase's candidates are the even
// phase's (comm_serial.cpp:68 leaves out only the ghosts the even phase made).
// k_halo_count counts them per tile of the candidates, its last block to finish
// scans the tiles; k_halo_place finds each particle's rank and writes its image.
// The number of candidates and the room left are read on the device, so the three
// dimensions run without a read-back in between: seven operations and one wait
// (nine launches or copies and a wait per dimension took 150 us in a small system).
constexpr int HALO_THREADS = 256, HALO_PER = 4, HALO_TILE = HALO_THREADS * HALO_PER;
struct HaloState {
  int base[4];     // ghosts before dimension d; after the last
  int upper[3];    // ghosts of the upper face
  int overflow;    // particles needed when they were more than the capacity
  unsigned done[3];  // blocks of k_halo_count that finished
};
static_assert(sizeof(HaloState) <= kHostInts * sizeof(int), "read back through the pinned scratch");

// a tile's flags: bit k and 16 + k of the thread's candidate 4 tid + k, upper and lower
__device__ __forceinline__ int halo_flags(const double4_32a* __restrict__ x4, int first, int n, int dim, double hi,
                                          double lo) {
  int m = 0;
#pragma unroll
  for (int k = 0; k < HALO_PER; ++k)
    if (first + k < n) {
      const double c = comp(x4[first + k], dim);
      m |= (c >= hi ? 1 << k : 0) | (c <= lo ? 0x10000 << k : 0);
    }
  return m;
}
__device__ __forceinline__ int halo_counts(int m) { return __popc(m & 0xffff) | __popc(m >> 16) << 16; }

// exclusive block scan (256 threads) and total of an int that holds two 16-bit counts
__device__ __forceinline__ int halo_scan(int v, int& total) {
  __shared__ int sh[HALO_THREADS / 32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(FULL_MASK, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) sh[w] = x;
  __syncthreads();
  int off = 0;
  total = 0;
#pragma unroll
  for (int k = 0; k < HALO_THREADS / 32; ++k) {
    off += k < w ? sh[k] : 0;
    total += sh[k];
  }
  __syncthreads();
  return off + x - v;
}

// tiles: (upper, lower) counts, then ranks of each tile's first
__global__ void __launch_bounds__(HALO_THREADS) k_halo_count(const double4_32a* __restrict__ x4, int n_local,
                                                             int capacity, int dim, double hi, double lo,
                                                             HaloState* st, int2* __restrict__ tiles) {
  __shared__ bool s_last;
  __shared__ int s_run[2];
  const int n = n_local + st->base[dim], nt = (n + HALO_TILE - 1) / HALO_TILE;
  if (blockIdx.x < nt && !st->overflow) {
    int total;
    const int m = halo_flags(x4, blockIdx.x * HALO_TILE + threadIdx.x * HALO_PER, n, dim, hi, lo);
    halo_scan(halo_counts(m), total);
    if (threadIdx.x == 0) tiles[blockIdx.x] = int2{total & 0xffff, total >> 16};
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) {
    s_last = atomicAdd(&st->done[dim], 1u) == gridDim.x - 1;
    s_run[0] = s_run[1] = 0;
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  if (st->overflow) return;
  for (int t0 = 0; t0 < nt; t0 += HALO_THREADS) {
    const int t = t0 + threadIdx.x;
    const int2 c = t < nt ? __ldcg(tiles + t) : int2{0, 0};
    // a tile's counts reach 1,024: two scans
    int tu, tl;
    const int u = halo_scan(c.x, tu), l = halo_scan(c.y, tl);
    const int ru = s_run[0], rl = s_run[1];
    if (t < nt) tiles[t] = int2{ru + u, rl + l};
    __syncthreads();
    if (threadIdx.x == 0) {
      s_run[0] = ru + tu;
      s_run[1] = rl + tl;
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    const long long need = (long long)n + s_run[0] + s_run[1];
    st->upper[dim] = s_run[0];
    st->base[dim + 1] = st->base[dim] + s_run[0] + s_run[1];
    if (need > capacity) st->overflow = int(min(need, 0x7fffffffLL));
  }
}

struct HaloParticles {
  double4_32a* x4;
  double *v, *q;
  int *id, *type, *pack, *owner, *img;
};
// ghost g: the image of particle i across a face of dimension dim
__device__ __forceinline__ void halo_image(const HaloParticles& P, int n_local, int dim, bool lower, double L, int i,
                                           int g) {
  const int dst = n_local + g;
  const double shift = lower ? L : -L;
  double4_32a p = P.x4[i];
  const double v0 = P.v[3 * size_t(i)], v1 = P.v[3 * size_t(i) + 1], v2 = P.v[3 * size_t(i) + 2], qi = P.q[i];
  const int idi = P.id[i], ti = P.type[i];
  const int own = i < n_local ? i : P.owner[i - n_local], im = i < n_local ? 0 : P.img[i - n_local];
  if (dim == 0) p.x += shift;
  else if (dim == 1) p.y += shift;
  else p.z += shift;
  P.x4[dst] = p;
  P.v[3 * size_t(dst)] = v0;
  P.v[3 * size_t(dst) + 1] = v1;
  P.v[3 * size_t(dst) + 2] = v2;
  P.q[dst] = qi;
  P.id[dst] = idi;
  P.type[dst] = ti;
  P.pack[g] = i;
  P.owner[g] = own;
  P.img[g] = im | 1 << (2 * dim + (lower ? 1 : 0));
}

__global__ void __launch_bounds__(HALO_THREADS) k_halo_place(HaloParticles P, int n_local, int dim, double hi,
                                                             double lo, double L, const HaloState* __restrict__ st,
                                                             const int2* __restrict__ tiles) {
  const int base = st->base[dim], n = n_local + base;
  if (blockIdx.x * HALO_TILE >= n || st->overflow) return;
  const int first = blockIdx.x * HALO_TILE + threadIdx.x * HALO_PER;
  const int m = halo_flags(P.x4, first, n, dim, hi, lo);
  int total;
  const int before = halo_scan(halo_counts(m), total);
  // the tile's images in order, so that every thread copies one at a time
  __shared__ unsigned short list[2 * HALO_TILE];
  const int nu = total & 0xffff, nl = total >> 16;
  int u = before & 0xffff, l = nu + (before >> 16);
#pragma unroll
  for (int k = 0; k < HALO_PER; ++k) {
    if (m >> k & 1) list[u++] = (unsigned short)(threadIdx.x * HALO_PER + k);
    if (m >> (16 + k) & 1) list[l++] = (unsigned short)(threadIdx.x * HALO_PER + k);
  }
  __syncthreads();
  const int2 tile = tiles[blockIdx.x];
  for (int e = threadIdx.x; e < nu + nl; e += HALO_THREADS) {
    const bool lower = e >= nu;
    const int i = blockIdx.x * HALO_TILE + list[e];
    const int g = lower ? base + st->upper[dim] + tile.y + e - nu : base + tile.x + e;
    halo_image(P, n_local, dim, lower, L, i, g);
  }
}

// The halo of a small system by one CTA (864 atoms: seven operations, 41 us, 27 in
// one; 64 atoms: 40 and 15).  `st` is the pinned read-back scratch: a copy after
// the kernel cost 8 us of a rebuild step (204 us with it, 196 without).
constexpr int HALO_SMALL = 1024, HALO_SMALL_THREADS = 1024;
struct HaloBounds {
  double hi[3], lo[3], L[3];
};
__global__ void __launch_bounds__(HALO_SMALL_THREADS) k_halo_small(HaloParticles P, int n_local, int capacity,
                                                                   HaloBounds B, HaloState* st) {
  __shared__ int wu[32], wl[32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const unsigned lt = (1u << lane) - 1u;
  HaloState h{};
  for (int dim = 0; dim < 3; ++dim) {
    const int base = h.base[dim], n = n_local + base;
    const double hi = B.hi[dim], lo = B.lo[dim];
    int nu = 0, nl = 0;
    for (int i0 = 0; i0 < n; i0 += HALO_SMALL_THREADS) {
      const int i = i0 + tid;
      const double c = i < n ? comp(P.x4[i], dim) : 0.0;
      nu += __syncthreads_count(i < n && c >= hi);
      nl += __syncthreads_count(i < n && c <= lo);
    }
    h.upper[dim] = nu;
    h.base[dim + 1] = base + nu + nl;
    if (n + nu + nl > capacity) {
      h.overflow = n + nu + nl;
      break;
    }
    int gu = base, gl = base + nu;  // ghosts of the next tile
    for (int i0 = 0; i0 < n; i0 += HALO_SMALL_THREADS) {
      const int i = i0 + tid;
      const double c = i < n ? comp(P.x4[i], dim) : 0.0;
      const bool u = i < n && c >= hi, l = i < n && c <= lo;
      const unsigned bu = __ballot_sync(FULL_MASK, u), bl = __ballot_sync(FULL_MASK, l);
      if (lane == 0) {
        wu[warp] = __popc(bu);
        wl[warp] = __popc(bl);
      }
      __syncthreads();
      int ru = gu + __popc(bu & lt), rl = gl + __popc(bl & lt);
      for (int k = 0; k < 32; ++k) {
        ru += k < warp ? wu[k] : 0;
        rl += k < warp ? wl[k] : 0;
        gu += wu[k];
        gl += wl[k];
      }
      if (u) halo_image(P, n_local, dim, false, B.L[dim], i, ru);
      if (l) halo_image(P, n_local, dim, true, B.L[dim], i, rl);
      __syncthreads();
    }
  }
  if (tid == 0) *st = h;
}

// TagHaloUpdateSelf for all six phases at once: every ghost is its owner
// shifted by +-L in each dimension it was imaged across; each coordinate is
// shifted at most once, so this equals the reference's chained phases bit
// for bit.
__global__ void k_halo_update(double4_32a* __restrict__ x4, const int* __restrict__ owner,
                              const int* __restrict__ img, int n_local, int n_ghost, double lx, double ly,
                              double lz, BinCentres ctr, float4* __restrict__ xl) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= n_ghost) return;
  const int m = img[g];
  double4_32a p = x4[owner[g]];
  if (m & 1) p.x -= lx;
  if (m & 2) p.x += lx;
  if (m & 4) p.y -= ly;
  if (m & 8) p.y += ly;
  if (m & 16) p.z -= lz;
  if (m & 32) p.z += lz;
  x4[n_local + g] = p;  // w (the type) is the owner's, as the halo build copied it
  if (xl) {  // mixed form: FP32 position relative to the ghost's bin centre
    const double4_32a q = ctr.at(n_local + g);
    xl[n_local + g] = make_float4(float(p.x - q.x), float(p.y - q.y), float(p.z - q.z), __int_as_float(int(p.w)));
  }
}

// TagHaloForceSelf for one phase (comm_serial.h:200-213).  Within a phase
// every source index appears once, so plain adds are race free.
__global__ void k_halo_force(double* __restrict__ f, const int* __restrict__ pack, int count, int ghost_base) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= count) return;
  const int i = pack[k];
  const int g = ghost_base + k;
  f[3 * i] += f[3 * g];
  f[3 * i + 1] += f[3 * g + 1];
  f[3 * i + 2] += f[3 * g + 2];
}

// The six phases in order by one CTA, or one cluster of eight, which goes past L1
// because a phase reads what another CTA wrote.  Six launches take 24.8 us whatever their
// additions, up to 250,000 ghosts; one CTA 14.5 for 5,841 ghosts, the cluster 18.6 for 13,275
// and 19.4 for 42,381, but 24.8 for 50,760, 30.9 for 59,895 and 53.4 for 160,191: eight
// SMs, so the launches take over at 50,000.
constexpr int HALO_FORCE_MAX = 50000, HALO_FORCE_ONE = 8192, HALO_FORCE_CTAS = 8, HALO_FORCE_THREADS = 1024;
struct HaloPhases {
  int pack[6], count[6], ghost[6];
};
template <bool CLUSTER>
__global__ void __launch_bounds__(HALO_FORCE_THREADS)
    k_halo_force_all(double* __restrict__ f, const int* __restrict__ pack, HaloPhases P) {
  for (int phase = 5; phase >= 0; --phase) {
    for (int k = blockIdx.x * HALO_FORCE_THREADS + threadIdx.x; k < P.count[phase];
         k += gridDim.x * HALO_FORCE_THREADS) {
      const int i = pack[P.pack[phase] + k], g = P.ghost[phase] + k;
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        double *fi = f + 3 * size_t(i) + d, *fg = f + 3 * size_t(g) + d;
        if (CLUSTER) __stcg(fi, __ldcg(fi) + __ldcg(fg));
        else *fi += *fg;
      }
    }
    if (phase == 0) break;
    if (CLUSTER) cooperative_groups::this_cluster().sync();
    else __syncthreads();
  }
}

}  // namespace

static void reserve_particles(Ctx& c, size_t need) {
  const size_t n = need + 1;
  c.x4.reserve(n, c.stream, true);
  c.v.reserve(3 * n, c.stream, true);
  c.f.reserve(3 * n, c.stream, true);
  c.q.reserve(n, c.stream, true);
  c.type.reserve(n, c.stream, true);
  c.id.reserve(n, c.stream, true);
}

static void grow_particles(Ctx& c, int need) {
  if (need <= c.N_max) return;
  reserve_particles(c, size_t(need));
  // new force rows are cleared by the per-step deep_copy(f, 0) (emd_zero_forces)
  c.N_max = need;
}

}  // namespace emd

using namespace emd;

extern "C" {

emd_status emd_comm_init(emd_ctx* ctx, double comm_depth) {
  EMD_API_BEGIN
  require(comm_depth > 0, EMD_ERR_ARG, "emd_comm_init: comm_depth must be positive");
  c.comm_depth = comm_depth;
  EMD_API_END
}

emd_status emd_comm_exchange(emd_ctx* ctx) {
  EMD_API_BEGIN
  c.x_version++;
  if (c.N_local == 0) return EMD_OK;
  TimedLaunch t(c, "comm_exchange");
  c.xl_ok &= ~1;
  k_exchange<<<blocks_for(c.N_local, 256), 256, 0, c.stream>>>(c.x4.p, c.N_local, c.domain[0], c.domain[1],
                                                               c.domain[2]);
  EMD_CHECK_LAUNCH();
  EMD_API_END
}

emd_status emd_comm_exchange_halo(emd_ctx* ctx, int* n_ghost_out) {
  EMD_API_BEGIN
  require(c.comm_depth > 0, EMD_ERR_STATE, "emd_comm_exchange_halo: emd_comm_init not called");
  for (int d = 0; d < 3; ++d)
    require(c.comm_depth < c.domain[d], EMD_ERR_ARG,
            "emd_comm_exchange_halo: comm_depth must be smaller than the box (one periodic image per face)");
  const int N_local = c.N_local;
  c.neigh_ready = false;
  c.xl_ok &= ~2;
  c.halo_state.reserve(sizeof(HaloState), c.stream);
  HaloState* st = reinterpret_cast<HaloState*>(c.halo_state.p);
  HaloState h{};
  while (N_local > 0) {
    // room for particles; the reference grows System and the pack list, then
    // redoes the phase
    const size_t room = std::min({c.x4.cap, c.v.cap / 3, c.f.cap / 3, c.q.cap, c.type.cap, c.id.cap}) - 1;
    const int capacity = int(std::min<size_t>(room, 0x7ffffffe));
    const size_t ghosts = size_t(std::max(0, capacity - N_local)) + 1;
    const int blocks = (capacity + HALO_TILE - 1) / HALO_TILE;
    c.pack.reserve(ghosts, c.stream);
    c.ghost_owner.reserve(ghosts, c.stream);
    c.ghost_img.reserve(ghosts, c.stream);
    c.halo_tiles.reserve(size_t(blocks) + 1, c.stream);
    const HaloParticles P{c.x4.p, c.v.p, c.q.p, c.id.p, c.type.p, c.pack.p, c.ghost_owner.p, c.ghost_img.p};
    HaloBounds B;
    for (int d = 0; d < 3; ++d) {
      B.hi[d] = c.sub_hi[d] - c.comm_depth;
      B.lo[d] = c.sub_lo[d] + c.comm_depth;
      B.L[d] = c.domain[d];
    }
    if (N_local <= HALO_SMALL) {
      TimedLaunch t(c, "comm_halo_small");
      // the counts straight into the pinned read-back scratch
      k_halo_small<<<1, HALO_SMALL_THREADS, 0, c.stream>>>(P, N_local, capacity, B,
                                                           reinterpret_cast<HaloState*>(c.h_int));
      EMD_CHECK_LAUNCH();
    } else {
      EMD_CUDA(cudaMemsetAsync(st, 0, sizeof(HaloState), c.stream));
      for (int dim = 0; dim < 3; ++dim) {
        {
          TimedLaunch t(c, "comm_halo_count");
          k_halo_count<<<blocks, HALO_THREADS, 0, c.stream>>>(c.x4.p, N_local, capacity, dim, B.hi[dim], B.lo[dim], st,
                                                              c.halo_tiles.p);
          EMD_CHECK_LAUNCH();
        }
        TimedLaunch t(c, "comm_halo_place");
        k_halo_place<<<blocks, HALO_THREADS, 0, c.stream>>>(P, N_local, dim, B.hi[dim], B.lo[dim], B.L[dim], st,
                                                            c.halo_tiles.p);
        EMD_CHECK_LAUNCH();
      }
      EMD_CUDA(cudaMemcpyAsync(c.h_int, st, sizeof(HaloState), cudaMemcpyDeviceToHost, c.stream));
    }
    EMD_CUDA(cudaStreamSynchronize(c.stream));
    std::memcpy(&h, c.h_int, sizeof h);
    require((long long)N_local + std::max(h.base[1], h.base[2]) < (1LL << 30), EMD_ERR_OVERFLOW_GHOST,
            "emd_comm_exchange_halo: more than 2^30 particles");
    require(h.overflow < 0x7fffffff, EMD_ERR_OVERFLOW_GHOST, "emd_comm_exchange_halo: more than 2^31 particles");
    if (!h.overflow) break;
    // at least what is known to be needed, and what a uniform density needs
    double part = 1.0;
    for (int d = 0; d < 3; ++d)
      part *= 1.0 + 2.0 * c.comm_depth / c.domain[d];
    const size_t known = size_t(h.overflow);
    const size_t guess = size_t(std::min(double(0x7ffffffe), std::max(double(known), N_local * part)));
    try {
      reserve_particles(c, guess);
    } catch (const Error& e) {
      if (e.code != EMD_ERR_NOMEM || guess == known) throw;
      reserve_particles(c, known);
    }
  }
  const int N_ghost = h.base[3];
  grow_particles(c, N_local + N_ghost);
  for (int dim = 0; dim < 3; ++dim) {
    c.num_ghost[2 * dim] = h.upper[dim];
    c.num_ghost[2 * dim + 1] = h.base[dim + 1] - h.base[dim] - h.upper[dim];
    c.ghost_offsets[2 * dim] = N_local + h.base[dim];
    c.ghost_offsets[2 * dim + 1] = N_local + h.base[dim] + h.upper[dim];
  }
  c.N_ghost = N_ghost;
  if (n_ghost_out) *n_ghost_out = N_ghost;
  EMD_API_END
}

emd_status emd_comm_update_halo(emd_ctx* ctx) {
  EMD_API_BEGIN
  if (c.N_ghost == 0) return EMD_OK;
  TimedLaunch t(c, "comm_update_halo");
  const bool live = mixed_xl_active(c);
  k_halo_update<<<blocks_for(c.N_ghost, 256), 256, 0, c.stream>>>(
      c.x4.p, c.ghost_owner.p, c.ghost_img.p, c.N_local, c.N_ghost, c.domain[0], c.domain[1], c.domain[2],
      bin_centres(c), live ? c.xl.p : nullptr);
  if (!live) c.xl_ok &= ~2;
  EMD_CHECK_LAUNCH();
  EMD_API_END
}

emd_status emd_comm_update_force(emd_ctx* ctx) {
  EMD_API_BEGIN
  int pack_off[6];
  int acc = 0;
  for (int p = 0; p < 6; ++p) {
    pack_off[p] = acc;
    acc += c.num_ghost[p];
  }
  materialize_kick(c);  // owned forces are about to change
  materialize_zero(c, true, true);
  if (acc > 0 && acc <= HALO_FORCE_MAX) {
    HaloPhases P;
    for (int p = 0; p < 6; ++p) {
      P.pack[p] = pack_off[p];
      P.count[p] = c.num_ghost[p];
      P.ghost[p] = c.ghost_offsets[p];
    }
    TimedLaunch t(c, "comm_update_force");
    if (acc <= HALO_FORCE_ONE) {
      k_halo_force_all<false><<<1, HALO_FORCE_THREADS, 0, c.stream>>>(c.f.p, c.pack.p, P);
      EMD_CHECK_LAUNCH();
      return EMD_OK;
    }
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(HALO_FORCE_CTAS);
    cfg.blockDim = dim3(HALO_FORCE_THREADS);
    cfg.stream = c.stream;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = HALO_FORCE_CTAS;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    EMD_CUDA(cudaLaunchKernelEx(&cfg, k_halo_force_all<true>, c.f.p, static_cast<const int*>(c.pack.p), P));
    return EMD_OK;
  }
  for (int phase = 5; phase >= 0; --phase) {
    const int count = c.num_ghost[phase];
    if (count == 0) continue;
    TimedLaunch t(c, "comm_update_force");
    k_halo_force<<<blocks_for(count, 256), 256, 0, c.stream>>>(c.f.p, c.pack.p + pack_off[phase], count,
                                                              c.ghost_offsets[phase]);
    EMD_CHECK_LAUNCH();
  }
  EMD_API_END
}

emd_status emd_comm_get_ghosts(emd_ctx* ctx, int num_ghost[6], int* pack_indices) {
  EMD_API_BEGIN
  int total = 0;
  for (int p = 0; p < 6; ++p) {
    if (num_ghost) num_ghost[p] = c.num_ghost[p];
    total += c.num_ghost[p];
  }
  if (pack_indices && total > 0) {
    EMD_CUDA(cudaMemcpyAsync(pack_indices, c.pack.p, sizeof(int) * total, cudaMemcpyDeviceToHost, c.stream));
    EMD_CUDA(cudaStreamSynchronize(c.stream));
  }
  EMD_API_END
}

}  // extern "C"
