// Batched LJ ensemble: many independent periodic systems of uneven size
// advanced together, mixed precision.
//
// One CTA owns one system for the whole launch and runs its timesteps back
// to back; systems never talk to each other, so no grid-wide
// synchronisation is needed.  Per system the CTA runs the same step as the
// single-system path:
//   - NVE half kick and drift;
//   - every `every` steps: wrap, halo rebuilt by three sweeps (x, y, z, each
//     over the owned atoms and the ghosts of the earlier sweeps), counting-sort
//     binning in shared memory, FP32 bin-relative positions, and the full
//     neighbour list in packed column-major rows;
//   - otherwise the halo refresh;
//   - the mixed LJ force (lj_pair.cuh);
//   - the final half kick.
// Phases are separated by __syncthreads.
//
// Systems are ordered largest first, so their CTAs start first.  The host
// captures a run's launches (`steps_per_launch` steps each) in a CUDA graph.
//
// A second, phased form keeps the per-system rebuild (wrap, halo, binning)
// on one CTA per system and runs the rest over chunks of all systems, so one
// large system no longer sets the time of a step.  A step is two launches: halo
// refresh (or, on a rebuild step, the rebuild and the neighbour rows, a warp
// per bin), then force, final half kick and the next step's half kick and drift
// in one kernel that writes the new positions to a second set of buffers, since
// other atoms still read the old ones.  All of a run's launches again go into one
// CUDA graph.  Both forms do the same per-atom arithmetic in the same order.
// 1,360,000 atoms in 256 systems, ms per 20 steps: 9.7 with a launch per phase and
// rows an atom per thread, 5.9 as it is.
//
// emd_batch_tune picks the form, the CTA size and the steps per launch by
// timing the candidates on the ensemble itself.
//
// Differences from the single-system path:
//   - halo image order (sweeps instead of the six CommSerial phases);
//   - within-bin order (ascending index, like the reference's sorted binning).
// Both only change the order of the force summation; the pair set is the same.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <numeric>
#include <string>
#include <vector>

#include "../../include/emd_batch.h"
#include "emd_device.cuh"
#include "emd_internal.h"
#include "lj_pair.cuh"
#include "neigh_bin.cuh"
#include "neigh_rows.cuh"

namespace emd {
namespace {

constexpr int BATCH_MAX_THREADS = 1024;

struct BSys {
  double L[3];   // orthorhombic box [0, L)
  double w[3];   // bin widths
  int nb[3];     // interior bins per dimension (halo layer of one bin on each side)
  int n;         // owned atoms
  int base;      // first particle slot: owned atoms, then ghosts
  int cap;       // particle slots
  int bin_base;  // first bin slot: (nb+2)^3 bins + 1
  long long out;       // first atom in the caller's arrays
  long long row_base;  // first int of the neighbour rows (column-major quads, stride n, capacity K)
};

struct BArgs {
  const BSys* sys;
  double4_32a* x;  // FP64 positions (w unused)
  float4* xl;      // FP32 positions relative to the particle's bin centre
  double* v;       // 3 per particle slot (owned only)
  double* f;       // 3 per particle slot (owned only)
  int* owner;      // per particle slot: ghost -> owned particle (system-local)
  int* img;        // per particle slot: 2 bits per dimension, shift + 1
  int* binof;      // per particle slot: system-local bin
  ushort4* binc;   // per particle slot: its bin's coordinates and img
  const double* mid;  // k - 0.5: centre of bin k in bin widths
  double4_32a* xn;    // phased form: the next step's x and xl
  float4* xln;
  int* perm;       // per particle slot: particles sorted by bin (system-local indices)
  int* binstart;   // per bin slot: first position in perm
  int* num;        // per particle slot (owned): row length
  int* rows;
  int* nghost;     // per system
  unsigned* status;
  int K;
  double dt, dtf;
  double cut_nb, cutsq_nb;
  float nb_lo, nb_hi;  // FP32 decision band of the neighbour test
  LJParamsF P;
  int n_chunks;  // of owned atoms, in front of the ghosts' chunks
  int every;
  int step0, nsteps;   // steps step0+1 .. step0+nsteps
};

// inclusive scan within a warp
__device__ __forceinline__ int warp_incl(int x, int lane) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(FULL_MASK, x, o);
    if (lane >= o) x += y;
  }
  return x;
}

// exclusive block scan of one int per thread; `sh` holds 33 ints
__device__ __forceinline__ int block_excl(int v, int* sh, int& total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  const int x = warp_incl(v, lane);
  if (lane == 31) sh[warp] = x;
  __syncthreads();
  if (warp == 0) {
    const int t = lane < nw ? sh[lane] : 0;
    const int s = warp_incl(t, lane);
    if (lane < nw) sh[lane] = s;
  }
  __syncthreads();
  const int off = warp > 0 ? sh[warp - 1] : 0;
  total = sh[nw - 1];
  __syncthreads();
  return off + x - v;
}

__device__ __forceinline__ void bin_coords(const BSys& S, int b, int& bx, int& by, int& bz) {
  const int ny = S.nb[1] + 2, nz = S.nb[2] + 2;
  bx = b / (ny * nz);
  by = (b / nz) % ny;
  bz = b % nz;
}

__device__ __forceinline__ float4 rel_to_bin(const BArgs& A, const BSys& S, const double4_32a& p, ushort4 b) {
  return make_float4(float(fma(-A.mid[b.x], S.w[0], p.x)), float(fma(-A.mid[b.y], S.w[1], p.y)),
                     float(fma(-A.mid[b.z], S.w[2], p.z)), 0.f);
}

// exact FP64 neighbour test of a candidate inside the FP32 band (out of line:
// see lj_pair.cuh)
__device__ __noinline__ bool nb_fp64(const double4_32a* __restrict__ x, int i, int j, double cutsq) {
  const double4_32a a = x[i], b = x[j];
  const double dx = a.x - b.x, dy = a.y - b.y, dz = a.z - b.z;
  return dx * dx + dy * dy + dz * dz <= cutsq;
}

// neighbour row of owned atom i (system-local), stencil bins x slowest,
// each bin in ascending index
__device__ void build_row(const BArgs& A, const BSys& S, int i) {
  const double4_32a* x = A.x + S.base;
  const float4* xl = A.xl + S.base;
  const int* binof = A.binof + S.base;
  const int* perm = A.perm + S.base;
  const int* bstart = A.binstart + S.bin_base;
  int* rows = A.rows + S.row_base;
  const int n = S.n;
  const float wx = float(S.w[0]), wy = float(S.w[1]), wz = float(S.w[2]);
  const float4 xi = xl[i];
  int bx, by, bz;
  bin_coords(S, binof[i], bx, by, bz);
  // A stencil bin whose box (centre d w in i's frame, half-width w / 2 plus
  // a margin far above rounding) lies farther than the band's upper edge
  // (x 1.001) from i holds no candidate i would accept or re-test: skipped,
  // which leaves the row unchanged.
  const float hx = 0.5001f * wx, hy = 0.5001f * wy, hz = 0.5001f * wz;
  const float prune_sq = A.nb_hi * 1.001f;
  int cnt = 0;
  for (int dx = -1; dx <= 1; ++dx)
    for (int dy = -1; dy <= 1; ++dy)
      for (int dz = -1; dz <= 1; ++dz) {
        const float ex = fmaxf(fabsf(xi.x - float(dx) * wx) - hx, 0.f);
        const float ey = fmaxf(fabsf(xi.y - float(dy) * wy) - hy, 0.f);
        const float ez = fmaxf(fabsf(xi.z - float(dz) * wz) - hz, 0.f);
        if (ex * ex + ey * ey + ez * ez > prune_sq) continue;
        const int bj = ((bx + dx) * (S.nb[1] + 2) + (by + dy)) * (S.nb[2] + 2) + (bz + dz);
        const float sx = -dx * wx, sy = -dy * wy, sz = -dz * wz;
        const int code = ((dx + 1) << 4) | ((dy + 1) << 2) | (dz + 1);
        const int e1 = bstart[bj + 1];
        for (int k = bstart[bj]; k < e1; ++k) {
          const int j = perm[k];
          if (j == i) continue;
          const float4 xj = xl[j];
          const float ddx = (xi.x - xj.x) + sx, ddy = (xi.y - xj.y) + sy, ddz = (xi.z - xj.z) + sz;
          const float rsq = ddx * ddx + ddy * ddy + ddz * ddz;
          bool in = rsq < A.nb_lo;
          if (!in && rsq <= A.nb_hi) in = nb_fp64(x, i, j, A.cutsq_nb);
          if (in) {
            if (cnt < A.K) rows[quad_index(i, cnt, n)] = (j << 6) | code;
            ++cnt;
          }
        }
      }
  A.num[S.base + i] = cnt;
  if (cnt > A.K) latch_status(A.status, ST_NEIGH);
}

// floor(x / w), the division only where FP32 leaves it open: one CTA bins a whole
// system, and three FP64 divisions a particle took most of the rebuild.  Within [lo, hi]
// whatever x is: conversions saturate, and f32_bits makes an infinity of a NaN
__device__ __noinline__ int bin_fp64(double x, double w) { return __double2int_rd(x / w); }
__device__ __forceinline__ int bin_of(double x, double w, float winv, int lo, int hi) {
  const float t = f32_bits(x) * winv;  // within 2.5e-7 |t|
  const float b = floorf(t), r = t - b, e = 4e-7f * (fabsf(t) + 1.f);
  return min(max(r < e || r > 1.f - e ? bin_fp64(x, w) : __float2int_rz(b), lo), hi);
}

// a double's order as an integer's (the integer pipe compares 8 times as fast here)
__device__ __forceinline__ long long order_key(double v) {
  const long long b = __double_as_longlong(v);
  return b >= 0 ? b : (b ^ 0x7fffffffffffffffLL);
}

// a bin's positions of the permutation into ascending index, by one warp
__device__ __forceinline__ void sort_bin(int* perm, int n, int lane) {
  if (n <= 64) {
    const int v0 = lane < n ? perm[lane] : 0x7fffffff, v1 = lane + 32 < n ? perm[lane + 32] : 0x7fffffff;
    int r0 = 0, r1 = 0;  // particles before v0, v1
    for (int k = 0; k < min(n, 32); ++k) {
      const int u = __shfl_sync(FULL_MASK, v0, k);
      r0 += u < v0;
      r1 += u < v1;
    }
    for (int k = 32; k < n; ++k) {
      const int u = __shfl_sync(FULL_MASK, v1, k - 32);
      r0 += u < v0;
      r1 += u < v1;
    }
    if (lane < n) perm[r0] = v0;
    if (lane + 32 < n) perm[r1] = v1;
  } else if (lane == 0) {
    for (int k = 1; k < n; ++k) {
      const int v = perm[k];
      int m = k - 1;
      while (m >= 0 && perm[m] > v) {
        perm[m + 1] = perm[m];
        --m;
      }
      perm[m + 1] = v;
    }
  }
}

__device__ void rebuild(const BArgs& A, const BSys& S, int* sh, int* hist) {
  const int tid = threadIdx.x, T = blockDim.x;
  double4_32a* x = A.x + S.base;
  float4* xl = A.xl + S.base;
  int* owner = A.owner + S.base;
  int* img = A.img + S.base;
  int* binof = A.binof + S.base;
  ushort4* binc = A.binc + S.base;
  int* perm = A.perm + S.base;
  int* bstart = A.binstart + S.bin_base;
  const int n = S.n;
  // exchange: wrap owned atoms back into the box (CommSerial::exchange)
  for (int i = tid; i < n; i += T) {
    double4_32a p = x[i];
    double* c = &p.x;
    for (int d = 0; d < 3; ++d) {
      const long long key = order_key(c[d]);
      if (key >= order_key(S.L[d])) c[d] -= S.L[d];
      else if (key < -1) c[d] += S.L[d];  // -1: minus zero
    }
    x[i] = p;
    owner[i] = i;
    img[i] = 0x15;
  }
  __syncthreads();
  // halo: three sweeps, each imaging owned atoms and earlier ghosts within
  // cut_nb of a face of that dimension
  int ng = 0;
  bool over = false;
  for (int d = 0; d < 3; ++d) {
    const int cur = min(n + ng, S.cap);
    // in the lower face's range [-inf, cut_nb), the upper one's [L - cut_nb, inf]: a NaN is in neither
    constexpr long long kinf = 0x7ff0000000000000LL, kninf = -0x7ff0000000000001LL;
    const long long khi = order_key(S.L[d] - A.cut_nb);
    const unsigned long long nlo = order_key(A.cut_nb) - kninf, nhi = kinf - khi;
    // four candidates a thread and scan: a scan's barriers cost more than its sweep
    for (int c0 = 0; c0 < cur; c0 += 4 * T) {
      const int c1 = c0 + 4 * tid;
      int faces = 0;  // bits 2 k and 2 k + 1: candidate c1 + k at the lower, the upper face
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (c1 + k < cur) {
          const long long key = order_key((&x[c1 + k].x)[d]);
          faces |= ((unsigned long long)key - kninf < nlo ? 1 << (2 * k) : 0) |
                   ((unsigned long long)key - khi <= nhi ? 2 << (2 * k) : 0);
        }
      int tot;
      int g = n + ng + block_excl(__popc(faces), sh, tot);
      while (faces) {
        const int bit = __ffs(faces) - 1, c = c1 + (bit >> 1), s = bit & 1;
        faces &= faces - 1;
        if (g >= S.cap) {
          over = true;
          break;
        }
        double4_32a q = x[c];
        double* qc = &q.x;
        qc[d] += s == 0 ? S.L[d] : -S.L[d];
        x[g] = q;
        owner[g] = owner[c];
        img[g] = (img[c] & ~(3 << (2 * d))) | ((s == 0 ? 2 : 0) << (2 * d));
        ++g;
      }
      ng += tot;
    }
    __syncthreads();
  }
  if (over) latch_status(A.status, ST_GHOST);
  ng = min(ng, S.cap - n);
  if (tid == 0) A.nghost[blockIdx.x] = ng;
  const int np = n + ng;
  // binning: counting sort in shared memory, then each bin in ascending index
  const int nbt = (S.nb[0] + 2) * (S.nb[1] + 2) * (S.nb[2] + 2);
  for (int b = tid; b < nbt; b += T) hist[b] = 0;
  __syncthreads();
  const float wi[3] = {float(1.0 / S.w[0]), float(1.0 / S.w[1]), float(1.0 / S.w[2])};
  for (int p = tid; p < np; p += T) {
    const double4_32a q = x[p];
    // owned atoms stay in the interior bins, also one that rounds onto the upper face
    const int o = p < n ? 1 : 0;
    const int bx = bin_of(q.x, S.w[0], wi[0], o - 1, S.nb[0] - o) + 1;
    const int by = bin_of(q.y, S.w[1], wi[1], o - 1, S.nb[1] - o) + 1;
    const int bz = bin_of(q.z, S.w[2], wi[2], o - 1, S.nb[2] - o) + 1;
    const int b = (bx * (S.nb[1] + 2) + by) * (S.nb[2] + 2) + bz;
    binof[p] = b;
    const ushort4 c = make_ushort4(bx, by, bz, img[p]);
    binc[p] = c;
    if (A.nsteps > 0) xl[p] = rel_to_bin(A, S, q, c);  // phased form: BP_REL, on all SMs
    atomicAdd(&hist[b], 1);
  }
  __syncthreads();
  // exclusive scan of the histogram: each thread a contiguous chunk
  const int chunk = (nbt + T - 1) / T;
  const int b0 = min(tid * chunk, nbt), b1 = min(b0 + chunk, nbt);
  int local = 0;
  for (int b = b0; b < b1; ++b) local += hist[b];
  int tot;
  int run = block_excl(local, sh, tot);
  for (int b = b0; b < b1; ++b) {
    const int c = hist[b];
    bstart[b] = run;
    hist[b] = run;  // becomes the scatter cursor
    run += c;
  }
  if (tid == 0) bstart[nbt] = np;
  __syncthreads();
  for (int p = tid; p < np; p += T) perm[atomicAdd(&hist[binof[p]], 1)] = p;
  __syncthreads();
  for (int b = tid >> 5; b < nbt; b += T >> 5) sort_bin(perm + bstart[b], bstart[b + 1] - bstart[b], tid & 31);
  __syncthreads();
  // full neighbour list, one owned atom per thread
  if (A.nsteps > 0)
    for (int i = tid; i < n; i += T) build_row(A, S, i);
  __syncthreads();
}

__device__ __forceinline__ void halo_ghost(const BArgs& A, const BSys& S, int g) {
  double4_32a* x = A.x + S.base;
  double4_32a p = x[A.owner[S.base + g]];
  const ushort4 b = A.binc[S.base + g];
  // most ghosts are images in one dimension, and neighbours in the same one: no FP64
  // addition for the others
  auto shift = [](double& v, int code, double L) {
    if (code != 1) v += code == 2 ? L : -L;
  };
  shift(p.x, b.w & 3, S.L[0]);
  shift(p.y, (b.w >> 2) & 3, S.L[1]);
  shift(p.z, (b.w >> 4) & 3, S.L[2]);
  x[g] = p;
  A.xl[S.base + g] = rel_to_bin(A, S, p, b);
}

__device__ void halo_refresh(const BArgs& A, const BSys& S, int ng) {
  for (int g = S.n + threadIdx.x; g < S.n + ng; g += blockDim.x) halo_ghost(A, S, g);
}

template <bool NC>
__device__ __forceinline__ double3 force_of(const BArgs& A, const BSys& S, int i) {
  const float4* xl = A.xl + S.base;
  const int4* rows4 = reinterpret_cast<const int4*>(A.rows + S.row_base);
  PairCtx C;
  C.xi = xl[i];
  C.i = i;
  C.ti = 0;
  C.set_bin_width(float(S.w[0]), float(S.w[1]), float(S.w[2]));
  C.x4 = A.x + S.base;
  Acc acc;
  lj_row<NC>(i, rows4 + i, min(A.num[S.base + i], A.K), S.n, [&](const int4& e) { lj_quad<true>(C, e, xl, A.P, acc); });
  return make_double3(double(acc.sxy.x) - double(acc.cxy.x), double(acc.sxy.y) - double(acc.cxy.y),
                      double(acc.sz) - double(acc.cz));
}

template <bool NC>
__device__ __forceinline__ void force_atom(const BArgs& A, const BSys& S, int i) {
  const double3 t = force_of<NC>(A, S, i);
  double* f = A.f + 3 * size_t(S.base);
  f[3 * i] = t.x;
  f[3 * i + 1] = t.y;
  f[3 * i + 2] = t.z;
}

__device__ void force(const BArgs& A, const BSys& S) {
  for (int i = threadIdx.x; i < S.n; i += blockDim.x) force_atom<false>(A, S, i);
}

// IntegratorNVE::initial_integrate, with the FP32 bin-relative copy
__device__ __forceinline__ void nve_initial_atom(const BArgs& A, const BSys& S, int i) {
  double* v = A.v + 3 * size_t(S.base);
  const double* f = A.f + 3 * size_t(S.base);
  double4_32a* x = A.x + S.base;
  const double vx = fma(A.dtf, f[3 * i], v[3 * i]);
  const double vy = fma(A.dtf, f[3 * i + 1], v[3 * i + 1]);
  const double vz = fma(A.dtf, f[3 * i + 2], v[3 * i + 2]);
  v[3 * i] = vx;
  v[3 * i + 1] = vy;
  v[3 * i + 2] = vz;
  double4_32a p = x[i];
  p.x = fma(A.dt, vx, p.x);
  p.y = fma(A.dt, vy, p.y);
  p.z = fma(A.dt, vz, p.z);
  x[i] = p;
  A.xl[S.base + i] = rel_to_bin(A, S, p, A.binc[S.base + i]);
}

// IntegratorNVE::final_integrate
__device__ __forceinline__ void nve_final_atom(const BArgs& A, const BSys& S, int i) {
  double* v = A.v + 3 * size_t(S.base);
  const double* f = A.f + 3 * size_t(S.base);
  v[3 * i] = fma(A.dtf, f[3 * i], v[3 * i]);
  v[3 * i + 1] = fma(A.dtf, f[3 * i + 1], v[3 * i + 1]);
  v[3 * i + 2] = fma(A.dtf, f[3 * i + 2], v[3 * i + 2]);
}

// One CTA per system: nsteps timesteps (the persistent form), or with nsteps = 0
// wrap, halo and binning only (the phased form's rebuild).
__global__ void __launch_bounds__(BATCH_MAX_THREADS) k_batch(BArgs A) {
  extern __shared__ int hist[];
  __shared__ int sh[33];
  const BSys S = A.sys[blockIdx.x];
  if (A.nsteps == 0) {
    rebuild(A, S, sh, hist);
    return;
  }
  int ng = A.nghost[blockIdx.x];
  for (int s = 1; s <= A.nsteps; ++s) {
    const int step = A.step0 + s;
    for (int i = threadIdx.x; i < S.n; i += blockDim.x) nve_initial_atom(A, S, i);
    __syncthreads();
    if (step % A.every == 0) {
      rebuild(A, S, sh, hist);
      ng = min(A.nghost[blockIdx.x], S.cap - S.n);
    } else {
      halo_refresh(A, S, ng);
      __syncthreads();
    }
    force(A, S);
    // each thread integrates the atoms it computed the force of
    for (int i = threadIdx.x; i < S.n; i += blockDim.x) nve_final_atom(A, S, i);
    __syncthreads();
  }
}

// Phased form: 128-atom chunks of one system per CTA (chunk table: system,
// first atom; ghosts relative to the first ghost slot), bins for the rows.
constexpr int BP_THREADS = 128;
struct BChunk {
  int sys, first;
};
enum { BP_NVE_INITIAL, BP_HALO, BP_REL, BP_FORCE, BP_STEP, BP_LAST };

template <int PHASE>
__global__ void __launch_bounds__(BP_THREADS) k_batch_phase(BArgs A, const BChunk* __restrict__ chunks) {
  const BChunk ch = chunks[blockIdx.x];
  const BSys& S = A.sys[ch.sys];
  const int k = ch.first + threadIdx.x;
  if (PHASE == BP_REL) {  // owned atoms' chunks, then ghosts'
    const int p = blockIdx.x < A.n_chunks ? k : S.n + k;
    if (p < (blockIdx.x < A.n_chunks ? S.n : S.n + min(A.nghost[ch.sys], S.cap - S.n)))
      A.xl[S.base + p] = rel_to_bin(A, S, A.x[S.base + p], A.binc[S.base + p]);
    return;
  }
  if (PHASE == BP_HALO) {
    const int ng = min(A.nghost[ch.sys], S.cap - S.n);
    if (k < ng) halo_ghost(A, S, S.n + k);
    return;
  }
  if (k >= S.n) return;
  if (PHASE == BP_NVE_INITIAL) {
    nve_initial_atom(A, S, k);
    return;
  }
  if (PHASE == BP_FORCE) {
    force_atom<true>(A, S, k);
    return;
  }
  // force and final half kick; BP_STEP: also the next step's half kick and drift
  const double3 f = force_of<true>(A, S, k);
  double* v = A.v + 3 * size_t(S.base + k);
  double vx = fma(A.dtf, f.x, v[0]), vy = fma(A.dtf, f.y, v[1]), vz = fma(A.dtf, f.z, v[2]);
  if (PHASE == BP_STEP) {
    vx = fma(A.dtf, f.x, vx);
    vy = fma(A.dtf, f.y, vy);
    vz = fma(A.dtf, f.z, vz);
    double4_32a p = A.x[S.base + k];
    p.x = fma(A.dt, vx, p.x);
    p.y = fma(A.dt, vy, p.y);
    p.z = fma(A.dt, vz, p.z);
    A.xn[S.base + k] = p;
    A.xln[S.base + k] = rel_to_bin(A, S, p, A.binc[S.base + k]);
  } else {
    double* fo = A.f + 3 * size_t(S.base + k);
    fo[0] = f.x;
    fo[1] = f.y;
    fo[2] = f.z;
  }
  v[0] = vx;
  v[1] = vy;
  v[2] = vz;
}

// neighbour rows, one warp per interior bin
constexpr int BR_WARPS = 4;
__global__ void __launch_bounds__(32 * BR_WARPS) k_batch_rows(BArgs A, const BChunk* __restrict__ chunks) {
  __shared__ __align__(16) RowStage st[BR_WARPS];
  const BChunk ch = chunks[blockIdx.x];
  const BSys& S = A.sys[ch.sys];
  const int warp = threadIdx.x >> 5, bin = ch.first + warp;
  if (bin >= S.nb[0] * S.nb[1] * S.nb[2]) return;
  RowArgs r;
  r.x4 = A.x + S.base;
  r.xl = A.xl + S.base;
  r.permute = A.perm + S.base;
  r.nby = S.nb[1] + 2;
  r.nbz = S.nb[2] + 2;
  r.wx = float(S.w[0]);
  r.wy = float(S.w[1]);
  r.wz = float(S.w[2]);
  r.n_local = S.n;
  r.newton = 0;
  r.cutsq = A.cutsq_nb;
  r.cut_lo = A.nb_lo;
  r.cut_hi = A.nb_hi;
  r.num_neighs = A.num + S.base;
  r.rows = A.rows + S.row_base;
  r.stride = S.n;
  r.K = A.K;
  const int* bstart = A.binstart + S.bin_base;
  const int mx = rows_of_bin<false, true>(r, st[warp], bin / (S.nb[1] * S.nb[2]) + 1, (bin / S.nb[2]) % S.nb[1] + 1,
                                          bin % S.nb[2] + 1, [&](int b, int& off) {
                                            off = bstart[b];
                                            return bstart[b + 1] - off;
                                          });
  if (mx > A.K && (threadIdx.x & 31) == 0) latch_status(A.status, ST_NEIGH);
}

// owned atoms of a slot array (stride doubles a slot) in the caller's order
__global__ void __launch_bounds__(BP_THREADS) k_batch_pack(BArgs A, const BChunk* __restrict__ chunks,
                                                           const double* __restrict__ src, int stride,
                                                           double* __restrict__ out) {
  const BChunk ch = chunks[blockIdx.x];
  const BSys& S = A.sys[ch.sys];
  const int m = 3 * min(BP_THREADS, S.n - ch.first);
  for (int t = threadIdx.x; t < m; t += BP_THREADS) {
    const int i = t / 3, d = t - 3 * i;
    out[3 * (S.out + ch.first) + t] = src[size_t(S.base + ch.first + i) * stride + d];
  }
}

// per system: sum m v^2 over owned atoms and the shifted LJ energy (FP64,
// full rows, 1/2 per ordered pair), fixed-order block sums
__global__ void __launch_bounds__(256) k_batch_thermo(BArgs A, double mass, double lj1, double lj2,
                                                      double cutsq, double* out) {
  __shared__ double sh[8];
  const BSys S = A.sys[blockIdx.x];
  const double4_32a* x = A.x + S.base;
  const double* v = A.v + 3 * size_t(S.base);
  const int* num = A.num + S.base;
  const int* rows = A.rows + S.row_base;
  const double r2c = 1.0 / cutsq, r6c = r2c * r2c * r2c;
  double mv2 = 0.0, pe = 0.0;
  for (int i = threadIdx.x; i < S.n; i += blockDim.x) {
    mv2 += mass * (v[3 * i] * v[3 * i] + v[3 * i + 1] * v[3 * i + 1] + v[3 * i + 2] * v[3 * i + 2]);
    const double4_32a xi = x[i];
    const int cnt = min(num[i], A.K);
    for (int k = 0; k < cnt; ++k) {
      const int j = rows[quad_index(i, k, S.n)] >> 6;
      const double4_32a xj = x[j];
      const double dx = xi.x - xj.x, dy = xi.y - xj.y, dz = xi.z - xj.z;
      const double rsq = dx * dx + dy * dy + dz * dz;
      if (rsq < cutsq) {
        const double r2inv = 1.0 / rsq, r6inv = r2inv * r2inv * r2inv;
        pe += 0.5 * (r6inv * (lj1 / 12.0 * r6inv - lj2 / 6.0) - r6c * (lj1 / 12.0 * r6c - lj2 / 6.0));
      }
    }
  }
  const double a = block_sum(mv2, sh);
  const double b = block_sum(pe, sh);
  if (threadIdx.x == 0) {
    out[2 * blockIdx.x] = a;
    out[2 * blockIdx.x + 1] = b;
  }
}

}  // namespace
}  // namespace emd

using namespace emd;

struct emd_batch {
  int device = 0;
  cudaStream_t stream = nullptr;
  std::string last_error;
  unsigned* d_status = nullptr;
  int nsys = 0;
  long long atoms = 0;
  std::vector<int> order;       // device slot -> caller's system index (largest first)
  std::vector<int> natoms;      // caller's order
  std::vector<long long> in_off;  // caller's atom offsets
  std::vector<BSys> sys;        // device order
  BSys* d_sys = nullptr;
  DevBuf<double4_32a> x, x2;  // a.x is one of the two
  DevBuf<float4> xl, xl2;
  DevBuf<double> v, f, thermo, mid, pack;
  DevBuf<ushort4> binc;
  DevBuf<int> owner, img, binof, perm, binstart, num, rows, nghost;
  BArgs a{};
  double mass = 1.0, lj1 = 0, lj2 = 0, cutsq = 0;
  int threads = 512, steps_per_launch = 20;
  size_t smem = 0;
  long long steps_done = 0;
  size_t slots = 0;  // particle slots over all systems (owned + ghost capacity)
  // phased form: chunk tables of the owned atoms, of the ghost capacity and of the bins
  bool phased = false;
  BChunk* d_chunks = nullptr;  // the ghosts' behind the owned atoms'
  BChunk* d_bchunks = nullptr;
  int n_chunks = 0, n_gchunks = 0, n_bchunks = 0;
};

namespace {

#define BATCH_BEGIN            \
  if (!b) return EMD_ERR_ARG; \
  try {
#define BATCH_END                   \
  }                                 \
  catch (const ::emd::Error& e) {   \
    b->last_error = e.what();       \
    return e.code;                  \
  }                                 \
  catch (const std::exception& e) { \
    b->last_error = e.what();       \
    return EMD_ERR_CUDA;            \
  }                                 \
  return EMD_OK;

void batch_check(emd_batch* b) {
  unsigned st = 0;
  EMD_CUDA(cudaMemcpyAsync(&st, b->d_status, sizeof(unsigned), cudaMemcpyDeviceToHost, b->stream));
  EMD_CUDA(cudaStreamSynchronize(b->stream));
  if (st & ST_GHOST) throw Error(EMD_ERR_OVERFLOW_GHOST, "batch: ghost capacity exceeded (raise ghost_factor)");
  if (st & ST_NEIGH) throw Error(EMD_ERR_OVERFLOW_NEIGH, "batch: neighbour row capacity exceeded (raise max_neigh)");
  if (st) throw Error(EMD_ERR_BOUNDS, "batch: device status " + std::to_string(st));
}

// nsteps timesteps, or (nsteps == 0) wrap, halo and binning
void batch_launch(emd_batch* b, int step0, int nsteps, int threads) {
  BArgs a = b->a;
  a.step0 = step0;
  a.nsteps = nsteps;
  k_batch<<<b->nsys, threads, b->smem, b->stream>>>(a);
  EMD_CHECK_LAUNCH();
}

template <int PHASE>
void batch_phase(emd_batch* b) {
  const bool ghosts = PHASE == BP_HALO;
  const int blocks = PHASE == BP_REL ? b->n_chunks + b->n_gchunks : (ghosts ? b->n_gchunks : b->n_chunks);
  k_batch_phase<PHASE><<<blocks, BP_THREADS, 0, b->stream>>>(b->a, b->d_chunks + (ghosts ? b->n_chunks : 0));
  EMD_CHECK_LAUNCH();
}

void batch_rebuild(emd_batch* b, int threads) {
  batch_launch(b, 0, 0, threads);
  batch_phase<BP_REL>(b);
  k_batch_rows<<<b->n_bchunks, 32 * BR_WARPS, 0, b->stream>>>(b->a, b->d_bchunks);
  EMD_CHECK_LAUNCH();
}

// one timestep of the phased form; the drift to the next one is part of it
void batch_phased_step(emd_batch* b, long long step, int threads, bool last) {
  if (step % b->a.every == 0) {
    batch_rebuild(b, threads);
  } else {
    batch_phase<BP_HALO>(b);
  }
  if (last) return batch_phase<BP_LAST>(b);
  batch_phase<BP_STEP>(b);
  std::swap(b->a.x, b->a.xn);
  std::swap(b->a.xl, b->a.xln);
}

// f() unless device memory is short
template <typename F>
bool batch_fits(F&& f) {
  try {
    f();
  } catch (const Error& e) {
    if (e.code != EMD_ERR_NOMEM) throw;
    return false;
  }
  return true;
}

// runs nsteps in one CUDA graph: ceil(nsteps / spl) persistent launches, or
// the phased form's launches per step; without room for its second set of buffers
// the persistent form, which gives the same bits
void batch_run(emd_batch* b, int nsteps, int threads, int spl, bool phased) {
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  const BArgs before = b->a;
  if (phased && !batch_fits([&] {
        b->x2.reserve(b->slots, b->stream);
        b->xl2.reserve(b->slots, b->stream);
      })) {
    b->x2.release();  // not in use: the buffers have not changed places yet
    phased = false;
  }
  if (phased) {
    b->a.xn = b->a.x == b->x.p ? b->x2.p : b->x.p;
    b->a.xln = b->a.xl == b->xl.p ? b->xl2.p : b->xl.p;
  }
  auto clean = [&] {
    if (exec) cudaGraphExecDestroy(exec);
    if (graph) cudaGraphDestroy(graph);
  };
  EMD_CUDA(cudaStreamBeginCapture(b->stream, cudaStreamCaptureModeThreadLocal));
  bool capturing = true;
  try {
    if (phased) {
      batch_phase<BP_NVE_INITIAL>(b);
      for (int s = 1; s <= nsteps; ++s) batch_phased_step(b, b->steps_done + s, threads, s == nsteps);
    } else {
      for (int s = 0; s < nsteps; s += spl)
        batch_launch(b, int(b->steps_done + s), std::min(spl, nsteps - s), threads);
    }
    capturing = false;
    EMD_CUDA(cudaStreamEndCapture(b->stream, &graph));
    EMD_CUDA(cudaGraphInstantiate(&exec, graph, 0));
    EMD_CUDA(cudaGraphLaunch(exec, b->stream));
  } catch (...) {
    if (capturing) cudaStreamEndCapture(b->stream, &graph);
    clean();
    b->a = before;  // nothing has run: the buffers did not change places
    throw;
  }
  clean();
  b->steps_done += nsteps;
}

}  // namespace

extern "C" {

emd_status emd_batch_create(emd_batch** out, int device, int nsys, const int* natoms, const double* boxes,
                            const double* x, const double* v, double mass, double dt, double eps, double sigma,
                            double cut, double skin, int every, int max_neigh, double ghost_factor) {
  if (!out) return EMD_ERR_ARG;
  *out = nullptr;
  emd_batch* b = new emd_batch();
  BATCH_BEGIN
  require(nsys >= 1 && natoms && boxes && x && v, EMD_ERR_ARG, "emd_batch_create: arguments");
  require(mass > 0 && dt > 0 && eps > 0 && sigma > 0 && cut > 0 && skin >= 0 && every >= 1, EMD_ERR_ARG,
          "emd_batch_create: parameters");
  require(max_neigh >= 4 && ghost_factor >= 1.0, EMD_ERR_ARG, "emd_batch_create: capacities");
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || device < 0 || device >= ndev) {
    (void)cudaGetLastError();
    throw Error(EMD_ERR_CUDA, "emd_batch_create: no CUDA device " + std::to_string(device));
  }
  EMD_CUDA(cudaSetDevice(device));
  b->device = device;
  EMD_CUDA(cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking));
  EMD_CUDA(device_malloc(reinterpret_cast<void**>(&b->d_status), sizeof(unsigned)));
  EMD_CUDA(cudaMemsetAsync(b->d_status, 0, sizeof(unsigned), b->stream));
  b->nsys = nsys;
  b->mass = mass;
  const double cut_nb = cut + skin;
  const int K = (max_neigh + 3) & ~3;
  b->natoms.assign(natoms, natoms + nsys);
  b->in_off.assign(size_t(nsys) + 1, 0);
  for (int k = 0; k < nsys; ++k) {
    require(natoms[k] >= 1, EMD_ERR_ARG, "emd_batch_create: empty system");
    b->in_off[size_t(k) + 1] = b->in_off[size_t(k)] + natoms[k];
  }
  b->atoms = b->in_off[size_t(nsys)];
  require(b->atoms < (1LL << 31), EMD_ERR_ARG, "emd_batch_create: too many atoms");
  b->order.resize(size_t(nsys));
  std::iota(b->order.begin(), b->order.end(), 0);
  std::stable_sort(b->order.begin(), b->order.end(), [&](int p, int q) { return natoms[p] > natoms[q]; });
  long long slot = 0, bins = 0, rows = 0;
  int max_bins = 0, max_dim = 0;
  double max_w = 0.0;
  for (int s = 0; s < nsys; ++s) {
    const int k = b->order[size_t(s)];
    BSys S{};
    double vol = 1.0, outer = 1.0;
    for (int d = 0; d < 3; ++d) {
      S.L[d] = boxes[3 * k + d];
      require(S.L[d] > 2.0 * cut_nb, EMD_ERR_ARG, "emd_batch_create: every box edge must exceed 2 (cut + skin)");
      S.nb[d] = std::max(1, int(std::floor(S.L[d] / cut_nb)));
      S.w[d] = S.L[d] / S.nb[d];
      max_dim = std::max(max_dim, S.nb[d] + 2);
      max_w = std::max(max_w, S.w[d]);
      vol *= S.L[d];
      outer *= S.L[d] + 2.0 * cut_nb;
    }
    S.n = natoms[k];
    const int gcap = int(std::ceil(ghost_factor * S.n * (outer / vol - 1.0))) + 64;
    S.base = int(slot);
    S.out = b->in_off[size_t(k)];
    S.cap = S.n + gcap;
    S.bin_base = int(bins);
    S.row_base = rows;
    const int nbt = (S.nb[0] + 2) * (S.nb[1] + 2) * (S.nb[2] + 2);
    max_bins = std::max(max_bins, nbt);
    slot += S.cap;
    bins += nbt + 1;
    rows += (long long)S.n * K;
    b->sys.push_back(S);
  }
  require(slot < (1LL << 25), EMD_ERR_ARG, "emd_batch_create: packed rows need fewer than 2^25 slots per system");
  b->smem = sizeof(int) * size_t(max_bins);
  require(b->smem <= 200 * 1024, EMD_ERR_ARG, "emd_batch_create: a system's bin grid exceeds shared memory");
  allow_dyn_smem(k_batch);
  const size_t ns = size_t(slot);
  b->slots = ns;
  b->x.reserve(ns, b->stream);
  b->xl.reserve(ns, b->stream);
  b->v.reserve(3 * ns, b->stream);
  b->f.reserve(3 * ns, b->stream);
  b->owner.reserve(ns, b->stream);
  b->img.reserve(ns, b->stream);
  b->binof.reserve(ns, b->stream);
  b->binc.reserve(ns, b->stream);
  b->perm.reserve(ns, b->stream);
  b->num.reserve(ns, b->stream);
  b->binstart.reserve(size_t(bins), b->stream);
  b->rows.reserve(size_t(rows), b->stream);
  b->nghost.reserve(size_t(nsys), b->stream);
  b->thermo.reserve(2 * size_t(nsys), b->stream);
  EMD_CUDA(device_malloc(reinterpret_cast<void**>(&b->d_sys), sizeof(BSys) * size_t(nsys)));
  EMD_CUDA(cudaMemcpyAsync(b->d_sys, b->sys.data(), sizeof(BSys) * size_t(nsys), cudaMemcpyHostToDevice, b->stream));
  {
    std::vector<double> mid;
    for (int k = 0; k < max_dim; ++k) mid.push_back(k - 0.5);
    b->mid.reserve(mid.size(), b->stream);
    EMD_CUDA(cudaMemcpyAsync(b->mid.p, mid.data(), sizeof(double) * mid.size(), cudaMemcpyHostToDevice, b->stream));
    std::vector<BChunk> ch, gch, bch;
    for (int s = 0; s < nsys; ++s) {
      const BSys& S = b->sys[size_t(s)];
      for (int f0 = 0; f0 < S.n; f0 += BP_THREADS) ch.push_back(BChunk{s, f0});
      for (int f0 = 0; f0 < S.cap - S.n; f0 += BP_THREADS) gch.push_back(BChunk{s, f0});
      for (int f0 = 0; f0 < S.nb[0] * S.nb[1] * S.nb[2]; f0 += BR_WARPS) bch.push_back(BChunk{s, f0});
    }
    b->n_chunks = int(ch.size());
    b->n_gchunks = int(gch.size());
    b->n_bchunks = int(bch.size());
    EMD_CUDA(device_malloc(reinterpret_cast<void**>(&b->d_bchunks), sizeof(BChunk) * bch.size()));
    EMD_CUDA(cudaMemcpyAsync(b->d_bchunks, bch.data(), sizeof(BChunk) * bch.size(), cudaMemcpyHostToDevice,
                             b->stream));
    ch.insert(ch.end(), gch.begin(), gch.end());
    EMD_CUDA(device_malloc(reinterpret_cast<void**>(&b->d_chunks), sizeof(BChunk) * ch.size()));
    EMD_CUDA(cudaMemcpyAsync(b->d_chunks, ch.data(), sizeof(BChunk) * ch.size(), cudaMemcpyHostToDevice, b->stream));
    EMD_CUDA(cudaStreamSynchronize(b->stream));
  }
  // positions / velocities into the device slots (owned atoms keep the caller's order)
  std::vector<double4_32a> hx(ns, make_double4_32a(0, 0, 0, 0));
  std::vector<double> hv(3 * ns, 0.0);
  for (int s = 0; s < nsys; ++s) {
    const int k = b->order[size_t(s)];
    const BSys& S = b->sys[size_t(s)];
    for (int i = 0; i < S.n; ++i) {
      const long long src = b->in_off[size_t(k)] + i;
      hx[size_t(S.base + i)] = make_double4_32a(x[3 * src], x[3 * src + 1], x[3 * src + 2], 0.0);
      for (int d = 0; d < 3; ++d) hv[3 * size_t(S.base + i) + d] = v[3 * src + d];
    }
  }
  EMD_CUDA(cudaMemcpyAsync(b->x.p, hx.data(), sizeof(double4_32a) * ns, cudaMemcpyHostToDevice, b->stream));
  EMD_CUDA(cudaMemcpyAsync(b->v.p, hv.data(), sizeof(double) * 3 * ns, cudaMemcpyHostToDevice, b->stream));
  EMD_CUDA(cudaMemsetAsync(b->f.p, 0, sizeof(double) * 3 * ns, b->stream));
  EMD_CUDA(cudaMemsetAsync(b->nghost.p, 0, sizeof(int) * size_t(nsys), b->stream));
  // parameters
  BArgs& a = b->a;
  a.sys = b->d_sys;
  a.x = b->x.p;
  a.xl = b->xl.p;
  a.v = b->v.p;
  a.f = b->f.p;
  a.owner = b->owner.p;
  a.img = b->img.p;
  a.binof = b->binof.p;
  a.binc = b->binc.p;
  a.mid = b->mid.p;
  a.perm = b->perm.p;
  a.binstart = b->binstart.p;
  a.num = b->num.p;
  a.rows = b->rows.p;
  a.nghost = b->nghost.p;
  a.status = b->d_status;
  a.K = K;
  a.dt = dt;
  a.dtf = 0.5 * dt / mass;
  a.cut_nb = cut_nb;
  a.cutsq_nb = cut_nb * cut_nb;
  const double band = row_band(max_w, cut_nb);
  a.nb_lo = float(a.cutsq_nb * (1.0 - band));
  a.nb_hi = float(a.cutsq_nb * (1.0 + band));
  b->lj1 = 48.0 * eps * std::pow(sigma, 12.0);
  b->lj2 = 24.0 * eps * std::pow(sigma, 6.0);
  b->cutsq = cut * cut;
  a.P = LJParamsF{nullptr, nullptr, nullptr, nullptr, 1, float(b->lj1), float(b->lj2), float(b->cutsq), b->cutsq};
  a.every = every;
  a.n_chunks = b->n_chunks;
  // initial halo, binning, list and forces
  cudaDeviceProp prop{};
  EMD_CUDA(cudaGetDeviceProperties(&prop, device));
  b->threads = 512;
  batch_rebuild(b, b->threads);
  batch_phase<BP_FORCE>(b);
  batch_check(b);
  *out = b;
  return EMD_OK;
  }
  catch (const ::emd::Error& e) {
    std::fprintf(stderr, "emd_batch_create: %s\n", e.what());
    emd_batch_destroy(b);
    return e.code;
  }
  catch (const std::exception& e) {
    std::fprintf(stderr, "emd_batch_create: %s\n", e.what());
    emd_batch_destroy(b);
    return EMD_ERR_CUDA;
  }
}

void emd_batch_destroy(emd_batch* b) {
  if (!b) return;
  if (b->stream) cudaStreamSynchronize(b->stream);
  for (auto* p : {&b->owner, &b->img, &b->binof, &b->perm, &b->binstart, &b->num, &b->rows, &b->nghost}) p->release();
  b->x.release();
  b->xl.release();
  b->x2.release();
  b->xl2.release();
  b->mid.release();
  b->pack.release();
  b->binc.release();
  b->v.release();
  b->f.release();
  b->thermo.release();
  if (b->d_sys) cudaFree(b->d_sys);
  if (b->d_chunks) cudaFree(b->d_chunks);
  if (b->d_bchunks) cudaFree(b->d_bchunks);
  if (b->d_status) cudaFree(b->d_status);
  if (b->stream) cudaStreamDestroy(b->stream);
  delete b;
}

const char* emd_batch_last_error(const emd_batch* b) { return b ? b->last_error.c_str() : "null batch"; }

emd_status emd_batch_run(emd_batch* b, int nsteps) {
  BATCH_BEGIN
  const DeviceGuard device(b->device);
  require(nsteps >= 0, EMD_ERR_ARG, "emd_batch_run: nsteps");
  if (nsteps == 0) return EMD_OK;
  batch_run(b, nsteps, b->threads, b->steps_per_launch, b->phased);
  batch_check(b);
  BATCH_END
}

emd_status emd_batch_set_shape(emd_batch* b, int threads, int steps_per_launch) {
  BATCH_BEGIN
  require(threads >= 64 && threads <= BATCH_MAX_THREADS && threads % 32 == 0, EMD_ERR_ARG,
          "emd_batch_set_shape: threads must be a multiple of 32 in [64, 1024]");
  require(steps_per_launch >= 0, EMD_ERR_ARG, "emd_batch_set_shape: steps_per_launch");
  b->threads = threads;
  b->phased = steps_per_launch == 0;
  if (!b->phased) b->steps_per_launch = steps_per_launch;
  BATCH_END
}

emd_status emd_batch_tune(emd_batch* b, int trial_steps, int* threads_out, int* spl_out) {
  BATCH_BEGIN
  const DeviceGuard device(b->device);
  require(trial_steps >= 1, EMD_ERR_ARG, "emd_batch_tune: trial_steps");
  // every candidate runs the same trial from the same state, which is then restored
  const size_t ns = b->slots;
  DevBuf<double4_32a> x0;
  DevBuf<double> v0, f0;
  x0.reserve(ns, b->stream);
  v0.reserve(3 * ns, b->stream);
  f0.reserve(3 * ns, b->stream);
  EMD_CUDA(cudaMemcpyAsync(x0.p, b->a.x, sizeof(double4_32a) * ns, cudaMemcpyDeviceToDevice, b->stream));
  EMD_CUDA(cudaMemcpyAsync(v0.p, b->v.p, sizeof(double) * 3 * ns, cudaMemcpyDeviceToDevice, b->stream));
  EMD_CUDA(cudaMemcpyAsync(f0.p, b->f.p, sizeof(double) * 3 * ns, cudaMemcpyDeviceToDevice, b->stream));
  const long long saved_steps = b->steps_done;
  cudaEvent_t e0, e1;
  EMD_CUDA(cudaEventCreate(&e0));
  EMD_CUDA(cudaEventCreate(&e1));
  float best = 1e30f;
  int bt = b->threads, bs = b->steps_per_launch;
  bool bp = b->phased;
  const int every = b->a.every;
  for (int threads : {256, 512, 1024}) {
    // steps per launch; 0 = the phased form (its per-system rebuild on `threads`)
    for (int spl : {0, every, 5 * every, trial_steps}) {
      if (spl > trial_steps) continue;
      // state of the trial's start (a rebuild step boundary)
      EMD_CUDA(cudaMemcpyAsync(b->a.x, x0.p, sizeof(double4_32a) * ns, cudaMemcpyDeviceToDevice, b->stream));
      EMD_CUDA(cudaMemcpyAsync(b->v.p, v0.p, sizeof(double) * 3 * ns, cudaMemcpyDeviceToDevice, b->stream));
      EMD_CUDA(cudaMemcpyAsync(b->f.p, f0.p, sizeof(double) * 3 * ns, cudaMemcpyDeviceToDevice, b->stream));
      b->steps_done = saved_steps;
      batch_rebuild(b, threads);  // from the restored positions
      batch_phase<BP_FORCE>(b);
      EMD_CUDA(cudaEventRecord(e0, b->stream));
      batch_run(b, trial_steps, threads, std::max(spl, 1), spl == 0);
      EMD_CUDA(cudaEventRecord(e1, b->stream));
      EMD_CUDA(cudaEventSynchronize(e1));
      float ms = 0.f;
      EMD_CUDA(cudaEventElapsedTime(&ms, e0, e1));
      if (ms < best) {
        best = ms;
        bt = threads;
        bp = spl == 0;
        if (!bp) bs = spl;
      }
    }
  }
  EMD_CUDA(cudaMemcpyAsync(b->a.x, x0.p, sizeof(double4_32a) * ns, cudaMemcpyDeviceToDevice, b->stream));
  EMD_CUDA(cudaMemcpyAsync(b->v.p, v0.p, sizeof(double) * 3 * ns, cudaMemcpyDeviceToDevice, b->stream));
  EMD_CUDA(cudaMemcpyAsync(b->f.p, f0.p, sizeof(double) * 3 * ns, cudaMemcpyDeviceToDevice, b->stream));
  b->steps_done = saved_steps;
  batch_rebuild(b, bt);
  batch_phase<BP_FORCE>(b);
  batch_check(b);
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  x0.release();
  v0.release();
  f0.release();
  b->threads = bt;
  b->steps_per_launch = bs;
  b->phased = bp;
  if (threads_out) *threads_out = bt;
  if (spl_out) *spl_out = bp ? 0 : bs;
  BATCH_END
}

// The slots also hold ghosts, in the device's order of systems: packed on the
// device, a third of the bytes goes over the link and nothing is moved on the
// host (1.36 million atoms: 23.7 ms with the slots copied, 4.4 packed).  One system is
// copied as it lies (256 atoms: 53 us packed, 38 so).
emd_status emd_batch_get(emd_batch* b, double* x, double* v, double* f) {
  BATCH_BEGIN
  const DeviceGuard device(b->device);
  const size_t n3 = 3 * size_t(b->atoms);
  const bool pack = b->nsys > 1 && batch_fits([&] { b->pack.reserve(n3, b->stream); });
  auto get = [&](double* out, const double* src, int stride) {
    if (!out) return;
    if (!pack) {  // system by system
      for (const BSys& S : b->sys)
        if (stride == 3)
          EMD_CUDA(cudaMemcpyAsync(out + 3 * S.out, src + 3 * size_t(S.base), sizeof(double) * 3 * size_t(S.n),
                                   cudaMemcpyDeviceToHost, b->stream));
        else
          EMD_CUDA(cudaMemcpy2DAsync(out + 3 * S.out, 3 * sizeof(double), src + size_t(S.base) * stride,
                                   stride * sizeof(double), 3 * sizeof(double), size_t(S.n), cudaMemcpyDeviceToHost,
                                   b->stream));
      return;
    }
    k_batch_pack<<<b->n_chunks, BP_THREADS, 0, b->stream>>>(b->a, b->d_chunks, src, stride, b->pack.p);
    EMD_CHECK_LAUNCH();
    EMD_CUDA(cudaMemcpyAsync(out, b->pack.p, sizeof(double) * n3, cudaMemcpyDeviceToHost, b->stream));
  };
  get(x, &b->a.x->x, 4);
  get(v, b->v.p, 3);
  get(f, b->f.p, 3);
  EMD_CUDA(cudaStreamSynchronize(b->stream));
  BATCH_END
}

emd_status emd_batch_thermo(emd_batch* b, double* mv2, double* pe) {
  BATCH_BEGIN
  const DeviceGuard device(b->device);
  k_batch_thermo<<<b->nsys, 256, 0, b->stream>>>(b->a, b->mass, b->lj1, b->lj2, b->cutsq, b->thermo.p);
  EMD_CHECK_LAUNCH();
  std::vector<double> h(2 * size_t(b->nsys));
  EMD_CUDA(cudaMemcpyAsync(h.data(), b->thermo.p, sizeof(double) * h.size(), cudaMemcpyDeviceToHost, b->stream));
  EMD_CUDA(cudaStreamSynchronize(b->stream));
  for (int s = 0; s < b->nsys; ++s) {
    const int k = b->order[size_t(s)];
    if (mv2) mv2[k] = h[2 * size_t(s)];
    if (pe) pe[k] = h[2 * size_t(s) + 1];
  }
  BATCH_END
}

emd_status emd_batch_info(emd_batch* b, long long* atoms, int* threads, int* steps_per_launch, long long* steps_done) {
  BATCH_BEGIN
  if (atoms) *atoms = b->atoms;
  if (threads) *threads = b->threads;
  if (steps_per_launch) *steps_per_launch = b->phased ? 0 : b->steps_per_launch;
  if (steps_done) *steps_done = b->steps_done;
  BATCH_END
}

void* emd_batch_stream(emd_batch* b) { return b ? static_cast<void*>(b->stream) : nullptr; }

}  // extern "C"
