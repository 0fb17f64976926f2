// FP64 Lennard-Jones over a tile of rows per warp: force (full and half list)
// and energy (force_lj_neigh_impl.h:164-343).
//
// Bound by the FP64 pipe: with all four schedulers busy an SM of this part
// issues one FP64 warp instruction per 19 cycles, a scheduler one per 64 to 76
// whether or not it depends on the last (measured), so only the instruction
// count and the lanes in use matter, and four busy warps per SM fill the pipe.
// The layout keeps every FP64 lane busy and spends none on a pair that does
// not interact:
//   1. filter: 32 lanes read one row's entries, form r^2 in FP32 from the
//      positions' bits (integer conversions: the FP64 pipe is not touched) and
//      append the neighbours that may lie inside the cutoff to the warp's
//      shared list, in row order (ballot + popc);
//   2. pairs: the lanes take list slots 32 at a time, whatever row they belong
//      to, and evaluate them in FP64 with the reference's operations.  The
//      reciprocal starts from an FP32 seed (recip_rn, correctly rounded);
//   3. sums: lane (row, component) adds its row's slots in row order, so each
//      force component is the serial reference's sum, bit for bit (slots that
//      turn out beyond the cutoff hold +0.0, which changes no sum).
// A thread per row spent about 32 FP64 instructions on each of the 75 listed
// pairs (the divide, the type conversion and the test included), 3.75 ms for
// 905,728 atoms; this spends 22 on each of the 55 interacting ones and 9 per
// row for the sums, 2.6 ms (2.6 at the issue rate above).  864 atoms: 0.10 ->
// 0.014 ms, the rows spread over 432 warps instead of 27.
#pragma once
#include <type_traits>

#include "emd_device.cuh"
#include "neigh_rows.cuh"

namespace emd {
namespace {

struct LJParams {
  const double* lj1;
  const double* lj2;
  const double* cutsq;
  int ntypes;
  const double* intensity;  // lj/cut/idial: repeat count per type pair (as doubles)
  const int* type;          // per particle, read when the type pairs differ
  double lj1_0, lj2_0, cutsq_0;  // the values when every type pair shares them
  double cutsq_max;
};

// pair force over r: the plain LJ term, or (IDIAL) ForceLJIDialNeigh's
// repeated evaluation, each repeat adding 1/intensity of the term
// (force_lj_idial_neigh_impl.h:137-149)
template <bool IDIAL>
__device__ __forceinline__ double lj_fpair(double rsq, double lj1, double lj2, double inten) {
  if (!IDIAL) {
    const double r2inv = recip_rn(rsq);
    const double r6inv = r2inv * r2inv * r2inv;
    return (r6inv * (lj1 * r6inv - lj2)) * r2inv;
  }
  double fpair = 0.0;
  for (int repeat = 0; repeat < inten; repeat++) {
    const double r2inv = 1.0 / rsq;
    const double r6inv = r2inv * r2inv * r2inv;
    fpair += (r6inv * (lj1 * r6inv - lj2)) * r2inv / inten;
  }
  return fpair;
}

enum { LJ_FULL = 0, LJ_HALF = 1, LJ_ENERGY = 2 };
constexpr int LJT_WARPS = 4;
constexpr int LJT_THREADS = 32 * LJT_WARPS;
constexpr int LJT_ROWS = 9;  // most rows per warp (lj_tile_rows picks their number)

// slots of a warp's list for `rows` rows (about 55 interacting neighbours each
// at liquid density, half of them in a half list; a fuller list is emptied in
// between), a multiple of 16.  A slot is a position or force, the row's number
// (with the partner's type where the pairs differ) and, for a half list, the
// partner's index.
__host__ __device__ constexpr int ljt_cap(int rows, bool half) { return ((half ? 28 : 56) * rows + 40 + 15) & ~15; }
__host__ __device__ constexpr size_t ljt_warp_bytes(int cap, bool half, bool uni) {
  return size_t(cap) * (24 + (half ? 4 : 0) + (uni ? 1 : 4)) + size_t(LJT_ROWS) * 24 + 8;
}

struct LJTile {
  const double4_32a* x4;
  double* f;
  ListView L;
  LJParams P;
  int n, rows, cap;  // owned atoms, rows per warp, slots of its list
  int half;        // the list is a half list
  int packed;      // entries are (j << 6) | code
  int longest;     // longest row
  double* part;    // energy: one partial per CTA
};

// UNI: one parameter set for every type pair
template <int MODE, bool UNI, bool IDIAL, bool ZERO>
__global__ void __launch_bounds__(LJT_THREADS) k_lj_fp64(LJTile T) {
  extern __shared__ __align__(16) unsigned char ljt_smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int cap = T.cap;
  unsigned char* base = ljt_smem + size_t(warp) * ljt_warp_bytes(cap, T.half, UNI);
  double* sx = reinterpret_cast<double*>(base);  // slot: position of j, then the pair force
  double* sy = sx + cap;
  double* sz = sy + cap;
  double* xi_s = sz + cap;                        // rows x 3
  int* sj = reinterpret_cast<int*>(xi_s + 3 * LJT_ROWS);  // slot: j (half lists)
  using Tag = std::conditional_t<UNI, unsigned char, int>;
  Tag* sa = reinterpret_cast<Tag*>(sj + (T.half ? cap : 0));  // slot: row (| type of j << 4)
  const unsigned lt = (1u << lane) - 1u;
  const int row_l = lane / 3, comp_l = lane - 3 * row_l;  // this lane's sum
  const double lj1_0 = T.P.lj1_0, lj2_0 = T.P.lj2_0, cutsq_0 = T.P.cutsq_0;
  // r^2 < cutsq for non-negative r^2 as an unsigned comparison of the bits (a
  // NaN compares above every cutoff)
  const unsigned long long cbits = cutsq_0 > 0.0 ? static_cast<unsigned long long>(__double_as_longlong(cutsq_0)) : 0ull;
  // shifted energy of the shared type pair: c12 r^-12 - c6 r^-6 - ecut
  double c12_0 = 0.0, c6_0 = 0.0, ecut_0 = 0.0;
  if constexpr (MODE == LJ_ENERGY && UNI) {
    const double r2c = 1.0 / cutsq_0, r6c = r2c * r2c * r2c;
    c12_0 = lj1_0 / 12.0;
    c6_0 = lj2_0 / 6.0;
    ecut_0 = r6c * (c12_0 * r6c - c6_0);
  }
  const float cutsq_f = __double2float_ru(T.P.cutsq_max);
  const int tiles = (T.n + T.rows - 1) / T.rows;
  double esum = 0.0;
  const int step = MODE == LJ_ENERGY ? gridDim.x * LJT_WARPS : tiles;
  for (int tile = blockIdx.x * LJT_WARPS + warp; tile < tiles; tile += step) {
    const int i0 = tile * T.rows, nrow = min(T.rows, T.n - i0);
    double acc = 0.0;             // the sum of (row_l, comp_l)
    int seg_b = 0, seg_e = 0;     // its slots in the list
    int cnt = 0;
    // pairs and sums of the listed slots
    auto flush = [&]() {
      __syncwarp();
      for (int k = lane; k < cnt; k += 32) {
        const int tag = sa[k];
        const int a = tag & 15;
        const double dx = xi_s[3 * a] - sx[k], dy = xi_s[3 * a + 1] - sy[k], dz = xi_s[3 * a + 2] - sz[k];
        const double rsq = dx * dx + dy * dy + dz * dz;
        double lj1 = lj1_0, lj2 = lj2_0, cutsq = cutsq_0, inten = 1.0;
        bool in;
        if constexpr (UNI) {
          in = static_cast<unsigned long long>(__double_as_longlong(rsq)) < cbits;
          if constexpr (IDIAL) inten = __ldg(T.P.intensity);
        } else {
          const int tp = __ldg(T.P.type + i0 + a) * T.P.ntypes + (tag >> 4);
          lj1 = __ldg(T.P.lj1 + tp);
          lj2 = __ldg(T.P.lj2 + tp);
          cutsq = __ldg(T.P.cutsq + tp);
          in = rsq < cutsq;
          if constexpr (IDIAL) inten = __ldg(T.P.intensity + tp);
        }
        if constexpr (MODE == LJ_ENERGY) {
          if (in) {
            // shifted energy (force_lj_neigh_impl.h:259-343), weight 1/2 per
            // listed pair of a full list, 1 (owned j) or 1/2 of a half list
            const double r2inv = recip_rn(rsq), r6inv = r2inv * r2inv * r2inv;
            double c12 = c12_0, c6 = c6_0, ecut = ecut_0;
            if constexpr (!UNI) {
              const double r2c = 1.0 / cutsq, r6c = r2c * r2c * r2c;
              c12 = lj1 / 12.0;
              c6 = lj2 / 6.0;
              ecut = r6c * (c12 * r6c - c6);
            }
            esum += (T.half && sj[k] < T.n ? 1.0 : 0.5) * (r6inv * (c12 * r6inv - c6) - ecut);
          }
        } else {
          double fx = 0.0, fy = 0.0, fz = 0.0;
          if (in) {
            const double fpair = lj_fpair<IDIAL>(rsq, lj1, lj2, inten);
            fx = dx * fpair;
            fy = dy * fpair;
            fz = dz * fpair;
            if constexpr (MODE == LJ_HALF) {
              const int j = sj[k];
              // ForceLJIDialNeigh's half form scatters to owned partners only
              // (force_lj_idial_neigh_impl.h:199-203)
              if (!IDIAL || j < T.n) {
                double* fj = T.f + 3 * size_t(j);
                atomicAdd(fj, -fx);
                atomicAdd(fj + 1, -fy);
                atomicAdd(fj + 2, -fz);
              }
            }
          }
          sx[k] = fx;
          sy[k] = fy;
          sz[k] = fz;
        }
      }
      __syncwarp();
      if constexpr (MODE != LJ_ENERGY) {
        const double* s = sx + size_t(comp_l) * cap;
#pragma unroll 4
        for (int k = seg_b; k < seg_e; ++k) acc += s[k];
        seg_b = seg_e = 0;
        __syncwarp();
      }
      cnt = 0;
    };
    // row a on lane a: its length, its place in the list and its position
    int len_l = 0;
    size_t off_l = 0;
    double4_32a xl = make_double4_32a(0.0, 0.0, 0.0, 0.0);
    if (lane < nrow) {
      const Row row(T.L, i0 + lane);
      len_l = row.n;
      off_l = size_t(row.p - T.L.entries);
      xl = T.x4[i0 + lane];
      xi_s[3 * lane] = xl.x;
      xi_s[3 * lane + 1] = xl.y;
      xi_s[3 * lane + 2] = xl.z;
    }
    const float xf_l = f32_bits(xl.x), yf_l = f32_bits(xl.y), zf_l = f32_bits(xl.z);
    // Batches of 96 entries, a lane three of them; the next batch's entries
    // are loaded before this batch's positions are worked on, so a row costs
    // one trip to memory, not four (the FP64 pipe idles meanwhile)
    constexpr int NB = 3;
    int a = 0, k0 = 0;
    auto load_entries = [&](int ar, int kr, int* e) {
      const int len = __shfl_sync(FULL_MASK, len_l, ar & 31);
      const int* p = T.L.entries + __shfl_sync(FULL_MASK, static_cast<unsigned long long>(off_l), ar & 31);
#pragma unroll
      for (int h = 0; h < NB; ++h) {
        const int k = kr + 32 * h + lane;
        e[h] = -1;
        if (ar < nrow && k < len) {
          e[h] = __ldg(p + ((size_t(k >> 2) * T.L.stride) << 2) + (k & 3));
          if (T.packed) e[h] >>= 6;
        }
      }
    };
    int en[NB];
    load_entries(0, 0, en);
    while (a < nrow) {
      int e[NB];
      double4_32a p[NB];
#pragma unroll
      for (int h = 0; h < NB; ++h) {
        e[h] = en[h];
        if (e[h] >= 0) p[h] = T.x4[e[h]];
      }
      const int len = __shfl_sync(FULL_MASK, len_l, a);
      const bool last = k0 + 32 * NB >= len;
      load_entries(last ? a + 1 : a, last ? 0 : k0 + 32 * NB, en);
      const float xf = __shfl_sync(FULL_MASK, xf_l, a), yf = __shfl_sync(FULL_MASK, yf_l, a),
                  zf = __shfl_sync(FULL_MASK, zf_l, a);
      const float thr = f32_cut_threshold(cutsq_f, xf, yf, zf);
      if (MODE != LJ_ENERGY && row_l == a && k0 == 0) seg_b = seg_e = cnt;
#pragma unroll
      for (int h = 0; h < NB; ++h) {
        if (k0 + 32 * h >= len) break;
        bool keep = false;
        if (e[h] >= 0) {
          const float fx = xf - f32_bits(p[h].x), fy = yf - f32_bits(p[h].y), fz = zf - f32_bits(p[h].z);
          keep = !(fmaf(fz, fz, fmaf(fy, fy, fx * fx)) > thr);
        }
        const unsigned m = __ballot_sync(FULL_MASK, keep);
        if (cnt + __popc(m) > cap) flush();
        if (keep) {
          const int s = cnt + __popc(m & lt);
          sx[s] = p[h].x;
          sy[s] = p[h].y;
          sz[s] = p[h].z;
          if (MODE != LJ_FULL && T.half) sj[s] = e[h];
          sa[s] = Tag(UNI ? a : (a | (__ldg(T.P.type + e[h]) << 4)));
        }
        cnt += __popc(m);
        if (MODE != LJ_ENERGY && row_l == a) seg_e = cnt;
      }
      if (last) {
        ++a;
        k0 = 0;
      } else {
        k0 += 32 * NB;
      }
    }
    flush();
    if (MODE != LJ_ENERGY && row_l < nrow) {
      double* fi = T.f + 3 * size_t(i0 + row_l) + comp_l;
      if (MODE == LJ_HALF) atomicAdd(fi, acc);
      else if (ZERO) *fi = 0.0 + acc;  // the pending deep_copy(f, 0) folded into the store
      else *fi += acc;
    }
    __syncwarp();
  }
  if constexpr (MODE == LJ_ENERGY) {
    __shared__ double sh[LJT_WARPS];
    const double t = block_sum(esum, sh);
    if (threadIdx.x == 0) T.part[blockIdx.x] = t;
  }
}

// A thread per row, for very short and very long rows (lj_by_rows): the same operations
// in the same order.  Energy: a fixed number of CTAs, one partial each, as above.
constexpr int LJR_THREADS = 128;
template <int MODE, bool UNI, bool IDIAL, bool ZERO>
__global__ void __launch_bounds__(LJR_THREADS) k_lj_fp64_rows(LJTile T) {
  double esum = 0.0;
  const int step = MODE == LJ_ENERGY ? gridDim.x * LJR_THREADS : T.n;
  for (int i = blockIdx.x * LJR_THREADS + threadIdx.x; i < T.n; i += step) {
    const double4_32a xi = T.x4[i];
    const Row row(T.L, i);
    const int ti = UNI ? 0 : T.P.type[i] * T.P.ntypes;
    double fx = 0.0, fy = 0.0, fz = 0.0;
    for (int k = 0; k < row.n; ++k) {
      int j = row[k];
      if (T.packed) j >>= 6;
      const double4_32a xj = T.x4[j];
      const double dx = xi.x - xj.x, dy = xi.y - xj.y, dz = xi.z - xj.z;
      const double rsq = dx * dx + dy * dy + dz * dz;
      const int tp = UNI ? 0 : ti + __ldg(T.P.type + j);
      const double cutsq = UNI ? T.P.cutsq_0 : __ldg(T.P.cutsq + tp);
      if (!(rsq < cutsq)) continue;
      const double lj1 = UNI ? T.P.lj1_0 : __ldg(T.P.lj1 + tp), lj2 = UNI ? T.P.lj2_0 : __ldg(T.P.lj2 + tp);
      if constexpr (MODE == LJ_ENERGY) {
        const double r2inv = recip_rn(rsq), r6inv = r2inv * r2inv * r2inv;
        const double r2c = 1.0 / cutsq, r6c = r2c * r2c * r2c, c12 = lj1 / 12.0, c6 = lj2 / 6.0;
        esum += (T.half && j < T.n ? 1.0 : 0.5) * (r6inv * (c12 * r6inv - c6) - r6c * (c12 * r6c - c6));
      } else {
        const double fpair = lj_fpair<IDIAL>(rsq, lj1, lj2, IDIAL ? __ldg(T.P.intensity + tp) : 1.0);
        const double px = dx * fpair, py = dy * fpair, pz = dz * fpair;
        fx += px;
        fy += py;
        fz += pz;
        if (MODE == LJ_HALF && (!IDIAL || j < T.n)) {
          double* fj = T.f + 3 * size_t(j);
          atomicAdd(fj, -px);
          atomicAdd(fj + 1, -py);
          atomicAdd(fj + 2, -pz);
        }
      }
    }
    if constexpr (MODE != LJ_ENERGY) {
      double* fi = T.f + 3 * size_t(i);
      if (MODE == LJ_HALF) {
        atomicAdd(fi, fx);
        atomicAdd(fi + 1, fy);
        atomicAdd(fi + 2, fz);
      } else {  // ZERO: the pending deep_copy(f, 0) folded into the store
        fi[0] = (ZERO ? 0.0 : fi[0]) + fx;
        fi[1] = (ZERO ? 0.0 : fi[1]) + fy;
        fi[2] = (ZERO ? 0.0 : fi[2]) + fz;
      }
    }
  }
  if constexpr (MODE == LJ_ENERGY) {
    __shared__ double sh[LJR_THREADS / 32];
    const double t = block_sum(esum, sh);
    if (threadIdx.x == 0) T.part[blockIdx.x] = t;
  }
}

}  // namespace
}  // namespace emd
