// Neighbour rows of one bin's particles, one warp per bin (neighbor_csr.h:176-435).
//
// The warp stages the particles of the 27-bin stencil in the reference order
// (bx_j slowest, bz_j fastest; inside a bin in permutation order) in shared
// memory, as FP32 positions relative to the centre of ITS bin, and drops those
// farther than the cutoff from all of its centre atoms.  Each lane owns a centre
// atom.  32 candidates at a time every lane forms a mask of those within the
// cutoff, two r^2 per packed operation and four candidates per three shared-memory
// reads, and nothing else in that loop; then it walks its mask's bits (about 6 of
// 32) and appends them to its row, so row i lists its neighbours in exactly the
// order the serial reference appends them.  A lane with an r^2 in a band around
// the cutoff (row_band) goes over its 32 again and decides those pairs by the FP64
// positions, so every accept / reject equals the FP64 test `rsq <= neigh_cut^2`.
//
// Bound by instruction issue: about 7 instructions per candidate and lane and 13
// per listed pair (tests, order rule and append for every candidate took 20).
// Full lists, packed, 4,000,000 particles: 2.26 ms with one loop, 1.81 with masks.
// A gas's build is bound by the latency of its many short warps: an empty bin leaves
// first, and up to eight candidates take a quarter of the mask (256,000 particles, 0.2 / 0.5 / 1.1 a
// bin: 395 / 253 / 132 us with one loop, 411 / 286 / 155 with whole masks, 366 / 249 / 137 so).
#pragma once
#include "emd_device.cuh"
#include "emd_internal.h"
#include "neigh_rows.cuh"

namespace emd {
namespace {

constexpr int NB_CAP = 256;  // staged candidates

struct RowStage {  // one warp's shared memory
  float x[NB_CAP], y[NB_CAP], z[NB_CAP];
  int w[NB_CAP];  // row entry
  int pre[28], boff[27], self[32], pad;  // self: where a centre atom itself is staged
};

struct RowArgs {
  const double4_32a* x4;
  const float4* xl;  // FP32 position relative to the particle's bin centre
  const int* permute;
  int nby, nbz;      // bins per dimension, halo included
  float wx, wy, wz;  // bin widths
  int n_local, newton;
  double cutsq;
  float cut_lo, cut_hi;  // FP32 decision band
  int* num_neighs;
  int* rows;  // column-major, leading dimension `stride`, capacity K
  int stride, K;
};

// Half width of the band, relative to cutsq.  A coordinate difference of two
// FP32 bin-relative positions and a bin shift is off by less than 2^-24 (2.5 w + 3
// cut) (positions within 0.6 w of their bin centre; the shift, the sum and the
// difference round once each), r^2 by 2 sqrt(3) cut times that and three more
// roundings, 1e-6 for w = cut; five times that here.
inline double row_band(double w, double cut) { return 1e-6 * (2.0 + 3.0 * w / cut); }

// Exact FP64 re-test of a pair whose FP32 r^2 fell inside the guard band.
// Kept out of line: inlined, the compiler predicates it into the candidate
// loop and every batch of 32 candidates then issues its FP64 instructions
// (64 cycles each on this part) whether or not a lane needs them.
__device__ __noinline__ bool retest_fp64(const double4_32a* __restrict__ x4, int i, int j, double cutsq) {
  const double4_32a pi = x4[i], pj = x4[j];
  const double ddx = pi.x - pj.x, ddy = pi.y - pj.y, ddz = pi.z - pj.z;
  return (ddx * ddx + ddy * ddy + ddz * ddz) <= cutsq;
}

// monotone integer key of a double (exact ordering, integer pipe)
__device__ __forceinline__ long long okey(double v) {
  const long long b = __double_as_longlong(v);
  return b >= 0 ? b : (b ^ 0x7fffffffffffffffLL);
}

// The half list's order rule (neighbor_csr.h:287-291): j "above" i when
// (x_j, y_j, z_j) > (x_i, y_i, z_i) lexicographically, from the FP64
// positions.  Out of line for the same reason as retest_fp64.
__device__ __noinline__ bool above_fp64(const double4_32a* __restrict__ x4, int i, int j) {
  const double4_32a xi = x4[i], xj = x4[j];
  const long long ix = okey(xi.x), iy = okey(xi.y), iz = okey(xi.z);
  const long long jx = okey(xj.x), jy = okey(xj.y), jz = okey(xj.z);
  return (jx > ix) || ((jx == ix) && ((jy > iy) || ((jy == iy) && (jz > iz))));
}

// bit 31 - k: candidate k of the n <= 32 from `b` on is within the cutoff of xi (the
// first eight alone where there are no more: a gas's bins)
__device__ __forceinline__ unsigned row_mask(const RowArgs& a, const RowStage& st, int b, int n, const float4& xi, int i,
                                             bool packed) {
  const float2 m1 = make_float2(-1.f, -1.f);
  const float2 xx = make_float2(xi.x, xi.x), yy = make_float2(xi.y, xi.y), zz = make_float2(xi.z, xi.z);
  const float mid = 0.5f * (a.cut_lo + a.cut_hi), band = 0.501f * (a.cut_hi - a.cut_lo);
  const float2 nm = make_float2(-mid, -mid);
  unsigned mask = 0;
  float least = 3.0e38f;
  auto two = [&](float2 x, float2 y, float2 z) {
    const float2 dx = __ffma2_rn(x, m1, xx), dy = __ffma2_rn(y, m1, yy), dz = __ffma2_rn(z, m1, zz);
    const float2 rsq = __ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __fmul2_rn(dx, dx)));
    const float2 t = __fadd2_rn(rsq, nm);
    mask = __funnelshift_l(__float_as_uint(t.x), mask, 1);  // the sign of t
    mask = __funnelshift_l(__float_as_uint(t.y), mask, 1);
    least = fminf(least, fminf(fabsf(t.x), fabsf(t.y)));
  };
#pragma unroll
  for (int k = 0; k < 32; k += 4) {
    if (k == 8 && n <= 8) {
      mask <<= 24;
      break;
    }
    const float4 x = *reinterpret_cast<const float4*>(st.x + b + k);
    const float4 y = *reinterpret_cast<const float4*>(st.y + b + k);
    const float4 z = *reinterpret_cast<const float4*>(st.z + b + k);
    two(make_float2(x.x, x.y), make_float2(y.x, y.y), make_float2(z.x, z.y));
    two(make_float2(x.z, x.w), make_float2(y.z, y.w), make_float2(z.z, z.w));
  }
  if (least <= band) {
#pragma unroll 1
    for (int k = 0; k < 32; ++k) {
      const float dx = xi.x - st.x[b + k], dy = xi.y - st.y[b + k], dz = xi.z - st.z[b + k];
      const float rsq = __fmaf_rn(dz, dz, __fmaf_rn(dy, dy, __fmul_rn(dx, dx)));
      if (rsq < a.cut_lo || rsq > a.cut_hi) continue;
      const int j = packed ? (st.w[b + k] >> 6) : st.w[b + k];
      const unsigned bit = 0x80000000u >> k;
      mask = retest_fp64(a.x4, i, j, a.cutsq) ? (mask | bit) : (mask & ~bit);
    }
  }
  return mask;
}

// Rows of the particles of bin (bx, by, bz) that are owned; longest row of the
// warp's lanes.  `bin(b, off)`: particles of bin b and their first position in
// the permutation.
template <bool HALF, bool PACKED, typename Bin>
__device__ __forceinline__ int rows_of_bin(const RowArgs& a, RowStage& st, int bx, int by, int bz, Bin&& bin) {
  const int lane = threadIdx.x & 31;
  int cntb = 0, offb = 0;
  if (lane < 27) {
    const int dbx = lane / 9 - 1, dby = (lane / 3) % 3 - 1, dbz = lane % 3 - 1;
    cntb = bin(((bx + dbx) * a.nby + (by + dby)) * a.nbz + (bz + dbz), offb);
  }
  const int nc = __shfl_sync(FULL_MASK, cntb, 13), oc = __shfl_sync(FULL_MASK, offb, 13);
  if (nc == 0) return 0;
  // inclusive scan of the 27 stencil counts over the lanes
  int inc = cntb;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(FULL_MASK, inc, o);
    if (lane >= o) inc += v;
  }
  if (lane < 27) {
    st.pre[lane + 1] = inc;
    st.boff[lane] = offb;
  }
  if (lane == 0) st.pre[0] = 0;
  __syncwarp();
  const int M = st.pre[27];
  int mx = 0;
  // Candidates farther than the cutoff from every centre atom of the chunk
  // are dropped while staging, once per warp: the squared FP32 distance to the
  // bounding box of the chunk's centre atoms is at most a few roundings above
  // any centre atom's FP32 r^2, and a dropped candidate's exceeds cut_hi by a
  // 1e-5 margin, so no lane would accept the pair or re-test it in FP64.
  const float prune_sq = a.cut_hi * 1.00001f;
  // half lists: the FP32 x offset of a candidate from a centre atom has the
  // sign of the FP64 x difference once it exceeds the FP32 rounding of the
  // two offsets and the bin shift (below 2^-24 (3 w + 2 drift) in all); only
  // x ties within that bound need the FP64 order keys
  const float otol = 1e-6f * (1.0f + 4.0f * fmaxf(a.wx, fmaxf(a.wy, a.wz)));
  const unsigned lt = (1u << lane) - 1u;
  for (int a0 = 0; a0 < nc; a0 += 32) {
    // this lane's centre atom
    const int bi = a0 + lane;
    const int i = bi < nc ? a.permute[oc + bi] : -1;
    const bool own = i >= 0 && i < a.n_local;  // ghosts own no row
    float4 xi = make_float4(0.f, 0.f, 0.f, 0.f);
    if (own) xi = a.xl[i];
    // bounding box of the chunk's centre atoms that own rows
    float lox = own ? xi.x : 3.0e38f, loy = own ? xi.y : 3.0e38f, loz = own ? xi.z : 3.0e38f;
    float hix = own ? xi.x : -3.0e38f, hiy = own ? xi.y : -3.0e38f, hiz = own ? xi.z : -3.0e38f;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      lox = fminf(lox, __shfl_xor_sync(FULL_MASK, lox, o));
      loy = fminf(loy, __shfl_xor_sync(FULL_MASK, loy, o));
      loz = fminf(loz, __shfl_xor_sync(FULL_MASK, loz, o));
      hix = fmaxf(hix, __shfl_xor_sync(FULL_MASK, hix, o));
      hiy = fmaxf(hiy, __shfl_xor_sync(FULL_MASK, hiy, o));
      hiz = fmaxf(hiz, __shfl_xor_sync(FULL_MASK, hiz, o));
    }
    int cnt = 0, at = -1;  // entries; where i itself is staged
    // next slot of the row: +1 inside a 4-entry granule, then on to the
    // row's next granule (4 stride - 3 ints further)
    int* rp = a.rows + quad_index(own ? i : 0, 0, a.stride);
    const int jump = 4 * a.stride - 3;
    auto put = [&](int w) {
      *rp = w;
      rp += (cnt & 3) == 3 ? jump : 1;
      ++cnt;
    };
    auto append = [&](int b, int n) {  // the n <= 32 candidates from b on
      unsigned mask = row_mask(a, st, b, n, xi, i, PACKED);
      if (unsigned(at - b) < 32u) mask &= ~(0x80000000u >> (at - b));
      if (HALF) {
        // neighbor_csr.h:287-291: skip unless j is "above" i
        // lexicographically, or j is a ghost with newton off
        for (unsigned left = mask; left;) {
          const int k = __clz(left), w = st.w[b + k], j = PACKED ? (w >> 6) : w;
          const unsigned bit = 0x80000000u >> k;
          left &= ~bit;
          if (j >= a.n_local && !a.newton) continue;
          const float gx = __fsub_rn(st.x[b + k], xi.x);
          if (fabsf(gx) > otol ? !(gx > 0.f) : !above_fp64(a.x4, i, j)) mask &= ~bit;
        }
      }
      if (cnt + __popc(mask) <= a.K) {
        while (mask) {
          const int k = __clz(mask);
          mask &= ~(0x80000000u >> k);
          put(st.w[b + k]);
        }
      } else {  // overflow: the rest is counted
        while (mask) {
          const int k = __clz(mask);
          mask &= ~(0x80000000u >> k);
          if (cnt < a.K) put(st.w[b + k]);
          else ++cnt;
        }
      }
    };
    int m = 0;  // candidates staged
    st.self[lane] = -1;
    __syncwarp();
    for (int t0 = 0; t0 < M; t0 += 32) {
      const int g = t0 + lane;
      bool keep = false;
      float cx = 0.f, cy = 0.f, cz = 0.f;
      int w = 0;
      if (g < M) {
        int s = 0;  // stencil bin of candidate g: binary search of the prefix
#pragma unroll
        for (int h = 16; h >= 1; h >>= 1)
          if (s + h <= 27 && st.pre[s + h] <= g) s += h;
        const int j = a.permute[st.boff[s] + (g - st.pre[s])];
        const float4 p = a.xl[j];
        cx = p.x + float(s / 9 - 1) * a.wx;
        cy = p.y + float((s / 3) % 3 - 1) * a.wy;
        cz = p.z + float(s % 3 - 1) * a.wz;
        const int code = ((s / 9) << 4) | (((s / 3) % 3) << 2) | (s % 3);
        w = PACKED ? ((j << 6) | code) : j;
        const float ex = fmaxf(fmaxf(lox - cx, cx - hix), 0.f), ey = fmaxf(fmaxf(loy - cy, cy - hiy), 0.f),
                    ez = fmaxf(fmaxf(loz - cz, cz - hiz), 0.f);
        keep = __fmaf_rn(ez, ez, __fmaf_rn(ey, ey, __fmul_rn(ex, ex))) <= prune_sq;
      }
      const unsigned bal = __ballot_sync(FULL_MASK, keep);
      if (keep) {
        const int k = m + __popc(bal & lt), self = g - st.pre[13] - a0;
        if (unsigned(self) < 32u && g < st.pre[14]) st.self[self] = k;
        st.x[k] = cx;
        st.y[k] = cy;
        st.z[k] = cz;
        st.w[k] = w;
      }
      m += __popc(bal);
      if (m > NB_CAP - 32 || t0 + 32 >= M) {  // full, or the last
        const bool last = t0 + 32 >= M;
        const int full = last ? (m + 31) & ~31 : m & ~31;
        // the last 32 padded far outside the cutoff
        if (last && m + lane < full) {
          st.x[m + lane] = st.y[m + lane] = st.z[m + lane] = 1.0e4f;
          st.w[m + lane] = 0;
        }
        __syncwarp();
        at = st.self[lane];
        if (own)
          for (int b = 0; b < full; b += 32) append(b, m - b);
        __syncwarp();
        const int rest = last ? 0 : m - full;
        if (lane < rest) {
          cx = st.x[full + lane];
          cy = st.y[full + lane];
          cz = st.z[full + lane];
          w = st.w[full + lane];
        }
        __syncwarp();
        if (lane < rest) {
          st.x[lane] = cx;
          st.y[lane] = cy;
          st.z[lane] = cz;
          st.w[lane] = w;
        }
        st.self[lane] = at >= full ? at - full : -1;
        __syncwarp();  // the next candidates' lanes write self too
        m = rest;
      }
    }
    if (own) {
      a.num_neighs[i] = cnt;
      mx = max(mx, cnt);
    }
    __syncwarp();
  }
  return __reduce_max_sync(FULL_MASK, mx);
}

}  // namespace
}  // namespace emd
