// U_tot of the SNAP mixed form: the sums of k_snap_u from FP32 pairs (f32_pairs.cuh).
// U_tot is rounded to FP32 afterwards, so what counts is what the sums add to that
// rounding: at most 1e-12 of the neighbours' total weight for 26 neighbours (5e-8
// is the rounding; 1 in 2,500 elements comes out one FP32 step from where sums in
// FP64 round to), times the polynomials' coefficients (16 at twojmax 8).
#pragma once
#include "snap_kernel.cuh"

namespace emd {
namespace snapk {

// a row's powers of a; its powers of b times those of x
__device__ __forceinline__ void su_row_a(int J, float4* t, F2 ar, F2 ai) {
  const F2 nai{-ai.h, -ai.l};
  const float one = f2_base(1.f);
  F2 p{1.f, 0.f}, r{0.f, 0.f};
#pragma unroll 1
  for (int q = 0; q <= J; ++q) {
    t[q] = float4{p.h, p.l, r.h, r.l};
    f2_cmul(p, r, ar, ai, nai, one);
  }
}
__device__ __forceinline__ void su_row_b(int J, float4* col, F2 ar, F2 ai, F2 br, F2 bi, F2 w) {
  const F2 nbi{-bi.h, -bi.l};
  const float one = f2_base(1.f), wb = f2_base(fabsf(w.h));
  F2Sum sx{one, 0.f};
  sx.add(ar, ar);
  sx.add(ai, ai);
  sx.add(F2{-br.h, -br.l}, br);
  sx.add(nbi, bi);
  const F2 x = sx.value(one);
  F2 u = w, v{0.f, 0.f};
#pragma unroll 1
  for (int T = 0; T <= J; ++T) {
    F2 uk = u, vk = v;
    *col++ = float4{uk.h, uk.l, vk.h, vk.l};
#pragma unroll 1
    for (int k = 1; k <= (J - T) / 2; ++k) {
      F2Sum su{wb, 0.f}, sv{wb, 0.f};
      su.add(uk, x);
      sv.add(vk, x);
      uk = su.value(wb);
      vk = sv.value(wb);
      *col++ = float4{uk.h, uk.l, vk.h, vk.l};
    }
    f2_cmul(u, v, br, bi, nbi, wb);
  }
}

// su_store from the sums over the powers of x (xs: per entry, p u, r u, p v, r v)
__device__ __forceinline__ void su_store32(const SnapDev& S, int e, const F2Sum* xs, float base, Cplx<float>* U) {
  const Entry& E = S.ent[e];
  const int k = (E.j - E.q - E.T) / 2;
  const float2* m = S.mono + E.mo;
  F2 s[4];
#pragma unroll
  for (int h = 0; h < 4; ++h) s[h] = F2{0.f, 0.f};
  for (int l = 0; l <= k; ++l) {
    const float2 cm = __ldg(m + l);
    const F2Sum* x = xs + 4 * (e - k + l);
#pragma unroll
    for (int h = 0; h < 4; ++h) f2_dot(s[h], F2{cm.x, cm.y}, x[h].value(base));
  }
  const F2 pu = s[0], ru = s[1], pv = s[2], rv = s[3];
  const F2 nru{-ru.h, -ru.l}, nrv{-rv.h, -rv.l};
  const int2 h = S.half[e];
  U[h.x] = Cplx<float>{f2_sum(pu, rv, E.T > 0 ? 0.f : float(S.wself)), f2_sum(pv, nru, 0.f)};
  if (h.y >= 0) {
    const float sg = E.T & 1 ? -1.f : 1.f;
    U[h.y] = Cplx<float>{sg * f2_sum(pu, nrv, 0.f), -sg * f2_sum(pv, ru, 0.f)};
  }
}

// One warp per atom as in k_snap_u, 16 neighbours at a time: 16 lanes form the
// powers of a and 16 those of b (a table of 32 rows, each by one lane, left ten
// warps on an SM, 0.92 ms per 128,000 atoms; 0.87 so).  Then lanes = entries: the two
// columns of an entry give its four sums, for two 16-byte loads.
constexpr int SU_ROWS = 16;
static __global__ void __launch_bounds__(32) k_snap_u32(SnapArgs A) {
  const SnapDev& S = A.S;
  extern __shared__ __align__(16) unsigned char su_smem32[];
  F2Sum* xs = reinterpret_cast<F2Sum*>(su_smem32);             // 4 ne sums
  float4* tab = reinterpret_cast<float4*>(xs + 4 * S.ne);      // SU_ROWS rows
  const int al = blockIdx.x, lane = threadIdx.x, n = A.cnt[al];
  const size_t np = size_t(A.n) * A.cap;
  const float* pr = static_cast<const float*>(A.pr) + size_t(al) * A.cap;
  float weight = 0.f;
  for (int k = lane; k < n; k += 32) weight += fabsf(pr[PR_SF * np + k]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) weight += __shfl_xor_sync(FULL_MASK, weight, o);
  const float base = f2_base(1.001f * weight);
  for (int n0 = 0; n0 < max(n, 1); n0 += SU_ROWS) {
    const int m = min(SU_ROWS, n - n0), nb = lane & (SU_ROWS - 1);
    if (nb < m) {
      const float* q = pr + n0 + nb;
      auto get = [&](int h, int l) { return F2{q[h * np], q[l * np]}; };
      const F2 ar = get(PR_AR, PR_ARL), ai = get(PR_AI, PR_AIL);
      float4* t = tab + nb * S.cols;
      if (lane < SU_ROWS) su_row_a(S.twojmax, t, ar, ai);
      else su_row_b(S.twojmax, t + S.twojmax + 1, ar, ai, get(PR_BR, PR_BRL), get(PR_BI, PR_BIL), get(PR_SF, PR_SFL));
    }
    __syncwarp();
    for (int e0 = 0; e0 < S.ne; e0 += 96) {  // three entries per lane at once
      int2 col[3];
      F2Sum acc[3][4];
#pragma unroll
      for (int h = 0; h < 3; ++h) {
        const int e = e0 + 32 * h + lane;
        col[h] = e < S.ne ? __ldg(S.ucol + e) : int2{0, 0};
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[h][c] = e < S.ne && n0 > 0 ? xs[4 * e + c] : F2Sum{base, 0.f};
      }
      auto rows = [&](auto nh) {
#pragma unroll 2
        for (int k = 0; k < m; ++k) {
          const float4* t = tab + k * S.cols;
#pragma unroll
          for (int h = 0; h < decltype(nh)::value; ++h) {
            const float4 a = t[col[h].x], b = t[col[h].y];
            acc[h][0].add(F2{a.x, a.y}, F2{b.x, b.y});
            acc[h][1].add(F2{a.z, a.w}, F2{b.x, b.y});
            acc[h][2].add(F2{a.x, a.y}, F2{b.z, b.w});
            acc[h][3].add(F2{a.z, a.w}, F2{b.z, b.w});
          }
        }
      };
      if (e0 + 64 < S.ne) rows(std::integral_constant<int, 3>{});
      else if (e0 + 32 < S.ne) rows(std::integral_constant<int, 2>{});
      else rows(std::integral_constant<int, 1>{});
#pragma unroll
      for (int h = 0; h < 3; ++h) {
        const int e = e0 + 32 * h + lane;
        if (e < S.ne)
#pragma unroll
          for (int c = 0; c < 4; ++c) xs[4 * e + c] = acc[h][c];
      }
    }
    __syncwarp();
  }
  Cplx<float>* U = static_cast<Cplx<float>*>(A.U) + size_t(al) * S.nh;
  for (int e = lane; e < S.ne; e += 32) su_store32(S, __ldg(S.eord + e), xs, base, U);
}

inline void launch_u32(const SnapArgs& A, cudaStream_t s) {
  const size_t smem = sizeof(F2Sum) * 4 * size_t(A.S.ne) + SU_ROWS * 16 * size_t(A.S.cols);
  allow_dyn_smem(k_snap_u32);
  k_snap_u32<<<A.n, 32, smem, s>>>(A);
  EMD_CHECK_LAUNCH();
}

}  // namespace snapk
}  // namespace emd
