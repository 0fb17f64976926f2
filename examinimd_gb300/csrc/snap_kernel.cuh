// ForceSNAP on the device (force_snap_neigh_impl.h:160-724, sna_impl.hpp).
//
// The Wigner matrices of a neighbour depend on its Cayley-Klein pair (a, b)
// alone, and every element separates:
//   U_j(ma, mb) = N conj(a)^q b^T P_k(x)            (mb - ma = T >= 0)
//   U_j(ma, mb) = N conj(a)^q (-conj(b))^T P_k(x)   (ma - mb = T > 0)
// with q = j - ma - mb >= 0, j = q + T + 2k, x = |a|^2 - |b|^2, P_k the monic
// Jacobi polynomial P_k^(T, q) (three-term recurrence) and
// N = 2^-k j! / sqrt(ma! (j - ma)! mb! (j - mb)!).  q < 0 follows from the
// inversion U_j(j - ma, j - mb) = (-1)^(ma + mb) conj U_j(ma, mb).  This
// replaces the layer recursion of compute_uarray (sna_impl.hpp:642-720) and
// its derivative (compute_duarray, 729-893): no layers to keep, one polynomial
// for up to four elements, and lanes that all do the same thing.  An "entry"
// below is one (T, q, k): 95 of them at twojmax 8 for 285 elements.
//
// Per force call, over chunks of atoms:
//   k_snap_pairs  inside list and per-pair scalars (lanes = pairs)
//   k_snap_u      U_tot = wself + sum over the neighbours of w_j sfac U, from the
//                 four real products of conj(a)^q and b^T times powers of x (one warp
//                 per atom; lanes = neighbours, then sums)
//   k_snap_y      Z and Y (lanes = atoms, so the Clebsch-Gordan loops are
//                 uniform and every operand load is coalesced)
//   k_snap_force  pair forces (lanes = pairs): Phi = Re sum conj(U) Y and its
//                 gradient in (a, b), chain rule, scatter
// and for the energy k_snap_energy; for the fitting adjoint k_snap_dt (the
// directional derivative of X) and k_snap_pq.
//
// Precision forms: FP64 (the drop-in; snap.cu, -fmad=false) and mixed
// (snap_mixed.cu), where the pair scalars and the sums of U_tot are formed in FP32
// pairs of 48 bits and rounded to FP32, k_snap_y and the sums of k_snap_force run in
// FP32, and the cutoff test, the r^-14 repulsion and the force sums in FP64.  The
// recurrences and contractions use explicit fused multiply-adds in both forms.
#pragma once
#include <algorithm>
#include <cmath>
#include <type_traits>

#include "emd_device.cuh"
#include "emd_internal.h"
#include "f32_pairs.cuh"
#include "neigh_rows.cuh"

namespace emd {

ListView list_view(Ctx& c);

namespace snapk {

constexpr double MY_PI = 3.14159265358979323846;

template <typename R>
struct Cplx {
  R r, i;
};

// One (T, q, k) entry
struct Entry {
  double N;        // the elements' norm
  float Nf;
  double A, B;     // P_{k+1} = (x - A) P_k - B P_{k-1}
  int xo;          // first of its real sums: p u, [q>0] r u, [T>0] p v, [q>0, T>0] r v
  int mo;          // its coefficients of x^0 .. x^k, times N (SnapDev::mono)
  int T, q, j;
  int ep, em, mp, mm;  // full-grid elements (ma, mb) and (mb, ma), and their inversions
};

// The products of one (j1, j2) at one (2m, 2m') = (-q -+ T, -q +- T) of a Z task
struct ZRec {
  int p0, np, c0;      // products [p0, p0 + np), first coefficient
  short nj, d;         // number of j, the highest first; its distance from the task's highest j over 2
  int t0, z0;          // triple of the highest j; first kept Z
};
// One (T, q), one sign of T, and some of its records
struct ZTask {
  int rec0, rec1;      // records [rec0, rec1)
  int y0, kmax;        // its part of Y: slots y0 .. y0 + kmax, in the order of k
  int grp0, grp1, s0;  // FP32: groups [grp0, grp1), first word of the stream
};
// FP32: a task's products of equal nj and d, whatever their (j1, j2)
struct ZGrp {
  int w0, np;          // first word (from the task's s0), products
  short nj, d;
};

struct SnapDev {
  int twojmax, ne, nx, nuf;    // entries, real sums, elements of the full grid
  int cols;                    // pairs of columns of a neighbour's table (su_cols)
  int ntask, nfull, nz;        // Z tasks, (j1 >= j2, j) triples, kept Z values per atom
  int ncoeff, ncoeffall, nelem, ntypes;
  double rfac0, rmin0, cutsq, wself;
  int switchflag;
  const Entry* ent;
  const int* e0;       // (J + 1) x (J + 1): first entry of (T, q)
  const int2* xsum;    // nx: the two factors of a sum in a neighbour's row (k_snap_u, k_snap_dt)
  const int2* psum;    // the same where the row holds P_k (k_snap_u above SU_POWERS)
  const int2* ucol;    // ne: the mixed form's two columns of an entry
  const float2* mono;  // N P_k in powers of x, high and low part
  const double* monod; // the same in FP64
  const int* eord;     // entries, highest k first
  const ZTask* task;
  const ZRec* rec;
  const int2* prod;    // the two U elements of a product
  const double* zc;    // coefficients, nj per product
  // FP32: groups, and per element a stream (zs_n each) of every product's two
  // U elements (16 bits each) and coefficients times cY, zs_words(nj) words each
  const ZGrp* grp;
  const uint4* zs;
  int zs_n;
  const double* cY;    // nelem x nfull
  const double* AB;    // ne x 2
  const float* AB_f;
  const double* beta0;
  const double* wjelem;
  const double* pr;    // per element pair: rcut, rscale0, pi / (rcut - rmin0)
  const float2* pr32;  // the same, wjelem and -rmin0 as FP32 pairs
  const float2* wj32;
  float2 nrmin32;
  const int* map;      // ntypes
  // half-grid elements of an entry, +T and -T (-1: none); the kept Z values of
  // triple t with their elements, [zt0[t], zt0[t + 1]) of zt
  int nh;
  const int2* half;
  const int4* hfull;   // per half-grid element: its full-grid index, its inversion's, sign
  const int* zt0;
  const int2* zt;
  int ny;              // slots of Y
  const int4* ysrc;    // per half-grid element: first slot, slots between parts, parts
};

// ---- pair fields, one array each of stride `np` (pairs of the chunk)
enum { PD_FX, PD_FY, PD_FZ, PD_N32, PD_AR = PD_N32, PD_AI, PD_BR, PD_BI, PD_SF, PD_EP, PD_N };  // FP64 (mixed form: PD_N32)
// mixed form (FP32): a, b, sfac, dsfac, u, the three numbers da/dr and db/dr are
// made of, and what the rounding of a, b and sfac left out; FP64 form: a and b as compute_duidrj rounds
// them, dsfac, u and every derivative in the reference's operations
enum { PR_AR, PR_AI, PR_BR, PR_BI, PR_DSF, PR_UX, PR_UY, PR_UZ, PR_SF, PR_C1, PR_GR, PR_R0,
       PR_ARL, PR_AIL, PR_BRL, PR_BIL, PR_SFL, PR_N };
enum { PF_DAR = PR_SF, PF_DAI = PF_DAR + 3, PF_DBR = PF_DAI + 3, PF_DBI = PF_DBR + 3, PF_N = PF_DBI + 3 };

struct SnapArgs {
  SnapDev S;
  const double4_32a* x4;
  const int* type;
  ListView L;
  int first, n;        // atoms [first, first + n) of this chunk
  int n_local, cap;    // owned atoms; pair slots per atom
  int rows;            // k_snap_pairs: atoms per warp
  double* pd;          // PD_N or PD_N32 x (n cap)
  void* pr;            // PR_N x (n cap), force type (the FP64 form reads a, b and sfac from pd)
  int* pj;             // n cap
  int* cnt;            // n
  void* U;             // n x nh complex, force type
  void* Y;             // tiles x ny x 2 x TA, force type: parts of the Y of half-grid elements
  int ta, nsplit;      // atoms per tile, CTAs per tile
  double* zkeep;       // tiles x nz x 32 complex, or null
  double* f;
  double* eatom;       // energy
  // adjoint
  const double* g;
  const int* ghost_owner;
  int newton;
  Cplx<double>* D;     // n x nh
  Cplx<double>* H;     // tiles x 2 nh x 32: weighted U and D elements
  double* adj;         // (2 nfull + 1) x n_local
  int tsplit;          // k_snap_force: T groups
  int apc;             // k_snap_force: atoms per CTA
  const int* tmask;    // tsplit masks of T
};

// ------------------------------------------------------------------ pairs
// One warp takes `rows` atoms: their rows are filtered in FP32 (conservative,
// see f32_cut_threshold) into a shared list, then the lanes take listed pairs
// 32 at a time and write the scalars.  A listed pair that the FP64 test puts
// outside the cutoff is written with zero weight and force.
constexpr int SP_ROWS = 8;
constexpr int SP_CAP = 512;  // listed pairs per warp; a fuller list is emptied in between

template <typename R>
__global__ void __launch_bounds__(64) k_snap_pairs(SnapArgs A) {
  const SnapDev& S = A.S;
  __shared__ int s_j[2][SP_CAP];
  __shared__ int s_a[2][SP_CAP];  // atom of the warp | slot << 4
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned lt = (1u << lane) - 1u;
  const int a0 = (blockIdx.x * 2 + warp) * A.rows;
  if (a0 >= A.n) return;
  const int na = min(A.rows, A.n - a0);
  int* lj = s_j[warp];
  int* la = s_a[warp];
  const size_t np = size_t(A.n) * A.cap;
  constexpr bool kF64 = sizeof(R) == sizeof(double);
  R* pr = static_cast<R*>(A.pr);
  auto flush = [&](int cnt) {
    __syncwarp();
    for (int k = lane; k < cnt; k += 32) {
      const int al = a0 + (la[k] & 15), slot = la[k] >> 4, j = lj[k];
      const double4_32a pi = A.x4[A.first + al], pj = A.x4[j];
      const double x = pj.x - pi.x, y = pj.y - pi.y, z = pj.z - pi.z;
      const double rsq = x * x + y * y + z * z;
      const size_t p = size_t(al) * A.cap + slot;
      double* q = A.pd + p;
      const bool in = rsq < S.cutsq;
      const int ei = S.map[A.type[A.first + al]], ej = S.map[A.type[j]];
      const double* t = S.pr + 3 * (ei * S.nelem + ej);
      R* w = pr + p;
      if constexpr (kF64) {
        const double rcut = t[0], rscale0 = t[1], rsw = t[2];
        const double wj = in ? S.wjelem[ej] : 0.0;
        double sf = 1.0, dsf = 0.0;
        const double r = in ? sqrt(rsq) : 1.0;
        // compute_ui (sna_impl.hpp:174-187): a, b of compute_uarray
        const double theta0 = (r - S.rmin0) * S.rfac0 * MY_PI / (rcut - S.rmin0);
        const double z0u = r / tan(theta0);
        const double r0u = 1.0 / sqrt(r * r + z0u * z0u);
        q[PD_AR * np] = in ? r0u * z0u : 1.0;
        q[PD_AI * np] = in ? -r0u * z : 0.0;
        q[PD_BR * np] = in ? r0u * y : 0.0;
        q[PD_BI * np] = in ? -r0u * x : 0.0;
        // compute_duidrj + the prologue of compute_duarray (sna_impl.hpp:291-321, 729-778)
        const double th = (r - S.rmin0) * rscale0;
        const double cs = cos(th), sn = sin(th);
        const double z0 = r * cs / sn;
        const double dz0dr = z0 / r - (r * rscale0) * (rsq + z0 * z0) / rsq;
        const double rinv = 1.0 / r;
        const double uk[3] = {x * rinv, y * rinv, z * rinv};
        const double r0inv = 1.0 / sqrt(r * r + z0 * z0);
        w[PR_AR * np] = in ? z0 * r0inv : 1.0;
        w[PR_AI * np] = in ? -z * r0inv : 0.0;
        w[PR_BR * np] = in ? y * r0inv : 0.0;
        w[PR_BI * np] = in ? -x * r0inv : 0.0;
        const double dr0invdr = -(r0inv * r0inv * r0inv) * (r + z0 * dz0dr);
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          const double dr0inv = dr0invdr * uk[d], dz0 = dz0dr * uk[d];
          w[(PF_DAR + d) * np] = in ? dz0 * r0inv + z0 * dr0inv : 0.0;
          w[(PF_DAI + d) * np] = in ? -z * dr0inv + (d == 2 ? -r0inv : 0.0) : 0.0;
          w[(PF_DBR + d) * np] = in ? y * dr0inv + (d == 1 ? r0inv : 0.0) : 0.0;
          w[(PF_DBI + d) * np] = in ? -x * dr0inv + (d == 0 ? -r0inv : 0.0) : 0.0;
          w[(PR_UX + d) * np] = in ? uk[d] : 0.0;
        }
        // compute_sfac, compute_dsfac (sna_impl.hpp:1099-1128)
        if (S.switchflag != 0 && r > S.rmin0) {
          sf = r > rcut ? 0.0 : 0.5 * (cos((r - S.rmin0) * rsw) + 1.0);
          dsf = r > rcut ? 0.0 : -0.5 * sin((r - S.rmin0) * rsw) * rsw;
        }
        w[PR_DSF * np] = dsf * wj;
        // extra repulsion of the reference (force_snap_neigh_impl.h:705-711) and
        // its energy 1.25e5 / r^12 per ordered pair
        const double r2 = rsq * rsq, r4 = r2 * r2;
        const double fr = in ? -1.5e6 / (r4 * r2 * rsq) : 0.0;
        q[PD_FX * np] = x * fr;
        q[PD_FY * np] = y * fr;
        q[PD_FZ * np] = z * fr;
        q[PD_EP * np] = in ? 1.25e5 / (r4 * r2) : 0.0;
        q[PD_SF * np] = sf * wj;
      } else {
        // The same quantities in closed form, once, in FP32 pairs (48 bits): in
        // FP64, two sincos, a reciprocal root and the conversions took most of
        // the kernel (128,000 atoms: 0.83 ms, 0.28 in pairs).  With s =
        // sin(theta0), c = cos(theta0): z0 = r c / s and r0inv = s / r, so
        //   a = c - i z s / r, b = (y - i x) s / r,
        //   da/dr_k = -s rscale0 u_k - i (g u_k z + r0inv [k = z]), db/dr_k likewise,
        //   g = d(s / r)/dr = (c rscale0 r - s) / r^2 (the prologue of
        //   compute_duarray without its cancelling terms)
        const float2* t32 = S.pr32 + 3 * (ei * S.nelem + ej);
        auto f2 = [](float2 v) { return F2{v.x, v.y}; };
        const F2 one{1.f, 0.f}, zero{0.f, 0.f};
        const F2 rs = in ? f2_split(rsq) : one;
        const F2 rv = f2_rsqrt(rs), r = f2_mul(rs, rv), d = f2_add(r, f2(S.nrmin32));
        const F2 scale = f2(__ldg(t32 + 1)), slope = f2(__ldg(t32 + 2)), w32 = in ? f2(__ldg(S.wj32 + ej)) : zero;
        const F2 x2 = in ? f2_split(x) : zero, y2 = in ? f2_split(y) : zero, z2 = in ? f2_split(z) : zero;
        F2 sn, cs, sf = w32, dsf = zero;
        f2_sincos(f2_mul(d, scale), sn, cs);
        // r0inv is a positive root: beyond theta0 = pi (a pair past its own cutoff, inside
        // the common one, without switching) it is -s / r, and a, b change sign
        if (sn.h < 0.f) {
          sn = F2{-sn.h, -sn.l};
          cs = F2{-cs.h, -cs.l};
        }
        if (S.switchflag != 0 && d.h > 0.f) {
          F2 ss, cc;
          f2_sincos(f2_mul(d, slope), ss, cc);
          const bool far = f2_add(r, F2{-__ldg(t32).x, -__ldg(t32).y}).h > 0.f;  // beyond this pair's cutoff
          const F2 half = f2_add(cc, one);
          sf = far ? zero : f2_mul(F2{0.5f * half.h, 0.5f * half.l}, w32);
          dsf = far ? zero : f2_mul(f2_mul(F2{-0.5f * ss.h, -0.5f * ss.l}, slope), w32);
        }
        const F2 r0 = f2_mul(sn, rv);
        auto put = [&](int f, int l, F2 v) {
          v = f2_norm(v.h, v.l);
          w[f * np] = v.h;
          if (l >= 0) w[l * np] = v.l;
        };
        auto neg = [](F2 v) { return F2{-v.h, -v.l}; };
        put(PR_AR, PR_ARL, in ? cs : one);
        put(PR_AI, PR_AIL, neg(f2_mul(z2, r0)));
        put(PR_BR, PR_BRL, f2_mul(y2, r0));
        put(PR_BI, PR_BIL, neg(f2_mul(x2, r0)));
        put(PR_SF, PR_SFL, sf);
        put(PR_DSF, -1, dsf);
        put(PR_UX, -1, f2_mul(x2, rv));
        put(PR_UY, -1, f2_mul(y2, rv));
        put(PR_UZ, -1, f2_mul(z2, rv));
        put(PR_C1, -1, neg(f2_mul(sn, scale)));
        put(PR_GR, -1, f2_add(f2_mul(cs, scale), neg(r0)));
        put(PR_R0, -1, r0);
        // the r^-12 repulsion's force is FP64 from the FP64 r^2: its pair terms are of
        // the size of the net force and cancel in the sum over neighbours (from the 48
        // bits of 1 / r, r^-14 was off by 1e-13 of them)
        const double r2 = rsq * rsq, r4 = r2 * r2;
        const double fr = in ? -1.5e6 * recip_rn(r4 * r2 * rsq) : 0.0;
        q[PD_FX * np] = x * fr;
        q[PD_FY * np] = y * fr;
        q[PD_FZ * np] = z * fr;
      }
      A.pj[p] = j;
    }
    __syncwarp();
  };
  const float cutsq_f = __double2float_ru(S.cutsq);
  int cnt = 0;
  for (int al = 0; al < na; ++al) {
    const int i = A.first + a0 + al;
    const double4_32a xi = A.x4[i];
    const float xf = f32_bits(xi.x), yf = f32_bits(xi.y), zf = f32_bits(xi.z);
    const float thr = f32_cut_threshold(cutsq_f, xf, yf, zf);
    const Row row(A.L, i);
    int m = 0;  // pairs of this atom
    for (int k0 = 0; k0 < row.n; k0 += 32) {
      const int k = k0 + lane;
      bool keep = false;
      int j = 0;
      if (k < row.n) {
        j = row[k];
        const double4_32a p = A.x4[j];
        const float fx = xf - f32_bits(p.x), fy = yf - f32_bits(p.y), fz = zf - f32_bits(p.z);
        keep = !(fmaf(fz, fz, fmaf(fy, fy, fx * fx)) > thr);
      }
      const unsigned bal = __ballot_sync(FULL_MASK, keep);
      if (cnt + __popc(bal) > SP_CAP) {
        flush(cnt);
        cnt = 0;
      }
      if (keep) {
        const int s = __popc(bal & lt);
        lj[cnt + s] = j;
        la[cnt + s] = al | ((m + s) << 4);
      }
      cnt += __popc(bal);
      m += __popc(bal);
    }
    if (lane == 0) A.cnt[a0 + al] = m;
  }
  flush(cnt);
}

// ---------------------------------------------------------------------- U
// One warp per atom, 32 neighbours at a time.  Lanes = neighbours: the powers
// p_q + i r_q = a^q and u_T + i v_T = w b^T, the latter times the powers of x (the
// same for every q), go to the neighbour's row of a shared table.  Lanes = sums:
// each of the nx real sums is p or r times a power's u or v over the neighbours, one
// FP64 multiply-add per neighbour.  Then, once per atom, the sums over powers are
// combined into the polynomials' and those into the half-grid elements.  The powers'
// rounding is amplified by the polynomials' coefficients (16 at twojmax 8, 221 at
// 14); the forces' error against long double is what it was with P_k in the row
// (4e-15 of the RMS force).  Bound by the FP64 pipe: about 100 instructions for 32
// neighbours' rows (240 with P_k), nx / 32 for each neighbour; the table, half as
// wide, lets eleven warps share an SM instead of six (8,160 atoms: 0.33 -> 0.21 ms).
//
// Above twojmax 9 (SU_POWERS) the row holds u P_k and v P_k, so that nothing is
// amplified: forces of 54 and 128 atoms, RMS error against long double relative to the
// layer recursion's, 1.13 / 1.03 with powers and 1.06 / 1.02 with P_k at twojmax 10, 1.08
// and 1.01 at 11 (1.07 and 1.06, 1.08 and 1.05 at 8 and 9, where powers are kept); the
// bispectrum's own error 2.6e-15 and 1.0e-15 at 12.
//
// The mixed form, which rounds U_tot to FP32 anyway, takes k_snap_u32
// (snap_split.cuh): per 128,000 atoms 2.80 ms in FP64, 0.87 in FP32 pairs.
// pairs of columns of a neighbour's row: (p, r) of a^q; (u x^k, v x^k) of w b^T
inline int su_cols(int J) {
  int c = J + 1;
  for (int T = 0; T <= J; ++T) c += (J - T) / 2 + 1;
  return c | 1;  // odd: eight lanes' rows start in different banks
}

// doubles of an FP64 row (odd: rows start in different banks)
__host__ __device__ inline int su_stride(int cols) { return (2 * cols) | 1; }

constexpr int SU_POWERS = 9;

// columns of a row with P_k: p, r; u, v; u P_k, v P_k (k > 0)
__host__ __device__ inline int su_pcols(int J) {
  int c = 4 * (J + 1);
  for (int T = 0; T <= J; ++T)
    for (int q = 0; q <= J - T; ++q) c += (T ? 2 : 1) * ((J - T - q) / 2);
  return c | 1;
}

// that row
__device__ __forceinline__ void su_row_p(const SnapDev& S, double* t, double ar, double ai, double br, double bi,
                                         double w) {
  const int J = S.twojmax;
  double *uT = t + 2 * (J + 1), *prod = t + 4 * (J + 1);
  double p = 1.0, r = 0.0, u = w, v = 0.0;
#pragma unroll 1
  for (int q = 0; q <= J; ++q) {
    t[2 * q] = p;
    t[2 * q + 1] = r;
    uT[2 * q] = u;
    uT[2 * q + 1] = v;
    const double pn = fma(p, ar, -r * ai), un = fma(u, br, -v * bi);
    r = fma(p, ai, r * ar);
    v = fma(u, bi, v * br);
    p = pn;
    u = un;
  }
  const double x = fma(ar, ar, ai * ai) - fma(br, br, bi * bi);
  for (int T = 0; T <= J; ++T) {
    const double uu = uT[2 * T], vv = uT[2 * T + 1];
    for (int q = 0; q <= J - T - 2; ++q) {
      const double2* ab = reinterpret_cast<const double2*>(S.AB) + __ldg(S.e0 + T * (J + 1) + q);
      const int km = (J - T - q) / 2;
      double pm = 1.0, pk = x - __ldg(ab).x;
      *prod++ = uu * pk;
      if (T > 0) *prod++ = vv * pk;
      for (int k = 2; k <= km; ++k) {
        const double2 c = __ldg(ab + k - 1);
        const double pn = fma(x - c.x, pk, -c.y * pm);
        pm = pk;
        pk = pn;
        *prod++ = uu * pk;
        if (T > 0) *prod++ = vv * pk;
      }
    }
  }
}

// the neighbour's table row: powers of a, those of b times those of x
__device__ __forceinline__ void su_row(int J, double* t, double ar, double ai, double br, double bi, double w) {
  double* col = t + 2 * (J + 1);
  const double x = fma(ar, ar, ai * ai) - fma(br, br, bi * bi);
  double p = 1.0, r = 0.0, u = w, v = 0.0;
#pragma unroll 1
  for (int q = 0; q <= J; ++q) {
    t[2 * q] = p;
    t[2 * q + 1] = r;
    double uk = u, vk = v;
#pragma unroll 1
    for (int k = 0; k <= (J - q) / 2; ++k) {
      *col++ = uk;
      *col++ = vk;
      uk *= x;
      vk *= x;
    }
    const double pn = fma(p, ar, -r * ai), un = fma(u, br, -v * bi);
    r = fma(p, ai, r * ar);
    v = fma(u, bi, v * br);
    p = pn;
    u = un;
  }
}

// the half-grid elements of entry e from its sums over the powers of x (one group
// per k): conj(a)^q b^T = (p u + r v) + i (p v - r u); for -T: (-1)^T ((p u - r v)
// - i (p v + r u)); the coefficients hold N, the atom's own term is 1 on the
// diagonal (T = 0).  POLY: from the sums over P_k
template <bool POLY>
__device__ __forceinline__ void su_store(const SnapDev& S, int e, const double* xs, double self, Cplx<double>* U) {
  const Entry& E = S.ent[e];
  const bool hr = E.q > 0, hv = E.T > 0;
  const int k = POLY ? 0 : (E.j - E.q - E.T) / 2, g = (hr ? 2 : 1) * (hv ? 2 : 1);
  const double *m = S.monod + E.mo, *x = xs + E.xo - k * g;
  double pu = 0.0, ru = 0.0, pv = 0.0, rv = 0.0;
  for (int l = 0; l <= k; ++l, x += g) {
    const double c = POLY ? E.N : __ldg(m + l);
    pu = fma(c, x[0], pu);
    if (hr) ru = fma(c, x[1], ru);
    if (hv) pv = fma(c, x[hr ? 2 : 1], pv);
    if (hr && hv) rv = fma(c, x[3], rv);
  }
  const int2 h = S.half[e];
  U[h.x] = Cplx<double>{(pu + rv) + (hv ? 0.0 : self), pv - ru};
  if (h.y >= 0) {
    const double sg = E.T & 1 ? -1.0 : 1.0;
    U[h.y] = Cplx<double>{sg * (pu - rv), -sg * (pv + ru)};
  }
}

template <bool POLY>
__global__ void __launch_bounds__(32) k_snap_u(SnapArgs A) {
  const SnapDev& S = A.S;
  extern __shared__ __align__(16) double su_smem[];
  double* xs = su_smem;                       // nx sums
  double* tab = su_smem + ((S.nx + 1) & ~1);  // 32 rows
  const int al = blockIdx.x, lane = threadIdx.x;
  const int cols = POLY ? su_pcols(S.twojmax) : su_stride(S.cols), n = A.cnt[al];
  const int2* __restrict__ xsum = POLY ? S.psum : S.xsum;
  const size_t np = size_t(A.n) * A.cap;
  const double* pd = A.pd + size_t(al) * A.cap;
  for (int n0 = 0; n0 < max(n, 1); n0 += 32) {
    const int m = min(32, n - n0);
    if (lane < m) {
      const double* q = pd + n0 + lane;
      const double ar = q[PD_AR * np], ai = q[PD_AI * np], br = q[PD_BR * np], bi = q[PD_BI * np], w = q[PD_SF * np];
      if (POLY) su_row_p(S, tab + lane * cols, ar, ai, br, bi, w);
      else su_row(S.twojmax, tab + lane * cols, ar, ai, br, bi, w);
    }
    __syncwarp();
    for (int r0 = 0; r0 < S.nx; r0 += 96) {  // three sums per lane at once
      int2 s[3];
      double acc[3];
#pragma unroll
      for (int h = 0; h < 3; ++h) {
        const int r = r0 + 32 * h + lane;
        s[h] = r < S.nx ? __ldg(xsum + r) : int2{0, 0};
        acc[h] = r < S.nx && n0 > 0 ? xs[r] : 0.0;
      }
      if (r0 + 64 < S.nx) {
#pragma unroll 2
        for (int k = 0; k < m; ++k) {
          const double* t = tab + k * cols;
#pragma unroll
          for (int h = 0; h < 3; ++h) acc[h] = fma(t[s[h].x], t[s[h].y], acc[h]);
        }
      } else if (r0 + 32 < S.nx) {
        for (int k = 0; k < m; ++k) {
          const double* t = tab + k * cols;
#pragma unroll
          for (int h = 0; h < 2; ++h) acc[h] = fma(t[s[h].x], t[s[h].y], acc[h]);
        }
      } else {
        for (int k = 0; k < m; ++k) {
          const double* t = tab + k * cols;
          acc[0] = fma(t[s[0].x], t[s[0].y], acc[0]);
        }
      }
#pragma unroll
      for (int h = 0; h < 3; ++h)
        if (r0 + 32 * h + lane < S.nx) xs[r0 + 32 * h + lane] = acc[h];
    }
    __syncwarp();
  }
  Cplx<double>* U = static_cast<Cplx<double>*>(A.U) + size_t(al) * S.nh;
  for (int e = lane; e < S.ne; e += 32) su_store<POLY>(S, __ldg(S.eord + e), xs, S.wself, U);
}

// ------------------------------------------------------------------- Z, Y
// Lanes = atoms of a tile (ta of them; for ta < 32 the 32 / ta lane groups
// share a record's products), warps = tasks.  One (T, q) and sign of T owns
// Y_j(m, m') at (2m, 2m') = (-q -+ T, -q +- T) for every j, because Z_j at one
// (m, m') comes from products U_j1(m1, m1') U_j2(m - m1, m' - m1') that do not
// depend on j: each product is formed once (4 operations) and weighted by both
// Clebsch-Gordan factors for every j (2 each), where one Z at a time took 6 for
// each (compute_zi, sna_impl.hpp:197-283); for j1 = j2 the two orders of a pair
// of elements are one product.  The loops run over product lists, uniform over
// the lanes.  The longest lists are cut (SnapTables): each task writes its part
// of Y, and Y's readers sum the parts in order, so that a CTA's last warps end
// together and a tile can be shared by many CTAs (a warp alone issues one FP64
// instruction per 64 cycles, four or more share one per 19; 8,160 atoms, FP64:
// 2.49 ms with whole (T, q) as tasks, 1.88 with parts of 1/48, 2.15 and 1.95
// with 1/24 and 1/96; 64 atoms at twojmax 6: 52 -> 22 us).  Y_j = sum cY Z_j stays in
// registers; cY folds the linear
// coefficients with the (j+1)/(j1+1), (j+1)/(j2+1) weights of compute_dbidrj's
// three terms (sna_impl.hpp:330-539).
template <int NJ>
__device__ __forceinline__ void z_products(const ZRec& z, const SnapDev& S, const Cplx<double>* __restrict__ U, int str,
                                           int first, int step, Cplx<double>* Z) {
#pragma unroll
  for (int j = 0; j < NJ; ++j) Z[j] = Cplx<double>{0.0, 0.0};
  const int2* __restrict__ pl = S.prod + z.p0;
  const double* __restrict__ c = S.zc + z.c0;
#pragma unroll 2
  for (int k = first; k < z.np; k += step) {
    const int2 p = __ldg(pl + k);
    const Cplx<double> x = U[p.x * str], y = U[p.y * str];
    const double pr = fma(x.r, y.r, -x.i * y.i), pi = fma(x.r, y.i, x.i * y.r);
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
      const double w = __ldg(c + k * NJ + j);
      Z[j].r = fma(w, pr, Z[j].r);
      Z[j].i = fma(w, pi, Z[j].i);
    }
  }
}

// f(integral_constant<d>) for the uniform d: one block per value (f's marker
// keeps the compiler from folding them into an indexed, hence local-memory, y)
template <typename F>
__device__ __forceinline__ void at_offset(int d, F&& f) {
  if (d == 0) f(std::integral_constant<int, 0>{});
  else if (d == 1) f(std::integral_constant<int, 1>{});
  else if (d == 2) f(std::integral_constant<int, 2>{});
  else if (d == 3) f(std::integral_constant<int, 3>{});
  else if (d == 4) f(std::integral_constant<int, 4>{});
  else if (d == 5) f(std::integral_constant<int, 5>{});
  else if (d == 6) f(std::integral_constant<int, 6>{});
  else f(std::integral_constant<int, 7>{});
}

template <typename R>
__device__ __forceinline__ void shfl_add(Cplx<R>& z, int o) {
  z.r += __shfl_xor_sync(FULL_MASK, z.r, o);
  z.i += __shfl_xor_sync(FULL_MASK, z.i, o);
}

// a record's Z and its part of the task's Y (y[0]: the highest j)
template <int NM, int NJ, bool KEEP>
__device__ __forceinline__ void z_add(const ZRec& z, const SnapDev& S, const Cplx<double>* __restrict__ U, int str,
                                      const double* __restrict__ cY, int first, int step, Cplx<double>* y,
                                      Cplx<double>* zk) {
  Cplx<double> Z[NJ];
  z_products<NJ>(z, S, U, str, first, step, Z);
  double c[NJ];
#pragma unroll
  for (int j = 0; j < NJ; ++j) {
    c[j] = cY[z.t0 - j];
    if constexpr (KEEP) {
      for (int o = 32 / step; o < 32; o <<= 1) shfl_add(Z[j], o);
      if (first == 0) zk[size_t(z.z0 + j) * 32] = Z[j];
    }
  }
  at_offset(z.d, [&](auto dc) {
    constexpr int d = decltype(dc)::value;
    if constexpr (d + NJ <= NM) {
      asm volatile("// y + %0" ::"n"(d));
#pragma unroll
      for (int j = 0; j < NJ; ++j) {
        y[d + j].r = fma(c[j], Z[j].r, y[d + j].r);
        y[d + j].i = fma(c[j], Z[j].i, y[d + j].i);
      }
    }
  });
}

// a task's part of Y (y[0]: the highest j) to its slots
template <typename R, int NM>
__device__ __forceinline__ void y_store(const ZTask& K, const Cplx<R>* y, R* Yt, int ta) {
#pragma unroll
  for (int h = 0; h < NM; ++h)
    if (h <= K.kmax) {
      R* o = Yt + size_t(2) * (K.y0 + K.kmax - h) * ta;
      o[0] = y[h].r;
      o[ta] = y[h].i;
    }
}

// Y of half-grid element h (y: the atom's column of its tile), parts in order
template <typename R>
__device__ __forceinline__ Cplx<R> y_element(const SnapDev& S, int h, const R* y, int ta) {
  const int4 s = __ldg(S.ysrc + h);
  const R* p = y + size_t(2) * s.x * ta;
  Cplx<R> t{p[0], p[ta]};
  for (int k = 1; k < s.z; ++k) {
    p += size_t(2) * s.y * ta;
    t.r += p[0];
    t.i += p[ta];
  }
  return t;
}

// the tile's U, both halves of the grid, as [element][atom] with rows of ta + 1
template <typename R>
__device__ __forceinline__ void y_load_tile(const SnapArgs& A, int tile, int ta, Cplx<R>* U) {
  const SnapDev& S = A.S;
  const int str = ta + 1;
  for (int k = threadIdx.x; k < S.nh * ta; k += blockDim.x) {
    const int a = k / S.nh, h = k - a * S.nh, ga = tile * ta + a;
    const Cplx<R> u = ga < A.n ? static_cast<const Cplx<R>*>(A.U)[size_t(ga) * S.nh + h] : Cplx<R>{R(0), R(0)};
    const int4 f = __ldg(S.hfull + h);
    U[f.x * str + a] = u;
    if (f.y != f.x) U[f.y * str + a] = f.z > 0 ? Cplx<R>{u.r, -u.i} : Cplx<R>{-u.r, u.i};
  }
}

// FP64.  NM: most j of one (m, m') (5 up to twojmax 9, 8 up to 14); FULL: ta = 32
constexpr int SY_THREADS = 512;
template <int NM, bool KEEP, bool FULL>
__global__ void __launch_bounds__(SY_THREADS) k_snap_y(SnapArgs A) {
  const SnapDev& S = A.S;
  extern __shared__ __align__(16) unsigned char sy_smem[];
  __shared__ int s_next;
  Cplx<double>* U = reinterpret_cast<Cplx<double>*>(sy_smem);
  const int ta = FULL ? 32 : A.ta, str = ta + 1, tile = blockIdx.x / A.nsplit, split = blockIdx.x - tile * A.nsplit;
  const int lane = threadIdx.x & 31, at = FULL ? lane : lane % ta, sub = FULL ? 0 : lane / ta, nsub = FULL ? 1 : 32 / ta;
  const int al = tile * ta + at;
  if (threadIdx.x == 0) s_next = 0;
  y_load_tile(A, tile, ta, U);
  __syncthreads();
  const int ei = al < A.n ? S.map[A.type[A.first + al]] : 0;
  const double* cY = S.cY + size_t(ei) * S.nfull;
  double* Yt = static_cast<double*>(A.Y) + size_t(tile) * 2 * S.ny * ta + at;
  Cplx<double>* zk = reinterpret_cast<Cplx<double>*>(A.zkeep) + (KEEP ? size_t(al >> 5) * S.nz * 32 + (al & 31) : 0);
  const Cplx<double>* Ua = U + at;
  while (true) {
    int t = 0;
    if (lane == 0) t = atomicAdd(&s_next, 1);
    t = __shfl_sync(FULL_MASK, t, 0) * A.nsplit + split;  // tasks longest first
    if (t >= S.ntask) break;
    const ZTask K = S.task[t];
    Cplx<double> y[NM];
#pragma unroll
    for (int k = 0; k < NM; ++k) y[k] = Cplx<double>{0.0, 0.0};
#pragma unroll 1
    for (int r = K.rec0; r < K.rec1; ++r) {
      const ZRec z = S.rec[r];
      switch (z.nj) {  // uniform
        case 1: z_add<NM, 1, KEEP>(z, S, Ua, str, cY, sub, nsub, y, zk); break;
        case 2: z_add<NM, 2, KEEP>(z, S, Ua, str, cY, sub, nsub, y, zk); break;
        case 3: z_add<NM, 3, KEEP>(z, S, Ua, str, cY, sub, nsub, y, zk); break;
        case 4: z_add<NM, 4, KEEP>(z, S, Ua, str, cY, sub, nsub, y, zk); break;
        case 5: z_add<NM, 5, KEEP>(z, S, Ua, str, cY, sub, nsub, y, zk); break;
        default:
          if constexpr (NM > 5) {
            if (z.nj == 6) z_add<NM, 6, KEEP>(z, S, Ua, str, cY, sub, nsub, y, zk);
            else if (z.nj == 7) z_add<NM, 7, KEEP>(z, S, Ua, str, cY, sub, nsub, y, zk);
            else z_add<NM, 8, KEEP>(z, S, Ua, str, cY, sub, nsub, y, zk);
          }
      }
    }
    // the lane groups' parts (KEEP: every Z was completed already)
    for (int o = ta; o < 32 && !KEEP; o <<= 1)
#pragma unroll
      for (int k = 0; k < NM; ++k) shfl_add(y[k], o);
    if (sub == 0) y_store<double, NM>(K, y, Yt, ta);
  }
}

// FP32.  Here the FP64 pipe's slow cadence does not hide the rest, so
//  - the products of a task with equal nj and d form one group, whatever their
//    (j1, j2): cY is folded into the coefficients, Y is summed directly and the
//    309 groups (at twojmax 8) replace 1,285 records;
//  - the tables (200 KB) do not fit what the tile leaves of L1, so a task's
//    entries come as one stream through a shared buffer of the warp's own:
//    while one KB is worked on the next is on its way in registers;
//  - in large systems a lane takes two atoms (NA), so that every entry and its
//    addresses serve 64 atoms.
// Atoms of another element than the stream's are computed and not stored
// (one launch per element).
// Per 128,000 atoms: 3.77 ms with records and direct table reads, 2.47 with
// records streamed, 1.28 as it is with 16 warps, 1.23 with 24, 1.21 with packed
// multiply-adds: bound by the U operands from shared memory, 0.96 ms of wavefronts.
__host__ __device__ constexpr int zs_words(int nj) { return nj == 1 ? 2 : (nj <= 3 ? 4 : (nj <= 5 ? 8 : 16)); }
constexpr int ZS_CHUNK = 256;  // words per buffer
struct ZStream {
  const uint4* g;  // the chunk in registers
  uint4 r0, r1;
  uint4* buf;
  int cur;  // chunk in the buffer
  __device__ __forceinline__ void begin(const uint4* zs, int s0, int lane) {
    g = zs + s0 / 4 + lane;
    r0 = __ldg(g);
    r1 = __ldg(g + 32);
    cur = -1;
    next(lane);
  }
  __device__ __forceinline__ void next(int lane) {
    __syncwarp();
    buf[lane] = r0;
    buf[lane + 32] = r1;
    __syncwarp();
    g += 64;
    r0 = __ldg(g);
    r1 = __ldg(g + 32);
    ++cur;
  }
};
template <int NM, int NJ, int NA>
__device__ __forceinline__ void zg_add(const ZGrp& G, ZStream& st, const Cplx<float>* __restrict__ U, int str,
                                       int first, int step, Cplx<float> (*y)[NM]) {
  constexpr int W = zs_words(NJ);
  Cplx<float> Z[NA][NJ];
#pragma unroll
  for (int a = 0; a < NA; ++a)
#pragma unroll
    for (int j = 0; j < NJ; ++j) Z[a][j] = Cplx<float>{0.f, 0.f};
  int pos = G.w0, left = G.np;
  while (left > 0) {
    if (pos / ZS_CHUNK != st.cur) st.next(threadIdx.x & 31);
    const int m = min(left, (ZS_CHUNK - pos % ZS_CHUNK) / W);
    const unsigned* w = reinterpret_cast<const unsigned*>(st.buf) + pos % ZS_CHUNK;
#pragma unroll 4
    for (int k = first; k < m; k += step) {
      unsigned d[W];
      if constexpr (W == 2) {
        *reinterpret_cast<uint2*>(d) = *reinterpret_cast<const uint2*>(w + k * W);
      } else {
#pragma unroll
        for (int h = 0; h < (NJ + 4) / 4; ++h)
          reinterpret_cast<uint4*>(d)[h] = *reinterpret_cast<const uint4*>(w + k * W + 4 * h);
      }
      const Cplx<float>* px = U + (d[0] & 0xffffu) * str;
      const Cplx<float>* py = U + (d[0] >> 16) * str;
#pragma unroll
      for (int a = 0; a < NA; ++a) {
        const Cplx<float> x = px[32 * a], v = py[32 * a];
        const float pr = fmaf(x.r, v.r, -x.i * v.i), pi = fmaf(x.r, v.i, x.i * v.r);
#pragma unroll
        for (int j = 0; j < NJ; ++j) {
          const float c = __uint_as_float(d[1 + j]);
          const float2 t = __ffma2_rn(make_float2(c, c), make_float2(pr, pi), make_float2(Z[a][j].r, Z[a][j].i));
          Z[a][j] = Cplx<float>{t.x, t.y};
        }
      }
    }
    pos += m * W;
    left -= m;
  }
  at_offset(G.d, [&](auto dc) {
    constexpr int d = decltype(dc)::value;
    if constexpr (d + NJ <= NM) {
      asm volatile("// y + %0" ::"n"(d));
#pragma unroll
      for (int a = 0; a < NA; ++a)
#pragma unroll
        for (int j = 0; j < NJ; ++j) {
          y[a][d + j].r += Z[a][j].r;
          y[a][d + j].i += Z[a][j].i;
        }
    }
  });
}

__host__ __device__ constexpr int sy32_threads(int na) { return na == 2 ? 768 : 384; }
template <int NM, int NA, bool FULL>
__global__ void __launch_bounds__(sy32_threads(NA), NA == 2 ? 1 : 2) k_snap_y32(SnapArgs A, int elem) {
  const SnapDev& S = A.S;
  extern __shared__ __align__(16) unsigned char sy_smem[];
  __shared__ int s_next;
  Cplx<float>* U = reinterpret_cast<Cplx<float>*>(sy_smem);
  const int ta = FULL ? 32 * NA : A.ta, str = ta + 1, tile = blockIdx.x / A.nsplit, split = blockIdx.x - tile * A.nsplit;
  const int lane = threadIdx.x & 31, at = FULL ? lane : lane % ta, sub = FULL ? 0 : lane / ta, nsub = FULL ? 1 : 32 / ta;
  if (threadIdx.x == 0) s_next = 0;
  y_load_tile(A, tile, ta, U);
  __syncthreads();
  bool mine[NA];
#pragma unroll
  for (int a = 0; a < NA; ++a) {
    const int al = tile * ta + at + 32 * a;
    mine[a] = sub == 0 && al < A.n && S.map[A.type[A.first + al]] == elem;
  }
  float* Yt = static_cast<float*>(A.Y) + size_t(tile) * 2 * S.ny * ta + at;
  const Cplx<float>* Ua = U + at;
  ZStream st;
  st.buf = reinterpret_cast<uint4*>(sy_smem + ((sizeof(Cplx<float>) * size_t(S.nuf) * str + 15) & ~size_t(15))) +
           (threadIdx.x >> 5) * (ZS_CHUNK / 4);
  const uint4* zs = S.zs + size_t(elem) * S.zs_n;
  while (true) {
    int t = 0;
    if (lane == 0) t = atomicAdd(&s_next, 1);
    t = __shfl_sync(FULL_MASK, t, 0) * A.nsplit + split;  // tasks longest first
    if (t >= S.ntask) break;
    const ZTask K = S.task[t];
    st.begin(zs, K.s0, lane);
    Cplx<float> y[NA][NM];
#pragma unroll
    for (int a = 0; a < NA; ++a)
#pragma unroll
      for (int k = 0; k < NM; ++k) y[a][k] = Cplx<float>{0.f, 0.f};
#pragma unroll 1
    for (int g = K.grp0; g < K.grp1; ++g) {
      const ZGrp G = S.grp[g];
      switch (G.nj) {  // uniform
        case 1: zg_add<NM, 1, NA>(G, st, Ua, str, sub, nsub, y); break;
        case 2: zg_add<NM, 2, NA>(G, st, Ua, str, sub, nsub, y); break;
        case 3: zg_add<NM, 3, NA>(G, st, Ua, str, sub, nsub, y); break;
        case 4: zg_add<NM, 4, NA>(G, st, Ua, str, sub, nsub, y); break;
        case 5: zg_add<NM, 5, NA>(G, st, Ua, str, sub, nsub, y); break;
        default:
          if constexpr (NM > 5) {
            if (G.nj == 6) zg_add<NM, 6, NA>(G, st, Ua, str, sub, nsub, y);
            else if (G.nj == 7) zg_add<NM, 7, NA>(G, st, Ua, str, sub, nsub, y);
            else zg_add<NM, 8, NA>(G, st, Ua, str, sub, nsub, y);
          }
      }
    }
    for (int o = ta; o < 32; o <<= 1)  // the lane groups' parts
#pragma unroll
      for (int k = 0; k < NM; ++k) shfl_add(y[0][k], o);
#pragma unroll
    for (int a = 0; a < NA; ++a)
      if (mine[a]) y_store<float, NM>(K, y[a], Yt + 32 * a, ta);
  }
}

// ------------------------------------------------------------- pair forces
// Lanes = pairs, pooled over the CTA's atoms.  With a^q and w b^T = u + i v, and
// E = 2N (Y+ + (-1)^T Y-), O = 2N (Y+ - (-1)^T Y-) of an entry (formed when Y is
// loaded), twice the real part of conj(U) Y over both signs of T is
// u Re(a^q E) + v Im(a^q O) times P_k.  So Phi = sum_j 2 sum_half w
// Re(conj(U_j) Y_j) of one neighbour is sum_T u_T Re(Eh_T) + v_T Im(Oh_T) with
// Eh_T = sum_q a^q sum_k E P_k and Oh_T likewise, and the pair force needs only
// Phi and its gradient in (a, b):
//   F_k = dsfac u_k Phi + sfac dPhi/dp dp/dr_k + the r^-14 term,
// which equals sum_k beta_k dB_k/dr_ij of the reference.  About 1,250
// operations per neighbour at twojmax 8 (the layered adjoint took 4,100, half
// its lanes idle).  f_j -= F_ij with FP64 atomics (j may be a ghost;
// update_force follows) and f_i += sum_j F_ij in a fixed order.
//
// With twojmax a constant (2, 4, 6, 8) every loop is unrolled and the recurrences'
// constants are operands; other twojmax take the loops.  The mixed form forms the
// powers of a and b from their 48-bit values, keeps what the sum over T rounds off,
// sums even and odd q apart and takes the gradient's radial part off: 1,000 operations
// more (rms error against the FP64 form, W bcc 2,000 atoms at 0.05 A: 7.5e-6 eV/A without,
// 5.5e-6 with the first two, 4.9e-6 with all; U and Y alone account for a third).
// Bound by instruction issue and the latency of the phases; per 128,000 atoms
// mixed 0.88 ms as loops, 0.51 unrolled with the extra operations; 8,160 atoms FP64
// 0.64 and 0.55 (0.50 of FP64 issue).
constexpr int SF_THREADS = 256;
constexpr int SF_ATOMS = 8;

// Constants of the recurrences with T + q + 2k < SF_JMAX, in constant memory where
// an unrolled loop has them as operands (as in SnapDev::AB; k = 0 has no B)
constexpr int SF_JMAX = 8;
template <typename R>
struct JacTable {
  R a[SF_JMAX][SF_JMAX][SF_JMAX / 2], b[SF_JMAX][SF_JMAX][SF_JMAX / 2];
  constexpr JacTable() : a{}, b{} {
    for (int T = 0; T < SF_JMAX; ++T)
      for (int q = 0; q < SF_JMAX; ++q)
        for (int k = 0; k < SF_JMAX / 2; ++k) {
          const double s = 2.0 * k + T + q;
          a[T][q][k] = R(k == 0 ? (q - T) / (s + 2.0) : double(q * q - T * T) / (s * (s + 2.0)));
          b[T][q][k] = R(k == 0 ? 0.0 : 4.0 * k * (k + T) * (k + q) * (k + T + q) / (s * s * (s + 1.0) * (s - 1.0)));
        }
  }
};
static __constant__ JacTable<double> c_jac = JacTable<double>();
static __constant__ JacTable<float> c_jac32 = JacTable<float>();
template <typename R>
__device__ __forceinline__ R jac_a(int T, int q, int k) {
  if constexpr (sizeof(R) == sizeof(float)) return c_jac32.a[T][q][k];
  else return c_jac.a[T][q][k];
}
template <typename R>
__device__ __forceinline__ R jac_b(int T, int q, int k) {
  if constexpr (sizeof(R) == sizeof(float)) return c_jac32.b[T][q][k];
  else return c_jac.b[T][q][k];
}

// s + c += t, the sum of T's terms: what the addition rounds off goes to c
template <typename R>
struct TSum {
  R s = 0, c = 0;
  __device__ __forceinline__ void add(R t) {
    if constexpr (sizeof(R) == sizeof(float)) {
      const R z = add_rn(s, t), y = sub_rn(z, s);
      c = add_rn(c, add_rn(sub_rn(s, sub_rn(z, y)), sub_rn(t, y)));
      s = z;
    } else {
      s += t;
    }
  }
  __device__ __forceinline__ R value() const { return s + c; }
};

// one T's sums over q: Re Eh, Im Oh; the same with P'; dEh/da, dOh/da
template <typename R>
struct QSum {
  R er = 0, oi = 0, xer = 0, xoi = 0, e1r = 0, e1i = 0, o1r = 0, o1i = 0;
};

// T as a constant and as a variable (the compiler does not unroll so long a loop)
template <int T>
struct FixedT {
  static constexpr int value = T;
};
struct AnyT {
  int value;
};

// JC: twojmax (loops unrolled), or -1: any up to 14
template <typename R, int JC>
__global__ void __launch_bounds__(SF_THREADS, sizeof(R) == 4 ? 3 : 2) k_snap_force(SnapArgs A) {
  const SnapDev& S = A.S;
  constexpr bool kF64 = sizeof(R) == sizeof(double);
  static_assert(JC <= SF_JMAX, "recurrence constants");
  constexpr int NQ = JC >= 0 ? JC + 1 : 15, kUnroll = JC >= 0 ? 16 : 1;
  extern __shared__ __align__(16) unsigned char sf_smem[];
  __shared__ int s_off[SF_ATOMS + 1];
  __shared__ double s_sum[SF_ATOMS][3];
  const int J = JC >= 0 ? JC : S.twojmax, ny = 4 * S.ne, tid = threadIdx.x;
  const int apc = A.apc, a0 = blockIdx.x * apc, na = min(apc, A.n - a0);
  // groups of T on separate warps (small systems): each forms a part of F
  const int nthr = blockDim.x / A.tsplit, grp = tid / nthr, gt = tid - grp * nthr;
  R* ys = reinterpret_cast<R*>(sf_smem);                                   // apc x ny
  double* fs = reinterpret_cast<double*>(sf_smem + ((size_t(apc) * ny * sizeof(R) + 15) & ~size_t(15)));  // blockDim x 3
  const int ta = A.ta;
  const int la = tid % na, ls = blockDim.x / na, ga = a0 + la;
  const R* Yt = static_cast<const R*>(A.Y) + size_t(ga / ta) * 2 * S.ny * ta + ga % ta;
  for (int e = tid / na; tid < ls * na && e < S.ne; e += ls) {
    const int2 h = __ldg(S.half + e);
    const R N = kF64 ? R(S.ent[e].N) : R(S.ent[e].Nf), N2 = N + N;
    const Cplx<R> p = y_element(S, h.x, Yt, ta);
    R* o = ys + la * ny + 4 * e;
    if (h.y >= 0) {
      const Cplx<R> m = y_element(S, h.y, Yt, ta);
      const R sg = __ldg(S.hfull + h.x).z > 0 ? R(1) : R(-1);
      o[0] = N2 * fma(sg, m.r, p.r);
      o[1] = N2 * fma(sg, m.i, p.i);
      o[2] = N2 * fma(-sg, m.r, p.r);
      o[3] = N2 * fma(-sg, m.i, p.i);
    } else {  // q = 0 (the -T element is the inversion of the +T one), T = 0, or both
      const int T = S.ent[e].T, q = S.ent[e].q;
      o[0] = (T + q > 0 ? N2 : N) * p.r;
      o[1] = q > 0 ? N2 * p.i : R(0);
      o[2] = R(0);
      o[3] = T > 0 ? N2 * p.i : R(0);
    }
  }
  if (tid == 0) {
    int o = 0;
    for (int a = 0; a < na; ++a) {
      s_off[a] = o;
      o += A.cnt[a0 + a];
    }
    s_off[na] = o;
  }
  if (tid < 3 * SF_ATOMS) s_sum[tid / 3][tid % 3] = 0.0;
  __syncthreads();
  const int total = s_off[na];
  const size_t np = size_t(A.n) * A.cap;
  const R* AB = kF64 ? reinterpret_cast<const R*>(S.AB) : reinterpret_cast<const R*>(S.AB_f);
  const unsigned mask = A.tsplit > 1 ? unsigned(A.tmask[grp]) : 0xffffffffu;
  for (int s0 = 0; s0 < total; s0 += nthr) {
    const int s = s0 + gt;
    double F[3] = {0.0, 0.0, 0.0};
    size_t p = 0;
    if (s < total) {
      int a = 0;
      while (s >= s_off[a + 1]) ++a;
      p = size_t(a0 + a) * A.cap + (s - s_off[a]);
      const double* qd = A.pd + p;
      const R* qr = static_cast<const R*>(A.pr) + p;
      const R ar = qr[PR_AR * np], ai = qr[PR_AI * np], br = qr[PR_BR * np], bi = qr[PR_BI * np];
      // powers of a and b; in the mixed form from the 48-bit a and b and rounded once
      R pq[NQ], rq[NQ];
      pq[0] = R(1);
      rq[0] = R(0);
      R x;
      F2 b0{}, b1{}, nb1{}, u2{}, v2{};
      const float one = f2_base(1.f);
      if constexpr (kF64) {
#pragma unroll
        for (int q = 1; q < NQ; ++q) {
          pq[q] = fma(pq[q - 1], ar, -rq[q - 1] * ai);
          rq[q] = fma(pq[q - 1], ai, rq[q - 1] * ar);
        }
        x = fma(ar, ar, ai * ai) - fma(br, br, bi * bi);
      } else {
        const F2 c0{ar, qr[PR_ARL * np]}, c1{ai, qr[PR_AIL * np]}, nc1{-c1.h, -c1.l};
        b0 = F2{br, qr[PR_BRL * np]};
        b1 = F2{bi, qr[PR_BIL * np]};
        nb1 = F2{-b1.h, -b1.l};
        F2Sum sx{one, 0.f};
        sx.add(c0, c0);
        sx.add(c1, c1);
        sx.add(F2{-b0.h, -b0.l}, b0);
        sx.add(nb1, b1);
        x = sx.value(one).h;
        F2 pk{1.f, 0.f}, rk{0.f, 0.f};
#pragma unroll
        for (int q = 1; q < NQ; ++q) {
          if (q == 1) {
            pk = c0;
            rk = c1;
          } else {
            f2_cmul(pk, rk, c0, c1, nc1, one);
          }
          pq[q] = pk.h;
          rq[q] = rk.h;
        }
        u2 = F2{1.f, 0.f};
      }
      R u = R(1), v = R(0), um = R(0), vm = R(0);  // b^T, b^(T-1)
      TSum<R> phi, gx, gar, gai, gbr, gbi;
      const R* Y = ys + a * ny;
      const R* ab = AB;
      auto one_T = [&](auto t) __attribute__((always_inline)) {
        const int T = t.value;
        const int nT = (J - T + 2) * (J - T + 2) / 4;  // entries of T
        if (mask >> T & 1) {
          QSum<R> qs[kF64 ? 1 : 2];  // mixed form: of even and of odd q
          int e = 0;
#pragma unroll
          for (int q = 0; q < NQ; ++q) {
            if (q > J - T) break;
            const int km = (J - T - q) / 2;
            QSum<R>& Q = qs[kF64 ? 0 : q & 1];
            const R* y = Y + 4 * e;
            R g0 = y[0], g1 = y[1], g2 = y[2], g3 = y[3];  // sum_k E P_k, O P_k
            R h0 = 0, h1 = 0, h2 = 0, h3 = 0;              // sum_k E P'_k, O P'_k
            if (km > 0) {
              R pk = x - (JC >= 0 ? jac_a<R>(T, q, 0) : ab[2 * e]), pm = R(1), dk = R(1), dm = R(0);
              h0 = y[4];
              h1 = y[5];
              h2 = y[6];
              h3 = y[7];
              g0 = fma(h0, pk, g0);
              g1 = fma(h1, pk, g1);
              g2 = fma(h2, pk, g2);
              g3 = fma(h3, pk, g3);
#pragma unroll kUnroll
              for (int k = 2; k <= km; ++k) {
                const R t = x - (JC >= 0 ? jac_a<R>(T, q, k - 1) : ab[2 * (e + k - 1)]);
                const R c = JC >= 0 ? jac_b<R>(T, q, k - 1) : ab[2 * (e + k - 1) + 1];
                const R pn = fma(t, pk, -c * pm), dn = fma(t, dk, fma(-c, dm, pk));
                pm = pk;
                pk = pn;
                dm = dk;
                dk = dn;
                const R* yk = y + 4 * k;
                g0 = fma(yk[0], pk, g0);
                g1 = fma(yk[1], pk, g1);
                h0 = fma(yk[0], dk, h0);
                h1 = fma(yk[1], dk, h1);
                if (T > 0) {
                  g2 = fma(yk[2], pk, g2);
                  g3 = fma(yk[3], pk, g3);
                  h2 = fma(yk[2], dk, h2);
                  h3 = fma(yk[3], dk, h3);
                }
              }
            }
            Q.er = fma(pq[q], g0, Q.er);
            Q.xer = fma(pq[q], h0, Q.xer);
            if (q > 0) {
              const R qp = R(q) * pq[q - 1], qr1 = R(q) * rq[q - 1];
              Q.er = fma(-rq[q], g1, Q.er);
              Q.xer = fma(-rq[q], h1, Q.xer);
              Q.e1r = fma(qp, g0, fma(-qr1, g1, Q.e1r));
              Q.e1i = fma(qp, g1, fma(qr1, g0, Q.e1i));
              if (T > 0) {
                Q.oi = fma(rq[q], g2, Q.oi);
                Q.xoi = fma(rq[q], h2, Q.xoi);
                Q.o1r = fma(qp, g2, fma(-qr1, g3, Q.o1r));
                Q.o1i = fma(qp, g3, fma(qr1, g2, Q.o1i));
              }
            }
            if (T > 0) {
              Q.oi = fma(pq[q], g3, Q.oi);
              Q.xoi = fma(pq[q], h3, Q.xoi);
            }
            e += km + 1;
          }
          auto both = [&](auto f) { return kF64 ? qs[0].*f : qs[0].*f + qs[kF64 ? 0 : 1].*f; };
          const R er = both(&QSum<R>::er), oi = both(&QSum<R>::oi), xer = both(&QSum<R>::xer), xoi = both(&QSum<R>::xoi);
          const R e1r = both(&QSum<R>::e1r), e1i = both(&QSum<R>::e1i), o1r = both(&QSum<R>::o1r), o1i = both(&QSum<R>::o1i);
          phi.add(fma(u, er, v * oi));
          gx.add(fma(u, xer, v * xoi));
          gar.add(fma(u, e1r, v * o1i));
          gai.add(fma(-u, e1i, v * o1r));
          if (T > 0) {
            const R tu = R(T) * um, tv = R(T) * vm;
            gbr.add(fma(tu, er, tv * oi));
            gbi.add(fma(tu, oi, -tv * er));
          }
        }
        Y += 4 * nT;
        ab += 2 * nT;
        um = u;
        vm = v;
        if constexpr (kF64) {
          const R un = fma(u, br, -v * bi);
          v = fma(u, bi, v * br);
          u = un;
        } else {
          f2_cmul(u2, v2, b0, b1, nb1, one);
          u = u2.h;
          v = v2.h;
        }
      };
      if constexpr (JC >= 0) {
        [&]<int... T>(std::integer_sequence<int, T...>) {
          (one_T(FixedT<T>{}), ...);
        }(std::make_integer_sequence<int, JC + 1>{});
      } else {
#pragma unroll 1
        for (int T = 0; T <= J; ++T) one_T(AnyT{T});
      }
      const R gx2 = gx.value() + gx.value();
      R ga = fma(ar, gx2, gar.value()), gb = fma(ai, gx2, gai.value());
      R gc = fma(-br, gx2, gbr.value()), gd = fma(-bi, gx2, gbi.value());
      // |a|^2 + |b|^2 = 1, so the gradient's part along (a, b), which is the larger one (a
      // degree j times Phi), drops out of the force below. Rounded with the rest it left a
      // third of the mixed form's error; in the FP64 form it meets the rounding of the
      // reference's derivatives, large where theta0 nears pi (no switching: 1e-12 to 1e-11
      // of the RMS force, the layer recursion too; 1e-14 without it). Taken off before the
      // last roundings: ga = ar (gx2 - rho) + gar, gc = -br (gx2 + rho) + gbr
      const R rho = fma(ar, ga, fma(ai, gb, fma(br, gc, bi * gd)));
      if constexpr (kF64) {
        const R wa = gx2 - rho, wb = -gx2 - rho;
        ga = fma(ar, wa, gar.s);
        gb = fma(ai, wa, gai.s);
        gc = fma(br, wb, gbr.s);
        gd = fma(bi, wb, gbi.s);
      } else {
        const F2 wa = f2_two_sum(gx.s + gx.s, -rho), wb = f2_two_sum(-gx.s - gx.s, -rho);
        const R la = wa.l + (gx.c + gx.c), lb = wb.l - (gx.c + gx.c);
        ga = fma(ar, wa.h, gar.s) + fma(ar, la, gar.c);
        gb = fma(ai, wa.h, gai.s) + fma(ai, la, gai.c);
        gc = fma(br, wb.h, gbr.s) + fma(br, lb, gbr.c);
        gd = fma(bi, wb.h, gbi.s) + fma(bi, lb, gbi.c);
      }
      const R cp = qr[PR_DSF * np] * phi.value();
      const R uk[3] = {qr[PR_UX * np], qr[PR_UY * np], qr[PR_UZ * np]};
      if constexpr (kF64) {
        const double sf = qd[PD_SF * np];
#pragma unroll
        for (int d = 0; d < 3; ++d)
          F[d] = fma(cp, uk[d], sf * fma(ga, qr[(PF_DAR + d) * np],
                                         fma(gb, qr[(PF_DAI + d) * np],
                                             fma(gc, qr[(PF_DBR + d) * np], gd * qr[(PF_DBI + d) * np]))));
      } else {
        // along u_k through theta0 and s / r, then the direct terms
        const R sf = qr[PR_SF * np], c1 = qr[PR_C1 * np], gr = qr[PR_GR * np], r0 = sf * qr[PR_R0 * np];
        const R rad = fma(sf, fma(c1, ga, gr * fma(-uk[2], gb, fma(uk[1], gc, -uk[0] * gd))), cp);
        F[0] = double(fma(rad, uk[0], -r0 * gd));
        F[1] = double(fma(rad, uk[1], r0 * gc));
        F[2] = double(fma(rad, uk[2], -r0 * gb));
      }
    }
    if (A.tsplit > 1) {  // the groups' parts, in a fixed order
      for (int d = 0; d < 3; ++d) fs[3 * tid + d] = F[d];
      __syncthreads();
      if (grp == 0)
        for (int g = 1; g < A.tsplit; ++g)
          for (int d = 0; d < 3; ++d) F[d] += fs[3 * (g * nthr + gt) + d];
      __syncthreads();
    }
    if (grp == 0) {
      if (s < total) {
        const double* qd = A.pd + p;
        F[0] += qd[PD_FX * np];
        F[1] += qd[PD_FY * np];
        F[2] += qd[PD_FZ * np];
        double* fj = A.f + 3 * size_t(A.pj[p]);
        for (int d = 0; d < 3; ++d) atomicAdd(fj + d, -F[d]);
      }
      for (int d = 0; d < 3; ++d) fs[3 * gt + d] = F[d];
    }
    __syncthreads();
    // f_i: four lanes take every fourth neighbour
    if (tid < 32 * ((12 * na + 31) / 32)) {
      const int a = min(tid / 12, na - 1), d = tid % 12 / 4, l = tid & 3;
      const int b0 = max(s_off[a] - s0, 0), b1 = min(s_off[a + 1] - s0, nthr);
      double t = 0.0;
      for (int k = b0 + l; k < b1; k += 4) t += fs[3 * k + d];
      t += __shfl_xor_sync(FULL_MASK, t, 1);
      t += __shfl_xor_sync(FULL_MASK, t, 2);
      if (l == 0 && tid < 12 * na) s_sum[a][d] += t;
    }
    __syncthreads();
  }
  if (tid < 3 * na) {
    const int a = tid / 3, d = tid - 3 * a;
    atomicAdd(A.f + 3 * size_t(A.first + a0 + a) + d, s_sum[a][d]);
  }
}

// ------------------------------------------------------------------ energy
// beta_0 + (2/3) sum_j sum_half w Re(conj(U) Y) (B is cubic in U, so
// <U, dB/dU> = 3B) plus 1.25e5 / r^12 per inside pair; one warp per atom.
static __global__ void __launch_bounds__(128) k_snap_energy(SnapArgs A) {
  const SnapDev& S = A.S;
  const int lane = threadIdx.x & 31, al = blockIdx.x * 4 + (threadIdx.x >> 5);
  if (al >= A.n) return;
  const int ta = A.ta;
  const double* Y = static_cast<const double*>(A.Y) + size_t(al / ta) * 2 * S.ny * ta + al % ta;
  const Cplx<double>* U = static_cast<const Cplx<double>*>(A.U) + size_t(al) * S.nh;
  double acc = 0.0;
  for (int h = lane; h < S.nh; h += 32) {
    const Cplx<double> y = y_element(S, h, Y, ta), u = U[h];
    const int4 f = __ldg(S.hfull + h);
    acc += f.x == f.y ? 0.5 * (y.r * u.r) : fma(y.r, u.r, y.i * u.i);
  }
  const size_t np = size_t(A.n) * A.cap;
  const double* ep = A.pd + PD_EP * np + size_t(al) * A.cap;
  const int n = A.cnt[al];
  for (int k = lane; k < n; k += 32) acc += 1.5 * ep[k];
  acc = warp_sum(acc);
  if (lane == 0) {
    const int i = A.first + al;
    A.eatom[i] = S.beta0[S.map[A.type[i]]] + (2.0 / 3.0) * acc;
  }
}

// ----------------------------------------------------------------- adjoint
// For every full triple t = (j1, j2, j), with Z_t as k_snap_y kept it,
//   P_t = 2 sum_half w Re(conj(U_j) Z_t)        (= B_k when t is idxj triple k)
//   Q_t = 2 sum_half w Re(conj(D_j) Z_t),  D = sum_nb dU'_nb . (g_i - g_j)
// so that d/dbeta_k [sum_atoms g . F] over this atom's pairs is
// Q_t1 + (j+1)/(j1+1) Q_t2 + (j+1)/(j2+1) Q_t3 (compute_dbidrj's three terms,
// sna_impl.hpp:330-570, contracted with the loss gradient before the sum over
// k instead of after it).
//
// k_snap_dt: D as k_snap_u forms X, from each neighbour's table row and its
// derivative along g_i - g_j.  The rows hold u x^k and v x^k, the same for every q
// (columns as k_snap_u32's), and the sums are combined into the polynomials' once
// per atom: 310 FP64 instructions for 32 neighbours' rows where the products with
// every P_k took 720, and half the table (10,360 atoms in 28 calls: 2.76 -> 1.59 ms).
__device__ __forceinline__ void sd_row(const SnapDev& S, double* t, double* dt, double ar, double ai, double br,
                                       double bi, double w, double tar, double tai, double tbr, double tbi,
                                       double tw) {
  const int J = S.twojmax;
  double *col = t + 2 * (J + 1), *dcol = dt + 2 * (J + 1);
  const double x = fma(ar, ar, ai * ai) - fma(br, br, bi * bi);
  const double dx = 2.0 * (fma(ar, tar, ai * tai) - fma(br, tbr, bi * tbi));
  double p = 1.0, r = 0.0, u = w, v = 0.0, dp = 0.0, dr = 0.0, du = tw, dv = 0.0;
#pragma unroll 1
  for (int q = 0; q <= J; ++q) {
    t[2 * q] = p;
    t[2 * q + 1] = r;
    dt[2 * q] = dp;
    dt[2 * q + 1] = dr;
    double uk = u, vk = v, duk = du, dvk = dv;
#pragma unroll 1
    for (int k = 0; k <= (J - q) / 2; ++k) {
      *col++ = uk;
      *col++ = vk;
      *dcol++ = duk;
      *dcol++ = dvk;
      duk = fma(duk, x, uk * dx);
      dvk = fma(dvk, x, vk * dx);
      uk *= x;
      vk *= x;
    }
    const double dpn = fma(dp, ar, fma(-dr, ai, fma(p, tar, -r * tai)));
    const double drn = fma(dp, ai, fma(dr, ar, fma(p, tai, r * tar)));
    const double dun = fma(du, br, fma(-dv, bi, fma(u, tbr, -v * tbi)));
    const double dvn = fma(du, bi, fma(dv, br, fma(u, tbi, v * tbr)));
    const double pn = fma(p, ar, -r * ai), un = fma(u, br, -v * bi);
    r = fma(p, ai, r * ar);
    v = fma(u, bi, v * br);
    p = pn;
    u = un;
    dp = dpn;
    dr = drn;
    du = dun;
    dv = dvn;
  }
}

static __global__ void __launch_bounds__(32) k_snap_dt(SnapArgs A) {
  const SnapDev& S = A.S;
  extern __shared__ __align__(16) double sd_smem[];
  double* xs = sd_smem;
  double* tab = sd_smem + ((S.nx + 1) & ~1);
  const int al = blockIdx.x, lane = threadIdx.x, i = A.first + al;
  const int cols = su_stride(S.cols), n = A.cnt[al];
  const size_t np = size_t(A.n) * A.cap;
  const double gix = A.g[3 * i], giy = A.g[3 * i + 1], giz = A.g[3 * i + 2];
  for (int n0 = 0; n0 < max(n, 1); n0 += 32) {
    const int m = min(32, n - n0);
    if (lane < m) {
      const size_t p = size_t(al) * A.cap + n0 + lane;
      const double* q = A.pd + p;
      const double* w = static_cast<const double*>(A.pr) + p;
      // the pair's reaction force lands on j's owner (newton) or nowhere
      const int j = A.pj[p];
      const int jo = j < A.n_local ? j : (A.newton ? A.ghost_owner[j - A.n_local] : -1);
      const double dx = gix - (jo >= 0 ? A.g[3 * jo] : 0.0), dy = giy - (jo >= 0 ? A.g[3 * jo + 1] : 0.0),
                   dz = giz - (jo >= 0 ? A.g[3 * jo + 2] : 0.0);
      auto along = [&](int f) { return fma(w[f * np], dx, fma(w[(f + 1) * np], dy, w[(f + 2) * np] * dz)); };
      double* row = tab + 2 * lane * cols;
      sd_row(S, row, row + cols, w[PR_AR * np], w[PR_AI * np], w[PR_BR * np], w[PR_BI * np], q[PD_SF * np],
             along(PF_DAR), along(PF_DAI), along(PF_DBR), along(PF_DBI), w[PR_DSF * np] * along(PR_UX));
    }
    __syncwarp();
    for (int r = lane; r < S.nx; r += 32) {
      const int2 s = __ldg(S.xsum + r);
      double acc = n0 > 0 ? xs[r] : 0.0;
      for (int k = 0; k < m; ++k) {
        const double* t = tab + 2 * k * cols;
        const double* d = t + cols;
        acc = fma(d[s.x], t[s.y], fma(t[s.x], d[s.y], acc));
      }
      xs[r] = acc;
    }
    __syncwarp();
  }
  for (int e = lane; e < S.ne; e += 32) su_store<false>(S, __ldg(S.eord + e), xs, 0.0, A.D + size_t(al) * S.nh);
}

// half-grid elements of U and D, weighted (2, or 1 for the self-inverse ones,
// which are listed with an equal inversion), atom by atom -> lanes = atoms
static __global__ void __launch_bounds__(256) k_snap_half(SnapArgs A) {
  const SnapDev& S = A.S;
  const long long k = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int at = int(k & 31), tiles = (A.n + 31) / 32;
  const long long th = k >> 5;
  if (th >= (long long)tiles * S.nh) return;
  const int tile = int(th / S.nh), h = int(th - (long long)tile * S.nh), al = tile * 32 + at;
  const int4 f = S.hfull[h];
  const double w = f.x == f.y ? 1.0 : 2.0;
  for (int d = 0; d < 2; ++d) {
    const Cplx<double>* src = d ? A.D : static_cast<const Cplx<double>*>(A.U);
    const Cplx<double> u = al < A.n ? src[size_t(al) * S.nh + h] : Cplx<double>{0.0, 0.0};
    A.H[((size_t(tile) * 2 + d) * S.nh + h) * 32 + at] = Cplx<double>{w * u.r, w * u.i};
  }
}

// lanes = atoms, a warp per triple
static __global__ void __launch_bounds__(256) k_snap_pq(SnapArgs A) {
  const SnapDev& S = A.S;
  const int lane = threadIdx.x & 31, tile = blockIdx.x, t = blockIdx.y * 8 + (threadIdx.x >> 5);
  if (t >= S.nfull) return;
  const int al = tile * 32 + lane;
  const Cplx<double>* Z = reinterpret_cast<const Cplx<double>*>(A.zkeep) + size_t(tile) * S.nz * 32 + lane;
  const Cplx<double>* U = A.H + size_t(tile) * 2 * S.nh * 32 + lane;
  const Cplx<double>* D = U + size_t(S.nh) * 32;
  double p = 0.0, q = 0.0;
  for (int k = S.zt0[t]; k < S.zt0[t + 1]; ++k) {
    const int2 c = __ldg(S.zt + k);
    const Cplx<double> z = Z[size_t(c.x) * 32], u = U[size_t(c.y) * 32], d = D[size_t(c.y) * 32];
    p = fma(u.r, z.r, fma(u.i, z.i, p));
    q = fma(d.r, z.r, fma(d.i, z.i, q));
  }
  if (al < A.n) {
    const size_t i = size_t(A.first + al), n = size_t(A.n_local);
    A.adj[size_t(t) * n + i] = p;
    A.adj[size_t(S.nfull + t) * n + i] = q;
    if (t == 0) A.adj[size_t(2 * S.nfull) * n + i] = 1.0;  // atom count column (beta_0)
  }
}

// ---------------------------------------------------------------- launches
inline size_t snap_y_smem(const SnapDev& S, int ta, bool fp64) {
  const size_t u = ((fp64 ? 16 : 8) * size_t(S.nuf) * (ta + 1) + 15) & ~size_t(15);
  return u + (fp64 ? 0 : size_t(sy32_threads(ta == 64 ? 2 : 1)) / 32 * ZS_CHUNK * 4);
}

template <int NM, bool KEEP, bool FULL>
void launch_y(const SnapArgs& A, cudaStream_t s) {
  const int tiles = (A.n + A.ta - 1) / A.ta;
  allow_dyn_smem(k_snap_y<NM, KEEP, FULL>);
  k_snap_y<NM, KEEP, FULL><<<tiles * A.nsplit, SY_THREADS, snap_y_smem(A.S, A.ta, true), s>>>(A);
  EMD_CHECK_LAUNCH();
}
template <int NM>
void launch_y(const SnapArgs& A, cudaStream_t s) {
  if (A.zkeep) {
    if (A.ta == 32) launch_y<NM, true, true>(A, s);
    else launch_y<NM, true, false>(A, s);
  } else {
    if (A.ta == 32) launch_y<NM, false, true>(A, s);
    else launch_y<NM, false, false>(A, s);
  }
}
template <int NM, int NA, bool FULL>
void launch_y32(const SnapArgs& A, cudaStream_t s) {
  const int tiles = (A.n + A.ta - 1) / A.ta;
  allow_dyn_smem(k_snap_y32<NM, NA, FULL>);
  for (int e = 0; e < A.S.nelem; ++e) {
    k_snap_y32<NM, NA, FULL><<<tiles * A.nsplit, sy32_threads(NA), snap_y_smem(A.S, A.ta, false), s>>>(A, e);
    EMD_CHECK_LAUNCH();
  }
}

template <bool POLY>
void launch_u(const SnapArgs& A, cudaStream_t s) {
  const size_t cols = size_t(POLY ? su_pcols(A.S.twojmax) : su_stride(A.S.cols));
  const size_t smem = sizeof(double) * (size_t((A.S.nx + 1) & ~1) + 32 * cols);
  allow_dyn_smem(k_snap_u<POLY>);
  k_snap_u<POLY><<<A.n, 32, smem, s>>>(A);
  EMD_CHECK_LAUNCH();
}
inline void launch_u(const SnapArgs& A, cudaStream_t s) {
  if (A.S.twojmax > SU_POWERS) launch_u<true>(A, s);
  else launch_u<false>(A, s);
}

template <typename R, int JC>
void launch_force_j(const SnapArgs& A, int threads, cudaStream_t s) {
  const size_t smem = ((size_t(A.apc) * 4 * A.S.ne * sizeof(R) + 15) & ~size_t(15)) + size_t(threads) * 24;
  allow_dyn_smem(k_snap_force<R, JC>);
  k_snap_force<R, JC><<<(A.n + A.apc - 1) / A.apc, threads, smem, s>>>(A);
  EMD_CHECK_LAUNCH();
}
template <typename R>
void launch_force(const SnapArgs& A, int threads, cudaStream_t s) {
  switch (A.S.twojmax) {
    case 2: return launch_force_j<R, 2>(A, threads, s);
    case 4: return launch_force_j<R, 4>(A, threads, s);
    case 6: return launch_force_j<R, 6>(A, threads, s);
    case 8: return launch_force_j<R, 8>(A, threads, s);
    default: return launch_force_j<R, -1>(A, threads, s);
  }
}

// the kernels of one chunk, up to Y
template <typename R>
void launch_pairs(const SnapArgs& A, cudaStream_t s) {
  const int warps = (A.n + A.rows - 1) / A.rows;
  k_snap_pairs<R><<<(warps + 1) / 2, 64, 0, s>>>(A);
  EMD_CHECK_LAUNCH();
}

}  // namespace snapk
}  // namespace emd
