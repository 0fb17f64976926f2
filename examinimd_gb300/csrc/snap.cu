// ForceSNAP host side: tables, launches and the adjoint reduction
// (force_snap_neigh_impl.h:160-724, sna_impl.hpp).  The kernel is in
// snap_kernel.cuh; the mixed-form instantiation is compiled in snap_mixed.cu.
#include <algorithm>
#include <array>
#include <cmath>
#include <cstring>
#include <functional>
#include <memory>
#include <mutex>
#include <vector>

#include "snap_kernel.cuh"

namespace emd {

void snap_mixed_pairs(const snapk::SnapArgs& A, cudaStream_t s);
void snap_mixed_u(const snapk::SnapArgs& A, cudaStream_t s);
void snap_mixed_y(const snapk::SnapArgs& A, cudaStream_t s);
void snap_mixed_force(const snapk::SnapArgs& A, int threads, cudaStream_t s);

namespace {

using namespace snapk;

struct SnapTables;

struct SnapHost {
  SnapDev d{};
  const int* tmask = nullptr;  // k_snap_force: groups of T
  const int4* zsrc = nullptr;  // the FP32 stream's products (SnapTables::src)
  const SnapTables* tab = nullptr;
  int precision = EMD_PREC_FP64;
  DevBuf<unsigned char> tables;  // every constant table, one allocation and copy
  DevBuf<double> coef;  // cY, then beta_0 of every element
  DevBuf<uint4> zs;
  // per-chunk work arrays
  DevBuf<double> pd, pr_f, U, Y, zk;
  DevBuf<int> pj, cnt;
  DevBuf<Cplx<double>> D, H;
  int fits = 1 << 30;  // atoms that memory had room for when it was short (snap_chunks)
  void release_work() {
    for (auto* b : {&pd, &pr_f, &U, &Y, &zk}) b->release();
    for (auto* b : {&pj, &cnt}) b->release();
    for (auto* b : {&D, &H}) b->release();
  }
  DevBuf<double> eatom;
  // adjoint: per-atom columns, their per-element sums, the loss gradient dL/dF
  DevBuf<double> adj, adj_sum, adj_g;
  // coefficient k's three dB/dr terms: full triples and factors (the cY fold)
  std::vector<int> k_t1, k_t2, k_t3;
  std::vector<double> k_f2, k_f3;
  std::vector<int> k_j;  // (j1, j2, j) of coefficient k
  // U_tot and the Z of the last FP64 force pass, kept for an adjoint
  // on the same positions and list (emd_snap_keep_for_adjoint)
  bool keep_on = false, keep_valid = false;
  unsigned long long keep_xver = 0;
  long long keep_builds = -1;
  int keep_n = -1;
  DevBuf<double> keep_u, keep_z;
};


// ---------------------------------------------------------------- host tables
constexpr int kFactorials = 32;  // the largest: 3 / 2 twojmax + 1 = 22
double factorial(int n) {
  static const std::array<double, kFactorials> table = [] {
    std::array<double, kFactorials> t{};
    t[0] = 1.0;
    for (int i = 1; i < kFactorials; i++) t[size_t(i)] = t[size_t(i - 1)] * i;
    return t;
  }();
  return table[size_t(n)];
}
double deltacg(int j1, int j2, int j) {
  const double s = factorial((j1 + j2 + j) / 2 + 1);
  return std::sqrt(factorial((j1 + j2 - j) / 2) * factorial((j1 - j2 + j) / 2) * factorial((-j1 + j2 + j) / 2) / s);
}
// Clebsch-Gordan coefficient by the quasi-binomial formula of Varshalovich,
// Moskalev, Khersonskii 8.2.1(3) in twice-angular-momentum integers (the
// table SNA::init_clebsch_gordan builds, sna_impl.hpp:1003-1046)
double clebsch_gordan(int j1, int j2, int j, int m1, int m2) {
  const int aa2 = 2 * m1 - j1, bb2 = 2 * m2 - j2;
  const int m = (aa2 + bb2 + j) / 2;
  if (m < 0 || m > j) return 0.0;
  double sum = 0.0;
  for (int z = std::max(0, std::max(-(j - j2 + aa2) / 2, -(j - j1 - bb2) / 2));
       z <= std::min((j1 + j2 - j) / 2, std::min((j1 - aa2) / 2, (j2 + bb2) / 2)); z++) {
    const int ifac = z % 2 ? -1 : 1;
    sum += ifac / (factorial(z) * factorial((j1 + j2 - j) / 2 - z) * factorial((j1 - aa2) / 2 - z) *
                   factorial((j2 + bb2) / 2 - z) * factorial((j - j2 + aa2) / 2 + z) * factorial((j - j1 - bb2) / 2 + z));
  }
  const int cc2 = 2 * m - j;
  return sum * deltacg(j1, j2, j) *
         std::sqrt(factorial((j1 + aa2) / 2) * factorial((j1 - aa2) / 2) * factorial((j2 + bb2) / 2) *
                   factorial((j2 - bb2) / 2) * factorial((j + cc2) / 2) * factorial((j - cc2) / 2) * (j + 1));
}

double jacobi_A(int al, int be, int k) {  // monic Jacobi P_k^(al, be): P_{k+1} = (x - A) P_k - B P_{k-1}
  const double s = 2.0 * k + al + be;
  if (k == 0) return (be - al) / (s + 2.0);
  return (double(be) * be - double(al) * al) / (s * (s + 2.0));
}
double jacobi_B(int al, int be, int k) {
  if (k == 0) return 0.0;
  const double s = 2.0 * k + al + be;
  return 4.0 * k * (k + al) * (k + be) * (k + al + be) / (s * s * (s + 1.0) * (s - 1.0));
}

long long rec_cost(const ZRec& z) { return (long long)z.np * (4 + 2 * z.nj); }  // operations
constexpr int ZS_PARTS = 48;        // a Z task has at most about this fraction of the work,
constexpr long long ZS_LEAST = 300; // unless that is less than this
constexpr int ZS_SPLIT = 16;        // CTAs that may share a tile

// The tables of one twojmax (see the structures in snap_kernel.cuh)
struct SnapTables {
  std::vector<Entry> ent;
  std::vector<int> e0, zt0, tmask, eord;
  std::vector<int2> xsum, psum, ucol, half, zt, prod;
  std::vector<float2> mono;
  std::vector<int4> hfull, ysrc;
  std::vector<ZTask> task;
  std::vector<ZRec> rec;
  std::vector<double> zc, AB, monod;
  std::vector<ZGrp> grp;
  std::vector<unsigned> words;  // the FP32 stream without its coefficients
  std::vector<int4> src;  // of a product in it: first word, coefficient, highest triple, number of j
  int nz = 0, nh = 0, ny = 0;
  // cost of the busiest of k + 1 CTAs that share a tile's tasks: FP64 in cycles,
  // mixed in instructions of the busiest of 12 or 16 warps
  double cta64[ZS_SPLIT], cta32[2][ZS_SPLIT];

  SnapTables(int J, const std::vector<int>& trip) {
    const int L = J + 1, ntrip = int(trip.size() / 3);
    auto uidx = [](int j, int ma, int mb) { return j * (j + 1) * (2 * j + 1) / 6 + ma * (j + 1) + mb; };
    // entries, real sums and their columns (powers of a, then those of b times
    // those of x in (T, k) order; psum: powers of a, of b, then those of b times
    // P_k, k > 0, in (T, q, k) order)
    e0.assign(size_t(L) * L, -1);
    int col = L, pcol = 4 * L;
    for (int T = 0; T <= J; ++T) {
      for (int q = 0; q <= J - T; ++q) {
        e0[size_t(T) * L + q] = int(ent.size());
        std::vector<double> pk{1.0}, pm;  // P_k and P_{k-1} in powers of x
        for (int k = 0; q + T + 2 * k <= J; ++k) {
          const int j = q + T + 2 * k, ma = (j - q - T) / 2, mb = (j - q + T) / 2;
          Entry E{};
          E.N = std::ldexp(factorial(j) / std::sqrt(factorial(ma) * factorial(j - ma) * factorial(mb) * factorial(j - mb)),
                           -k);
          E.Nf = float(E.N);
          E.A = jacobi_A(T, q, k);
          E.B = jacobi_B(T, q, k);
          AB.push_back(E.A);
          AB.push_back(E.B);
          E.T = T;
          E.q = q;
          E.j = j;
          E.ep = uidx(j, ma, mb);
          E.em = uidx(j, mb, ma);
          E.mp = uidx(j, j - ma, j - mb);
          E.mm = uidx(j, j - mb, j - ma);
          E.xo = int(xsum.size());
          const int cp = 2 * q, cr = 2 * q + 1, cu = 2 * (col + k), cv = cu + 1;
          const int pu = k == 0 ? 2 * L + 2 * T : pcol, pv = pu + 1;
          if (k > 0) pcol += T > 0 ? 2 : 1;
          xsum.push_back(int2{cp, cu}), psum.push_back(int2{cp, pu});
          if (q > 0) xsum.push_back(int2{cr, cu}), psum.push_back(int2{cr, pu});
          if (T > 0) xsum.push_back(int2{cp, cv}), psum.push_back(int2{cp, pv});
          if (q > 0 && T > 0) xsum.push_back(int2{cr, cv}), psum.push_back(int2{cr, pv});
          ucol.push_back(int2{q, col + k});
          E.mo = int(mono.size());
          for (double c : pk) monod.push_back(E.N * c), mono.push_back(float2{float(E.N * c), float(E.N * c - double(float(E.N * c)))});
          std::vector<double> pn(pk.size() + 1, 0.0);
          for (size_t l = 0; l < pk.size(); ++l) {
            pn[l + 1] += pk[l];
            pn[l] -= E.A * pk[l];
          }
          for (size_t l = 0; l < pm.size(); ++l) pn[l] -= E.B * pm[l];
          pm = pk;
          pk = pn;
          half.push_back(int2{nh, q > 0 && T > 0 ? nh + 1 : -1});
          nh += q > 0 && T > 0 ? 2 : 1;
          const int sign = T & 1 ? -1 : 1;  // (-1)^(ma + mb)
          hfull.push_back(int4{E.ep, E.mp, sign, 0});
          if (q > 0 && T > 0) hfull.push_back(int4{E.em, E.mm, sign, 0});
          ent.push_back(E);
        }
      }
      col += (J - T) / 2 + 1;
    }
    for (int e = 0; e < int(ent.size()); ++e) eord.push_back(e);
    std::stable_sort(eord.begin(), eord.end(), [&](int x, int y) {
      return ent[size_t(x)].j - ent[size_t(x)].q - ent[size_t(x)].T > ent[size_t(y)].j - ent[size_t(y)].q - ent[size_t(y)].T;
    });
    // Clebsch-Gordan coefficients of every (j1, j2): for each (m1, m2) the
    // allowed j from the highest down
    std::vector<int> cgo(size_t(L) * L), njt(size_t(L) * L), ttop(size_t(L) * L);
    std::vector<double> cg;
    for (int j1 = 0; j1 <= J; ++j1)
      for (int j2 = 0; j2 <= j1; ++j2) {
        const size_t pr = size_t(j1) * L + j2;
        const int lo = j1 - j2, hi = std::min(J - ((J + j1 + j2) & 1), j1 + j2);
        cgo[pr] = int(cg.size());
        njt[pr] = (hi - lo) / 2 + 1;
        for (int m1 = 0; m1 <= j1; ++m1)
          for (int m2 = 0; m2 <= j2; ++m2)
            for (int j = hi; j >= lo; j -= 2) cg.push_back(clebsch_gordan(j1, j2, j, m1, m2));
        for (int t = 0; t < ntrip; ++t)
          if (trip[3 * size_t(t)] == j1 && trip[3 * size_t(t) + 1] == j2 && trip[3 * size_t(t) + 2] == hi) ttop[pr] = t;
      }
    // Z tasks, longest first: one (T, q) and sign of T each, in as many parts
    // as keep a part near 1/ZS_PARTS of the whole
    struct Raw {
      ZTask t;
      std::vector<ZRec> r;
      long long cost;
      int h0, hs;  // half-grid element of k = 0, elements between two k
    };
    std::vector<int2> rp;    // products and coefficients in record order
    std::vector<double> rc;  // before the tasks are sorted
    std::vector<Raw> whole, raw;
    for (int T = 0; T <= J; ++T)
      for (int q = 0; q <= J - T; ++q)
        for (int s = 0; s < (T > 0 && q > 0 ? 2 : 1); ++s) {
          Raw w{};
          w.t.kmax = (J - q - T) / 2;
          const int top = q + T + 2 * w.t.kmax;
          const int2 h = half[size_t(e0[size_t(T) * L + q])];
          w.h0 = s ? h.y : h.x;
          w.hs = h.y >= 0 ? 2 : 1;
          for (int j1 = 0; j1 <= J; ++j1)
            for (int j2 = 0; j2 <= j1; ++j2) {
              if ((j1 + j2 - q - T) & 1) continue;
              const size_t pr = size_t(j1) * L + j2;
              const int hi = j1 - j2 + 2 * (njt[pr] - 1), lo = std::max(j1 - j2, q + T);
              if (hi < lo) continue;
              const int sT = s ? -T : T, M = (j1 + j2 - q - sT) / 2, Mp = (j1 + j2 - q + sT) / 2;
              ZRec z{};
              z.nj = short((hi - lo) / 2 + 1);
              z.d = short((top - hi) / 2);
              z.t0 = ttop[pr];
              z.p0 = int(rp.size());
              z.c0 = int(rc.size());
              for (int m1 = std::max(0, M - j2); m1 <= std::min(j1, M); ++m1)
                for (int n1 = std::max(0, Mp - j2); n1 <= std::min(j1, Mp); ++n1) {
                  const int m2 = M - m1, n2 = Mp - n1;
                  // j1 = j2: (m1, n1)(m2, n2) and (m2, n2)(m1, n1) are one product
                  if (j1 == j2 && (m2 < m1 || (m2 == m1 && n2 < n1))) continue;
                  const double twice = j1 == j2 && !(m1 == m2 && n1 == n2) ? 2.0 : 1.0;
                  rp.push_back(int2{uidx(j1, m1, n1), uidx(j2, m2, n2)});
                  for (int j = 0; j < z.nj; ++j)
                    rc.push_back(twice * cg[size_t(cgo[pr] + (m1 * (j2 + 1) + m2) * njt[pr] + j)] *
                                 cg[size_t(cgo[pr] + (n1 * (j2 + 1) + n2) * njt[pr] + j)]);
                }
              z.np = int(rp.size()) - z.p0;
              w.cost += rec_cost(z);
              w.r.push_back(z);
            }
          whole.push_back(std::move(w));
        }
    long long total = 0;
    for (const Raw& w : whole) total += w.cost;
    const long long most = std::max(ZS_LEAST, total / ZS_PARTS);
    ysrc.assign(size_t(nh), int4{0, 0, 0, 0});
    for (const Raw& w : whole) {
      const long long parts = (w.cost + most - 1) / most;
      long long done = 0;
      size_t r = 0;
      int np = 0;
      const int y0 = ny;
      for (long long k = 0; k < parts; ++k) {
        Raw v{};
        v.t = w.t;
        v.t.y0 = ny;
        v.h0 = w.h0;
        v.hs = w.hs;
        while (r < w.r.size() && (v.r.empty() || (done + rec_cost(w.r[r]) / 2) * parts < (k + 1) * w.cost)) {
          v.cost += rec_cost(w.r[r]);
          done += rec_cost(w.r[r]);
          v.r.push_back(w.r[r++]);
        }
        if (v.r.empty()) break;
        ny += w.t.kmax + 1;
        ++np;
        raw.push_back(std::move(v));
      }
      for (int k = 0; k <= w.t.kmax; ++k) ysrc[size_t(w.h0 + k * w.hs)] = int4{y0 + k, w.t.kmax + 1, np, 0};
    }
    std::stable_sort(raw.begin(), raw.end(), [](const Raw& x, const Raw& y) { return x.cost > y.cost; });
    std::vector<std::vector<int2>> by_t(static_cast<size_t>(ntrip));
    // FP32 stream: tasks start on 64 bytes, groups on their products' size
    auto align = [&](size_t n) { words.resize((words.size() + n - 1) / n * n, 0u); };
    for (Raw& w : raw) {
      align(16);
      w.t.s0 = int(words.size());
      w.t.rec0 = int(rec.size());
      for (ZRec& z : w.r) {
        const int rp0 = z.p0, rc0 = z.c0;
        z.p0 = int(prod.size());
        z.c0 = int(zc.size());
        prod.insert(prod.end(), rp.begin() + rp0, rp.begin() + rp0 + z.np);
        zc.insert(zc.end(), rc.begin() + rc0, rc.begin() + rc0 + z.np * z.nj);
        z.z0 = nz;
        for (int j = 0; j < z.nj; ++j) {  // highest j first: k = kmax - d - j
          by_t[size_t(z.t0 - j)].push_back(int2{nz, w.h0 + (w.t.kmax - z.d - j) * w.hs});
          ++nz;
        }
        rec.push_back(z);
      }
      w.t.rec1 = int(rec.size());
      w.t.grp0 = int(grp.size());
      std::vector<const ZRec*> rs;
      for (const ZRec& z : w.r) rs.push_back(&z);
      std::stable_sort(rs.begin(), rs.end(),
                       [](const ZRec* x, const ZRec* y) { return x->nj != y->nj ? x->nj > y->nj : x->d < y->d; });
      for (size_t k = 0; k < rs.size(); ++k) {
        const ZRec& z = *rs[k];
        const int nw = zs_words(z.nj);
        if (k == 0 || rs[k - 1]->nj != z.nj || rs[k - 1]->d != z.d) {
          align(size_t(nw));
          grp.push_back(ZGrp{int(words.size()) - w.t.s0, 0, z.nj, z.d});
        }
        for (int i = 0; i < z.np; ++i) {
          const int2 u = prod[size_t(z.p0 + i)];
          src.push_back(int4{int(words.size()), z.c0 + i * z.nj, z.t0, z.nj});
          words.push_back(unsigned(u.x) | unsigned(u.y) << 16);
          words.resize(words.size() + size_t(nw) - 1, 0u);
        }
        grp.back().np += z.np;
      }
      w.t.grp1 = int(grp.size());
      task.push_back(w.t);
    }
    // a task's turn in each case: the warp that is free first takes the next
    for (int k = 1; k <= ZS_SPLIT; ++k) {
      double c64 = 0.0, c32[2] = {0.0, 0.0};
      for (int s = 0; s < k; ++s) {
        double sum = 0.0, longest = 0.0;
        std::vector<double> load[2] = {std::vector<double>(sy32_threads(1) / 32, 0.0),
                                       std::vector<double>(sy32_threads(2) / 32, 0.0)};
        for (size_t t = size_t(s); t < raw.size(); t += size_t(k)) {
          const double c = double(raw[t].cost);
          sum += c;
          longest = std::max(longest, c);
          for (auto& l : load) *std::min_element(l.begin(), l.end()) += c;
        }
        c64 = std::max(c64, std::max(19.0 * sum, 64.0 * longest));
        for (int v = 0; v < 2; ++v) c32[v] = std::max(c32[v], *std::max_element(load[v].begin(), load[v].end()));
      }
      cta64[k - 1] = c64;
      for (int v = 0; v < 2; ++v) cta32[v][k - 1] = c32[v];
    }
    words.resize(((words.size() + 3) & ~size_t(3)) + 3 * ZS_CHUNK, 0u);  // a warp reads up to two chunks ahead
    for (const auto& v : by_t) {
      zt0.push_back(int(zt.size()));
      zt.insert(zt.end(), v.begin(), v.end());
    }
    zt0.push_back(int(zt.size()));
    // four groups of T of about equal work (k_snap_force)
    std::vector<long long> load(4, 0);
    tmask.assign(4, 0);
    std::vector<std::pair<long long, int>> tw;
    for (int T = 0; T <= J; ++T) {
      long long wk = 0;
      for (int q = 0; q <= J - T; ++q) wk += (T ? 2 : 1) * (8 + 8 * ((J - T - q) / 2));
      tw.push_back({-wk, T});
    }
    std::sort(tw.begin(), tw.end());
    for (const auto& w : tw) {
      const size_t g = size_t(std::min_element(load.begin(), load.end()) - load.begin());
      load[g] -= w.first;
      tmask[g] |= 1 << w.second;
    }
  }
};

// They depend on twojmax alone: built once per process, shared and read-only.
const SnapTables& snap_tables(int J, const std::vector<int>& trip) {
  static std::mutex mu;
  static std::unique_ptr<const SnapTables> tables[15];
  std::lock_guard<std::mutex> lock(mu);
  if (!tables[J]) tables[J] = std::make_unique<const SnapTables>(J, trip);
  return *tables[J];
}

// the FP32 stream's coefficients: the Clebsch-Gordan products times cY
__global__ void __launch_bounds__(256) k_zs_fill(SnapDev S, const int4* __restrict__ src, int n, unsigned* zs) {
  const int k = blockIdx.x * 256 + threadIdx.x, e = blockIdx.y;
  if (k >= n) return;
  const int4 p = src[k];
  const double* c = S.cY + size_t(e) * S.nfull + p.z;
  unsigned* w = zs + size_t(e) * S.zs_n * 4 + p.x + 1;
  for (int j = 0; j < p.w; ++j) w[j] = __float_as_uint(float(S.zc[p.y + j] * c[-j]));
}

// per-element column sums of the adjoint's per-atom outputs (fixed order)
__global__ void __launch_bounds__(256) k_adj_reduce(const double* __restrict__ adj, int n, int ncols,
                                                    const int* __restrict__ type, const int* __restrict__ map,
                                                    double* __restrict__ out) {
  __shared__ double sh[8];
  const int col = blockIdx.x, e = blockIdx.y;
  const double* a = adj + size_t(col) * n;
  double acc = 0.0;
  for (int i = threadIdx.x; i < n; i += 256)
    if (map[type[i]] == e) acc += a[i];
  const double t = block_sum(acc, sh);
  if (threadIdx.x == 0) out[size_t(e) * ncols + col] = t;
}

}  // namespace

static void drop_snap(SnapHost* h) {
  h->release_work();
  h->tables.release();
  h->zs.release();
  for (auto* b : {&h->coef, &h->eatom, &h->adj, &h->adj_sum, &h->adj_g, &h->keep_u, &h->keep_z}) b->release();
  delete h;
}
void free_snap(Ctx& c) {
  c.snap_pe_fused_valid = false;
  if (c.snap) drop_snap(static_cast<SnapHost*>(c.snap));
  c.snap = nullptr;
}

template <class T>
static void upload(Ctx& c, DevBuf<T>& b, const std::vector<T>& v) {
  b.reserve(v.size() + 1, c.stream);
  EMD_CUDA(cudaMemcpyAsync(b.p, v.data(), sizeof(T) * v.size(), cudaMemcpyHostToDevice, c.stream));
}

// the coefficients' part of the FP32 stream, where the form has one
static void fill_stream(Ctx& c, SnapHost* h) {
  if (h->precision != EMD_PREC_MIXED) return;
  const int n = int(h->tab->src.size());
  TimedLaunch t(c, "snap_stream");
  k_zs_fill<<<dim3(blocks_for(n, 256), h->d.nelem), 256, 0, c.stream>>>(h->d, h->zsrc, n,
                                                                        reinterpret_cast<unsigned*>(h->zs.p));
  EMD_CHECK_LAUNCH();
}

// Y's coefficients: beta_k folded onto the full triples of compute_dbidrj's
// three terms (sna_impl.hpp:330-570), per element, then every element's beta_0
std::vector<double> snap_fold_beta(const SnapHost& h, int nfull, int nelem, int ncoeffall, const double* beta) {
  std::vector<double> c(size_t(nelem) * (nfull + 1), 0.0);
  for (int e = 0; e < nelem; ++e) {
    const double* be = beta + size_t(e) * ncoeffall;
    c[size_t(nelem) * nfull + size_t(e)] = be[0];
    double* ce = &c[size_t(e) * nfull];
    for (size_t k = 0; k < h.k_t1.size(); ++k) {
      const int j1 = h.k_j[3 * k], j2 = h.k_j[3 * k + 1], j = h.k_j[3 * k + 2];
      const double bk = be[k + 1];
      ce[h.k_t1[k]] += bk;
      ce[h.k_t2[k]] += bk * (j + 1) / (j1 + 1.0);
      ce[h.k_t3[k]] += bk * (j + 1) / (j2 + 1.0);
    }
  }
  return c;
}

// Atoms are worked on in chunks so that the work arrays stay bounded: at most
// kChunk atoms and about kChunkBytes of pair fields.
constexpr int kChunk = 131072;
constexpr size_t kChunkBytes = size_t(3) << 30;

static int snap_chunk(int n, int cap, bool adjoint_z, const SnapDev& S) {
  size_t per = size_t(cap) * (8 * (PD_N + PF_N) + 4);
  if (adjoint_z) per += size_t(16) * S.nz;
  const size_t most = std::max<size_t>(32, std::min<size_t>(kChunk, kChunkBytes / per));
  const int chunks = int((size_t(n) + most - 1) / most);
  return std::min(n, ((n + chunks - 1) / chunks + 31) & ~31);
}

// work(first, n) for all atoms, `chunk` at a time.  It reserves its work arrays before its
// first launch; where they do not fit, they are given back and half as many atoms are
// taken (multiples of 32, the tiles of what an adjoint keeps), by later calls too.
template <typename Work>
static void snap_chunks(Ctx& c, SnapHost* h, int n, int chunk, Work&& work) {
  for (int first = 0; first < n;) {
    const int m = std::min({chunk, h->fits, n - first});
    try {
      work(first, m);
      first += m;
    } catch (const Error& e) {
      if (e.code != EMD_ERR_NOMEM || m <= 32) throw;
      EMD_CUDA(cudaStreamSynchronize(c.stream));
      h->release_work();
      h->fits = (m / 2 + 31) & ~31;
    }
  }
}

// Atoms per tile of k_snap_y and CTAs that share a tile's tasks: the smallest
// product of waves over the 152 SMs and time per CTA.  A tile costs the same
// whatever its lanes hold; with fewer atoms than lanes the lane groups share a
// record's products (0.89, 0.73, 0.53 of the lanes' work useful at 16, 8, 4
// atoms).  FP64: the SM issues one instruction per 19 cycles, a single warp one
// per 64.  Mixed: the busiest of the CTA's warps when each takes the next
// longest task (more CTAs than tasks per warp leave warps idle).
struct SnapTiling {
  int ta, nsplit;
};
static SnapTiling snap_tiling(const SnapDev& S, const SnapTables& tab, int n, bool fp64, bool keep) {
  // mixed form: two atoms per lane once the tiles' splits fill the SMs
  if (!fp64 && S.twojmax <= 9 && (n + 63) / 64 * 4 >= 2 * 152 && snap_y_smem(S, 64, fp64) <= kMaxDynSmem) {
    const long long tiles = (n + 63) / 64;
    SnapTiling best{64, 1};
    double best_cost = 1e300;
    for (int k = 1; k <= ZS_SPLIT; ++k) {
      const double cost = double((tiles * k + 151) / 152) * (tab.cta32[1][k - 1] + 1000.0);
      if (cost < best_cost) best.nsplit = k, best_cost = cost;
    }
    return best;
  }
  SnapTiling best{0, 1};
  double best_cost = 1e300;
  const double lanes[6] = {0.2, 0.2, 0.236, 0.342, 0.562, 1.0};  // cost of a tile of 1, 2, 4 .. 32 atoms
  for (int l = 5; l >= 0; --l) {
    const int ta = 1 << l;
    if (snap_y_smem(S, ta, fp64) > kMaxDynSmem) continue;
    if (best.ta != 0 && (keep || ta < 4)) break;
    const long long tiles = (n + ta - 1) / ta, wave = 152LL * (fp64 ? 1 : 2);
    for (int k = 1; k <= ZS_SPLIT; ++k) {
      const double cta = fp64 ? tab.cta64[k - 1] * lanes[l] + 4000.0 : tab.cta32[0][k - 1] * lanes[l] + 1000.0;
      const double cost = double((tiles * k + wave - 1) / wave) * cta;
      if (cost < best_cost) best = SnapTiling{ta, k}, best_cost = cost;
    }
  }
  return best;
}

// arguments of one chunk, work arrays reserved
static SnapArgs snap_args(Ctx& c, SnapHost* h, int first, int n, bool fp64, bool keep) {
  const SnapDev& S = h->d;
  const size_t real = fp64 ? 8 : 4;
  SnapArgs A{};
  A.S = S;
  A.x4 = c.x4.p;
  A.type = c.type.p;
  A.L = list_view(c);
  A.first = first;
  A.n = n;
  A.n_local = c.N_local;
  A.cap = std::max(1, c.neigh_maxrow);
  A.rows = std::min(SP_ROWS, std::max(1, n / (152 * 8)));
  const size_t np = size_t(n) * A.cap;
  h->pd.reserve((fp64 ? PD_N : PD_N32) * np, c.stream);
  h->pr_f.reserve(fp64 ? PF_N * np : (PR_N * np + 1) / 2, c.stream);
  h->pj.reserve(np, c.stream);
  h->cnt.reserve(size_t(n), c.stream);
  A.pd = h->pd.p;
  A.pr = h->pr_f.p;
  A.pj = h->pj.p;
  A.cnt = h->cnt.p;
  const SnapTiling tl = snap_tiling(S, *h->tab, n, fp64, keep);
  A.ta = tl.ta;
  A.nsplit = tl.nsplit;
  const int tiles = (n + A.ta - 1) / A.ta;
  h->Y.reserve((size_t(tiles) * 2 * S.ny * A.ta * real + 7) / 8, c.stream);
  A.Y = h->Y.p;
  A.f = c.f.p;
  A.tmask = h->tmask;
  return A;
}

// U_tot and Y of a chunk
static void snap_uy(Ctx& c, const SnapArgs& A, bool fp64) {
  {
    TimedLaunch t(c, "snap_pairs");
    if (fp64) launch_pairs<double>(A, c.stream);
    else snap_mixed_pairs(A, c.stream);
  }
  {
    TimedLaunch t(c, "snap_u");
    if (fp64) launch_u(A, c.stream);
    else snap_mixed_u(A, c.stream);
  }
  TimedLaunch t(c, fp64 ? "snap_y_fp64" : "snap_y_mixed");
  if (!fp64) snap_mixed_y(A, c.stream);
  else if (A.S.twojmax <= 9) launch_y<5>(A, c.stream);
  else launch_y<8>(A, c.stream);
}

static void snap_require_list(Ctx& c, const char* what) {
  require(c.neigh_ready && c.neigh_rows == c.N_local && !c.half_neigh, EMD_ERR_STATE, what);
  require(!c.neigh_packed, EMD_ERR_STATE, "SNAP reads plain neighbour rows");
}

static void snap_launch(Ctx& c, bool energy) {
  SnapHost* h = static_cast<SnapHost*>(c.snap);
  require(h != nullptr, EMD_ERR_STATE, "SNAP not initialised");
  snap_require_list(c, "SNAP needs a current full neighbour list");
  const int n = c.N_local;
  if (n == 0) return;
  if (!energy) {
    materialize_kick(c);  // the forces are about to be overwritten
    materialize_zero(c, true, true);
  }
  const SnapDev& S = h->d;
  const bool fp64 = h->precision == EMD_PREC_FP64 || energy;
  // asked for (emd_snap_request_energy): the per-atom energies in the same pass
  const bool fused = !energy && fp64 && c.snap_energy_request;
  const bool keep = !energy && fp64 && h->keep_on;
  if (energy || fused) h->eatom.reserve(size_t(n), c.stream);
  if (keep) {
    h->keep_u.reserve(2 * size_t(S.nh) * n, c.stream);
    h->keep_z.reserve(2 * size_t(S.nz) * ((size_t(n) + 31) & ~size_t(31)), c.stream);
  }
  const int chunk = snap_chunk(n, std::max(1, c.neigh_maxrow), false, S);
  snap_chunks(c, h, n, chunk, [&](int first, int m) {
    SnapArgs A = snap_args(c, h, first, m, fp64, fp64 && h->keep_on);
    if (keep) {
      A.U = h->keep_u.p + 2 * size_t(S.nh) * first;
      A.zkeep = h->keep_z.p + 2 * size_t(S.nz) * first;
    } else {
      h->U.reserve(2 * size_t(S.nh) * A.n, c.stream);
      A.U = h->U.p;
    }
    snap_uy(c, A, fp64);
    if (energy || fused) {
      A.eatom = h->eatom.p;
      TimedLaunch t(c, "snap_energy");
      k_snap_energy<<<(A.n + 3) / 4, 128, 0, c.stream>>>(A);
      EMD_CHECK_LAUNCH();
    }
    if (energy) return;
    // Eight atoms pool about 208 pairs for 256 lanes; a small system takes one
    // atom per CTA and spreads the T of a pair over four warps
    A.apc = std::max(1, std::min(SF_ATOMS, A.n / 152));
    A.tsplit = A.apc < 4 ? 4 : 1;
    const int threads = A.tsplit == 4 ? 32 * 4 * std::max(1, std::min(2, A.apc)) : SF_THREADS;
    TimedLaunch t(c, fp64 ? "snap_force_fp64" : "snap_force_mixed");
    if (!fp64) snap_mixed_force(A, threads, c.stream);
    else launch_force<double>(A, threads, c.stream);
  });
  if (fused) {
    c.snap_pe_fused_valid = true;
    c.snap_pe_fused_version = c.x_version;
  }
  if (keep) {
    h->keep_valid = true;
    h->keep_xver = c.x_version;
    h->keep_builds = c.neigh_builds;
    h->keep_n = n;
  }
}

// d/dbeta of (dL_dE * E + sum_i dL_dF_i . F_i) for a loss L(E, F) of the
// total SNAP energy and the owned atoms' forces (host arrays)
static void snap_adjoint(Ctx& c, const double* dL_dF, double dL_dE, double* grad) {
  SnapHost* h = static_cast<SnapHost*>(c.snap);
  require(h != nullptr, EMD_ERR_STATE, "SNAP not initialised");
  require(c.neigh_ready && c.neigh_rows == c.N_local && !c.half_neigh && !c.neigh_packed, EMD_ERR_STATE,
          "emd_snap_adjoint needs a current full neighbour list");
  const SnapDev& S = h->d;
  const int n = c.N_local, nelem = S.nelem, ncols = 2 * S.nfull + 1;
  std::vector<double> sums(size_t(nelem) * ncols, 0.0);
  if (n > 0) {
    h->adj_g.reserve(3 * size_t(n), c.stream);
    EMD_CUDA(cudaMemcpyAsync(h->adj_g.p, dL_dF, sizeof(double) * 3 * size_t(n), cudaMemcpyHostToDevice, c.stream));
    h->adj.reserve(size_t(ncols) * n, c.stream);
    h->adj_sum.reserve(size_t(nelem) * ncols, c.stream);
    // U_tot and Z from the last FP64 force pass, when it ran on these positions and this list
    const bool kept = h->keep_on && h->keep_valid && h->keep_xver == c.x_version && h->keep_builds == c.neigh_builds &&
                      h->keep_n == n;
    const int chunk = snap_chunk(n, std::max(1, c.neigh_maxrow), true, S);
    snap_chunks(c, h, n, chunk, [&](int first, int m) {
      SnapArgs A = snap_args(c, h, first, m, true, true);
      const int tiles = (A.n + 31) / 32;
      h->D.reserve(size_t(S.nh) * A.n, c.stream);
      h->H.reserve(size_t(tiles) * 2 * S.nh * 32, c.stream);
      if (kept) {
        A.U = h->keep_u.p + 2 * size_t(S.nh) * first;
        A.zkeep = h->keep_z.p + 2 * size_t(S.nz) * first;
        TimedLaunch t(c, "snap_pairs");
        launch_pairs<double>(A, c.stream);
      } else {
        h->U.reserve(2 * size_t(S.nh) * A.n, c.stream);
        h->zk.reserve(2 * size_t(S.nz) * tiles * 32, c.stream);
        A.U = h->U.p;
        A.zkeep = h->zk.p;
        snap_uy(c, A, true);
      }
      A.D = h->D.p;
      A.H = h->H.p;
      A.g = h->adj_g.p;
      A.ghost_owner = c.ghost_owner.p;
      A.newton = c.comm_newton;
      A.adj = h->adj.p;
      {
        TimedLaunch t(c, "snap_dt");
        const size_t smem = sizeof(double) * (size_t((S.nx + 1) & ~1) + 64 * size_t(su_stride(S.cols)));
        require(smem <= kMaxDynSmem, EMD_ERR_ARG, "SNAP adjoint: twojmax too large for shared memory");
        allow_dyn_smem(k_snap_dt);
        k_snap_dt<<<A.n, 32, smem, c.stream>>>(A);
        EMD_CHECK_LAUNCH();
      }
      TimedLaunch t(c, "snap_adjoint");
      k_snap_half<<<blocks_for((long long)tiles * S.nh * 32, 256), 256, 0, c.stream>>>(A);
      EMD_CHECK_LAUNCH();
      k_snap_pq<<<dim3(tiles, (S.nfull + 7) / 8), 256, 0, c.stream>>>(A);
      EMD_CHECK_LAUNCH();
    });
    {
      TimedLaunch t(c, "snap_adjoint_reduce");
      k_adj_reduce<<<dim3(ncols, nelem), 256, 0, c.stream>>>(h->adj.p, n, ncols, c.type.p, S.map, h->adj_sum.p);
      EMD_CHECK_LAUNCH();
    }
    EMD_CUDA(cudaMemcpyAsync(sums.data(), h->adj_sum.p, sizeof(double) * sums.size(), cudaMemcpyDeviceToHost,
                             c.stream));
    EMD_CUDA(cudaStreamSynchronize(c.stream));
  }
  for (int e = 0; e < nelem; ++e) {
    const double* P = &sums[size_t(e) * ncols];
    const double* Q = P + S.nfull;
    double* g = grad + size_t(e) * S.ncoeffall;
    g[0] = dL_dE * P[2 * S.nfull];  // E = sum_i (beta_0 + ...)
    for (int k = 0; k < S.ncoeff; ++k)
      g[k + 1] = dL_dE * P[h->k_t1[k]] + Q[h->k_t1[k]] + h->k_f2[k] * Q[h->k_t2[k]] + h->k_f3[k] * Q[h->k_t3[k]];
  }
}

}  // namespace emd

using namespace emd;

extern "C" {

emd_status emd_snap_adjoint(emd_ctx* ctx, const double* dL_dF, double dL_dE, double* grad_beta) {
  EMD_API_BEGIN
  require(grad_beta != nullptr && (dL_dF != nullptr || c.N_local == 0), EMD_ERR_ARG, "emd_snap_adjoint: null array");
  snap_adjoint(c, dL_dF, dL_dE, grad_beta);
  EMD_API_END
}

emd_status emd_snap_init(emd_ctx* ctx, int twojmax, double rfac0, double rmin0, int switchflag, double rcutfac,
                         int nelem, const double* radelem, const double* wjelem, const double* beta, int ncoeffall,
                         int ntypes, const int* map, int precision) {
  EMD_API_BEGIN
  require(twojmax >= 0 && twojmax <= 14, EMD_ERR_ARG, "emd_snap_init: twojmax must be in [0, 14]");
  require(nelem >= 1 && radelem && wjelem && beta && map && ntypes >= 1, EMD_ERR_ARG, "emd_snap_init: arguments");
  require(precision == EMD_PREC_FP64 || precision == EMD_PREC_MIXED, EMD_ERR_ARG, "emd_snap_init: precision");
  require(switchflag == 0 || switchflag == 1, EMD_ERR_ARG, "emd_snap_init: switchflag");
  for (int t = 0; t < ntypes; ++t)
    require(map[t] >= 0 && map[t] < nelem, EMD_ERR_ARG, "emd_snap_init: every type must map to an element");
  free_snap(c);
  std::unique_ptr<SnapHost, void (*)(SnapHost*)> made(new SnapHost(), drop_snap);  // the context's once it is complete
  SnapHost* h = made.get();
  h->precision = precision;
  SnapDev& S = h->d;
  S.twojmax = twojmax;
  // index lists (SNA::build_indexlist, sna_impl.hpp:88-139, diagonalstyle 3)
  std::vector<int> trip;
  std::vector<int> idxj;  // positions of the idxj triples (j >= j1) in the full list
  std::vector<int> idx3;
  for (int j1 = 0; j1 <= twojmax; j1++)
    for (int j2 = 0; j2 <= j1; j2++)
      for (int j = std::abs(j1 - j2); j <= std::min(twojmax, j1 + j2); j += 2) {
        trip.push_back(j1);
        trip.push_back(j2);
        trip.push_back(j);
        if (j >= j1) {
          idx3.push_back(j1);
          idx3.push_back(j2);
          idx3.push_back(j);
        }
      }
  S.nfull = int(trip.size() / 3);
  S.ncoeff = int(idx3.size() / 3);
  require(ncoeffall == S.ncoeff + 1, EMD_ERR_ARG, "emd_snap_init: ncoeffall does not match twojmax");
  S.ncoeffall = ncoeffall;
  auto find_full = [&](int a, int b, int cc) {
    for (int t = 0; t < S.nfull; ++t)
      if (trip[3 * t] == a && trip[3 * t + 1] == b && trip[3 * t + 2] == cc) return t;
    throw Error(EMD_ERR_ARG, "SNAP: triple not found");
  };
  const SnapTables& tab = snap_tables(twojmax, trip);
  S.ne = int(tab.ent.size());
  S.nx = int(tab.xsum.size());
  S.cols = su_cols(twojmax);
  S.nuf = (twojmax + 1) * (twojmax + 2) * (2 * twojmax + 3) / 6;
  S.ntask = int(tab.task.size());
  S.nz = tab.nz;
  S.nh = tab.nh;
  S.ny = tab.ny;
  for (int k = 0; k < S.ncoeff; ++k) {
    const int j1 = idx3[3 * k], j2 = idx3[3 * k + 1], j = idx3[3 * k + 2];
    h->k_t1.push_back(find_full(j1, j2, j));
    h->k_t2.push_back(find_full(std::max(j, j2), std::min(j, j2), j1));
    h->k_t3.push_back(find_full(std::max(j1, j), std::min(j1, j), j2));
    h->k_f2.push_back((j + 1) / (j1 + 1.0));
    h->k_f3.push_back((j + 1) / (j2 + 1.0));
    h->k_j.insert(h->k_j.end(), {j1, j2, j});
  }
  const std::vector<double> coef = snap_fold_beta(*h, S.nfull, nelem, ncoeffall, beta);
  double rcutmax = 0.0;
  for (int e = 0; e < nelem; e++) rcutmax = std::max(2.0 * radelem[e] * rcutfac, rcutmax);
  S.rfac0 = rfac0;
  S.rmin0 = rmin0;
  S.cutsq = rcutmax * rcutmax;
  S.wself = 1.0;
  S.switchflag = switchflag;
  S.nelem = nelem;
  S.ntypes = ntypes;
  // per element pair: cutoff, theta0 and switching slopes (compute_ui, compute_sfac)
  std::vector<double> pr;
  for (int a = 0; a < nelem; ++a)
    for (int b = 0; b < nelem; ++b) {
      const double rcut = (radelem[a] + radelem[b]) * rcutfac;
      pr.push_back(rcut);
      pr.push_back(rfac0 * MY_PI / (rcut - rmin0));
      pr.push_back(MY_PI / (rcut - rmin0));
    }
  const std::vector<float> ABf(tab.AB.begin(), tab.AB.end());
  auto pair32 = [](double v) { return float2{float(v), float(v - double(float(v)))}; };
  std::vector<float2> pr32, wj32;
  for (double v : pr) pr32.push_back(pair32(v));
  for (int e = 0; e < nelem; ++e) wj32.push_back(pair32(wjelem[e]));
  S.nrmin32 = pair32(-rmin0);
  std::vector<unsigned char> bytes;
  std::vector<std::function<void(unsigned char*)>> place;
  auto put = [&](auto& field, const auto& v) {
    const size_t at = (bytes.size() + 255) & ~size_t(255), n = v.size() * sizeof(v[0]);
    bytes.resize(at + n + 16);
    if (n) std::memcpy(&bytes[at], v.data(), n);
    place.push_back([&field, at](unsigned char* p) { field = reinterpret_cast<std::decay_t<decltype(field)>>(p + at); });
  };
  put(S.ent, tab.ent);
  put(S.task, tab.task);
  put(S.rec, tab.rec);
  put(S.e0, tab.e0);
  put(S.xsum, tab.xsum);
  put(S.psum, tab.psum);
  put(S.ucol, tab.ucol);
  put(S.monod, tab.monod);
  put(S.mono, tab.mono);
  put(S.eord, tab.eord);
  put(S.half, tab.half);
  put(S.zt0, tab.zt0);
  put(S.zt, tab.zt);
  put(h->tmask, tab.tmask);
  put(S.hfull, tab.hfull);
  put(S.ysrc, tab.ysrc);
  put(S.prod, tab.prod);
  put(S.zc, tab.zc);
  put(S.grp, tab.grp);
  put(S.AB, tab.AB);
  put(S.AB_f, ABf);
  put(S.pr, pr);
  put(S.pr32, pr32);
  put(S.wj32, wj32);
  put(S.wjelem, std::vector<double>(wjelem, wjelem + nelem));
  put(S.map, std::vector<int>(map, map + ntypes));
  if (precision == EMD_PREC_MIXED) put(h->zsrc, tab.src);
  upload(c, h->tables, bytes);
  for (auto& f : place) f(h->tables.p);
  upload(c, h->coef, coef);
  S.cY = h->coef.p;
  S.beta0 = h->coef.p + size_t(nelem) * S.nfull;
  S.zs_n = int(tab.words.size() / 4);
  h->tab = &tab;
  std::vector<unsigned> w;
  if (precision == EMD_PREC_MIXED) {
    for (int e = 0; e < nelem; ++e) w.insert(w.end(), tab.words.begin(), tab.words.end());
    h->zs.reserve(w.size() / 4, c.stream);
    EMD_CUDA(cudaMemcpyAsync(h->zs.p, w.data(), w.size() * sizeof(unsigned), cudaMemcpyHostToDevice, c.stream));
  }
  S.zs = h->zs.p;
  fill_stream(c, h);
  EMD_CUDA(cudaStreamSynchronize(c.stream));
  c.snap = made.release();
  EMD_API_END
}

emd_status emd_snap_keep_for_adjoint(emd_ctx* ctx, int on) {
  EMD_API_BEGIN
  SnapHost* h = static_cast<SnapHost*>(c.snap);
  require(h != nullptr, EMD_ERR_STATE, "emd_snap_keep_for_adjoint: SNAP not initialised");
  h->keep_on = on != 0;
  h->keep_valid = false;
  if (!h->keep_on) {
    h->keep_u.release();
    h->keep_z.release();
  }
  EMD_API_END
}

emd_status emd_snap_info(emd_ctx* ctx, int* nelem, int* ncoeffall) {
  EMD_API_BEGIN
  const SnapHost* h = static_cast<const SnapHost*>(c.snap);
  require(h != nullptr, EMD_ERR_STATE, "emd_snap_info: SNAP not initialised");
  if (nelem) *nelem = h->d.nelem;
  if (ncoeffall) *ncoeffall = h->d.ncoeffall;
  EMD_API_END
}

emd_status emd_snap_set_beta(emd_ctx* ctx, const double* beta) {
  EMD_API_BEGIN
  SnapHost* h = static_cast<SnapHost*>(c.snap);
  require(h != nullptr, EMD_ERR_STATE, "emd_snap_set_beta: SNAP not initialised");
  require(beta != nullptr, EMD_ERR_ARG, "emd_snap_set_beta: null beta");
  const std::vector<double> coef = snap_fold_beta(*h, h->d.nfull, h->d.nelem, h->d.ncoeffall, beta);
  EMD_CUDA(cudaMemcpyAsync(h->coef.p, coef.data(), sizeof(double) * coef.size(), cudaMemcpyHostToDevice, c.stream));
  fill_stream(c, h);
  EMD_CUDA(cudaStreamSynchronize(c.stream));
  EMD_API_END
}

emd_status emd_snap_compute(emd_ctx* ctx) {
  EMD_API_BEGIN
  struct EndRequest {  // a request serves this compute only
    Ctx& c;
    ~EndRequest() { c.snap_energy_request = false; }
  } end_request{c};
  c.snap_pe_fused_valid = false;
  snap_launch(c, false);
  EMD_API_END
}

emd_status emd_snap_request_energy(emd_ctx* ctx) {
  EMD_API_BEGIN
  require(c.snap != nullptr, EMD_ERR_STATE, "emd_snap_request_energy: SNAP not initialised");
  c.snap_energy_request = true;
  EMD_API_END
}

emd_status emd_snap_force_energy(emd_ctx* ctx, double* pe, int* available) {
  EMD_API_BEGIN
  require(pe && available, EMD_ERR_ARG, "emd_snap_force_energy: null output");
  *available = (c.snap_pe_fused_valid && c.snap_pe_fused_version == c.x_version) ? 1 : 0;
  *pe = 0.0;
  if (*available && c.N_local > 0) *pe = device_sum(c, static_cast<SnapHost*>(c.snap)->eatom.p, c.N_local);
  EMD_API_END
}

emd_status emd_snap_energy(emd_ctx* ctx, double* pe) {
  EMD_API_BEGIN
  require(pe != nullptr, EMD_ERR_ARG, "emd_snap_energy: null output");
  if (c.N_local == 0) {
    *pe = 0.0;
    return EMD_OK;
  }
  snap_launch(c, true);
  *pe = device_sum(c, static_cast<SnapHost*>(c.snap)->eatom.p, c.N_local);
  EMD_API_END
}

emd_status emd_snap_ncoeff(emd_ctx* ctx, int* ncoeff) {
  EMD_API_BEGIN
  require(c.snap != nullptr && ncoeff != nullptr, EMD_ERR_STATE, "emd_snap_ncoeff: SNAP not initialised");
  *ncoeff = static_cast<SnapHost*>(c.snap)->d.ncoeff;
  EMD_API_END
}

}  // extern "C"
