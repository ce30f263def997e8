// grad.cu -- analytic RHF nuclear gradient on the GPU.
//
// dE/dR_A = 2 sum_ij P_ij dH_ij/dR_A - 2 sum_ij W_ij dS_ij/dR_A
//         + sum_ijkl (2 P_ij P_kl - P_ik P_jl) d(ij|kl)/dR_A + dV_nn/dR_A
// with W = P F P, the reference's expression (mmd/forces.py:61-97, P = C_occ C_occ^T),
// evaluated without ever forming a derivative-integral tensor: the derivative integrals
// of a shell pair (one-electron terms) or of a unique shell quartet (two-electron terms)
// are contracted at once with the densities.
//
// A product of two Gaussians depends on its centres through P = (aA + bB)/p, which moves
// the Hermite functions, and through A - B, which changes the expansion coefficients:
//     d/dA = (a/p) d/dP + d/d(A-B),      d/dB = (b/p) d/dP - d/d(A-B),
// and d/dP raises a Hermite index by one.  So per primitive pair the kernels need the
// coefficients E' of the ERI code (cython/util.pxi:13-28, contraction, normalisation and
// p^{-3/2} folded in) and their three derivatives with respect to A - B, tabulated once per
// gradient (k_grad_pairs); centre-differentiated functions (2a G_{i+1} - i G_{i-1},
// cython/grad.pyx:101-108) are needed for the kinetic energy only.
#include <cuda_runtime.h>
#include <math.h>

#include <functional>

#include "md_kernels.cuh"
#include "grad.cuh"

using namespace mmdg;

namespace {

constexpr int kLmaxShell = 2;                 // d shells
constexpr int kEi = kLmaxShell + 2;           // kinetic terms: i up to l + 1, j up to l + 2
constexpr int kEj = kLmaxShell + 3;
constexpr int kEt = 2 * kLmaxShell + 4;       // t up to i + j
constexpr double kPi = 3.14159265358979323846;

__device__ __forceinline__ double comp_norm(int l) { return l >= 2 ? 0.57735026918962576 : 1.0; }

// Cartesian exponents of component c of a shell of angular momentum L (the order of
// mmd/molecule.py:104-115: x^L first, then decreasing x, then decreasing y)
__host__ __device__ constexpr int comp_x(int L, int c) {
  int x = L, left = c;
  while (left > L - x) {
    left -= L - x + 1;
    --x;
  }
  return x;
}
__host__ __device__ constexpr int comp_y(int L, int c) {
  int x = L, left = c;
  while (left > L - x) {
    left -= L - x + 1;
    --x;
  }
  return L - x - left;
}

// ------------------------------------------------------------------ primitive-pair tables
// One thread per primitive pair: (1/p, P), a/p, the coefficients E' in the layout of the ERI
// code (component pairs row-major, then t, u, v) and, behind 3 x the same offset, their
// derivatives with respect to A - B along x, y, z.  With X_PA = -(b/p) (A-B)_x and X_PB =
// (a/p) (A-B)_x the recursion E^{i+1,j}_t = E^{ij}_{t-1}/(2p) + X_PA E^{ij}_t + (t+1)
// E^{ij}_{t+1} is differentiated term by term from d E^{00}_0 = -2 mu (A-B)_x E^{00}_0.
__global__ void __launch_bounds__(64) k_grad_pairs(GradArgs a) {
  const int pp = blockIdx.x * blockDim.x + threadIdx.x;
  if (pp >= a.nprimpair) return;
  const int pr = a.pp_pair[pp], kk = a.pp_index[pp];
  const int sa = a.pa[pr], sb = a.pb[pr];
  const int la = a.L[sa], lb = a.L[sb], Kb = a.nprim[sb];
  const int ka = kk / Kb, kb = kk - ka * Kb;
  const double ea = a.exps[a.poff[sa] + ka], eb = a.exps[a.poff[sb] + kb];
  const double p = ea + eb, ip = 1.0 / p, mu = ea * eb * ip, i2p = 0.5 * ip;
  double AB[3], P[3], AB2 = 0.0;
  for (int d = 0; d < 3; ++d) {
    const double A = a.center[3 * sa + d], B = a.center[3 * sb + d];
    AB[d] = A - B;
    AB2 += AB[d] * AB[d];
    P[d] = (ea * A + eb * B) * ip;
  }
  const double K = exp(-mu * AB2) * a.coefs[a.poff[sa] + ka] * a.coefs[a.poff[sb] + kb] * (ip * sqrt(ip));
  a.pP[pp] = make_double4_32a(ip, P[0], P[1], P[2]);
  a.frac[pp] = ea * ip;
  double E[3][3][3][5], D[3][3][3][5];
  for (int d = 0; d < 3; ++d) {
    const double XPA = -(eb * ip) * AB[d], XPB = (ea * ip) * AB[d];
    E[d][0][0][0] = 1.0;
    D[d][0][0][0] = -2.0 * mu * AB[d];
    for (int i = 0; i <= la; ++i)
      for (int j = 0; j <= lb; ++j) {
        if (i == 0 && j == 0) continue;
        const int i0 = j > 0 ? i : i - 1, j0 = j > 0 ? j - 1 : 0;  // raise j if there is one, else i
        const double X = j > 0 ? XPB : XPA, dX = j > 0 ? ea * ip : -eb * ip;
        for (int t = 0; t <= i + j; ++t) {
          double v = 0.0, w = 0.0;
          if (t < i + j) {  // E^{i0,j0}_t exists
            v = X * E[d][i0][j0][t];
            w = X * D[d][i0][j0][t] + dX * E[d][i0][j0][t];
          }
          if (t > 0) {
            v += i2p * E[d][i0][j0][t - 1];
            w += i2p * D[d][i0][j0][t - 1];
          }
          if (t + 1 <= i + j - 1) {
            v += (t + 1) * E[d][i0][j0][t + 1];
            w += (t + 1) * D[d][i0][j0][t + 1];
          }
          E[d][i][j][t] = v;
          D[d][i][j][t] = w;
        }
      }
  }
  const int first = a.prb[pr], nnz = a.pair_nnz[pr];
  const long long o0 = a.eoff[pr] + (long long)(pp - first) * nnz;
  double* e = a.E64 + o0;
  double* r = a.ER + 3 * o0;
  for (int xa = la; xa >= 0; --xa)
    for (int ya = la - xa; ya >= 0; --ya)
      for (int xb = lb; xb >= 0; --xb)
        for (int yb = lb - xb; yb >= 0; --yb) {
          const int za = la - xa - ya, zb = lb - xb - yb;
          const double c = kSqrtTwoPi52 * K * comp_norm(xa) * comp_norm(ya) * comp_norm(za) * comp_norm(xb) *
                           comp_norm(yb) * comp_norm(zb);
          for (int t = 0; t <= xa + xb; ++t)
            for (int u = 0; u <= ya + yb; ++u)
              for (int v = 0; v <= za + zb; ++v, ++e, ++r) {
                const double ex = E[0][xa][xb][t], ey = E[1][ya][yb][u], ez = E[2][za][zb][v];
                *e = c * ex * ey * ez;
                r[0] = c * D[0][xa][xb][t] * ey * ez;
                r[nnz] = c * ex * D[1][ya][yb][u] * ez;
                r[2 * nnz] = c * ex * ey * D[2][za][zb][v];
              }
        }
}

// ------------------------------------------------------------------ compile-time tables
constexpr int hcount(int L) { return (L + 1) * (L + 2) * (L + 3) / 6; }
// Hermite index by order n = t+u+v, then t descending, then u descending (gen_md.herm)
constexpr int hidx(int t, int u, int v) {
  const int n = t + u + v, m = n - t;
  return n * (n + 1) * (n + 2) / 6 + m * (m + 1) / 2 + (m - u);
}

template <int LA, int LB>
struct PairTab {
  static constexpr int NA = ncart(LA), NB = ncart(LB), NAB = NA * NB, L = LA + LB, HP = hcount(L);
  static constexpr int count() {
    int n = 0;
    for (int ca = 0; ca < NA; ++ca)
      for (int cb = 0; cb < NB; ++cb) {
        const int x = comp_x(LA, ca) + comp_x(LB, cb), y = comp_y(LA, ca) + comp_y(LB, cb);
        n += (x + 1) * (y + 1) * (L - x - y + 1);
      }
    return n;
  }
  static constexpr int NNZ = count();
  struct Data {
    unsigned char h[NNZ];           // Hermite index of every term of E'
    unsigned short off[NAB + 1];    // first term of every component pair
  };
  static constexpr Data make() {
    Data d{};
    int n = 0, k = 0;
    for (int ca = 0; ca < NA; ++ca)
      for (int cb = 0; cb < NB; ++cb) {
        const int x = comp_x(LA, ca) + comp_x(LB, cb), y = comp_y(LA, ca) + comp_y(LB, cb), z = L - x - y;
        d.off[k++] = (unsigned short)n;
        for (int t = 0; t <= x; ++t)
          for (int u = 0; u <= y; ++u)
            for (int v = 0; v <= z; ++v) d.h[n++] = (unsigned char)hidx(t, u, v);
      }
    d.off[k] = (unsigned short)n;
    return d;
  }
};

template <int LA, int LB, int LC, int LD>
struct GradTab {
  using B = PairTab<LA, LB>;
  using K = PairTab<LC, LD>;
  static constexpr int M = B::L + K::L + 1, HM = hcount(M), HP = B::HP, HQ = K::HP, HQ1 = hcount(K::L + 1);
  static constexpr int CS = (HQ1 + 3) & ~3;  // row of comb, a multiple of four
  struct alignas(4) Data {
    typename B::Data bra;
    typename K::Data ket;
    unsigned char comb[HP * CS];   // index of h + k in the order-M table (padding: 0)
    unsigned char down[3 * HQ1];   // index of k - 1_d (255: none)
    unsigned char odd[HQ];         // parity of k
    unsigned short first[HQ + 1];  // the ket terms by Hermite index: first one, component pair, term
    unsigned char cd[K::NNZ];
    unsigned short term[K::NNZ];
    // recursion step of every entry of the order-M table: coordinate, factor, the two sources
    unsigned char rd[HM], rc[HM], r1[HM], r2[HM];
  };
  static constexpr Data make() {
    Data d{};
    d.bra = B::make();
    d.ket = K::make();
    int n = 0;
    for (int h = 0; h < HQ; ++h) {
      d.first[h] = (unsigned short)n;
      for (int cd = 0; cd < K::NAB; ++cd)
        for (int t = d.ket.off[cd]; t < d.ket.off[cd + 1]; ++t)
          if (d.ket.h[t] == h) {
            d.cd[n] = (unsigned char)cd;
            d.term[n++] = (unsigned short)t;
          }
    }
    d.first[HQ] = (unsigned short)n;
    for (int t = 0; t <= M; ++t)
      for (int u = 0; u <= M - t; ++u)
        for (int v = 0; v <= M - t - u; ++v) {
          const int i = hidx(t, u, v), n = t + u + v;
          if (n > 0) {
            const int c = t > 0 ? 0 : (u > 0 ? 1 : 2), m = c == 0 ? t : (c == 1 ? u : v);
            d.rd[i] = (unsigned char)c;
            d.rc[i] = (unsigned char)(m - 1);
            d.r1[i] = (unsigned char)hidx(t - (c == 0), u - (c == 1), v - (c == 2));
            d.r2[i] = (unsigned char)(m > 1 ? hidx(t - 2 * (c == 0), u - 2 * (c == 1), v - 2 * (c == 2)) : 0);
          }
          if (n <= K::L) d.odd[i] = (unsigned char)(n & 1);
          if (n <= K::L + 1) {
            d.down[i] = (unsigned char)(t > 0 ? hidx(t - 1, u, v) : 255);
            d.down[HQ1 + i] = (unsigned char)(u > 0 ? hidx(t, u - 1, v) : 255);
            d.down[2 * HQ1 + i] = (unsigned char)(v > 0 ? hidx(t, u, v - 1) : 255);
            for (int a = 0; a <= B::L; ++a)
              for (int b = 0; b <= B::L - a; ++b)
                for (int c = 0; c <= B::L - a - b; ++c)
                  d.comb[hidx(a, b, c) * CS + i] = (unsigned char)hidx(a + t, b + u, c + v);
          }
        }
    return d;
  }
};

// R^(n)_000, n = 0..M, with the sqrt(alpha) of the ERI code.  M = 9 ((dd|dd)) is one order
// past the Boys table: its series and downward recursion below T = 48, else upward
// recursion off F_0
template <int M>
__device__ __forceinline__ void hermite_r0_grad(const Geometry& g, const double4_32a& a, const double4_32a& b,
                                                double* Rn, double& X, double& Y, double& Z) {
  if constexpr (M <= kBoysLMax) {
    Ctx<double> c;
    c.g = &g;
    c.nasym = 0;
    c.template hermite_r0_pp<M>(a, b, Rn, X, Y, Z);
  } else {
    X = a.y - b.y;
    Y = a.z - b.z;
    Z = a.w - b.w;
    const double r = rsqrt_dd(a.x + b.x), alpha = r * r;
    const double T = alpha * fma(X, X, fma(Y, Y, Z * Z)), e = exp(-T);
    double F[M + 1];
    if (T < 48.0) {
      double term = 1.0 / (2 * M + 1), sum = term;
      for (int i = 0; i < 400; ++i) {
        term *= 2.0 * T / (2 * M + 2 * i + 3);
        sum += term;
        if (term < 1e-17 * sum) break;
      }
      F[M] = e * sum;
      for (int m = M; m > 0; --m) F[m - 1] = (2.0 * T * F[m] + e) / (2 * m - 1);
    } else {
      F[0] = kHalfSqrtPi * rsqrt(T);
      for (int m = 0; m < M; ++m) F[m + 1] = ((2 * m + 1) * F[m] - e) / (2.0 * T);
    }
    double c = r;
    for (int n = 0; n <= M; ++n) {
      Rn[n] = c * F[n];
      c *= -2.0 * alpha;
    }
  }
}

// Coefficients of the ket functions contracted with the density weights of one bra component
// pair: k[0] = sum_cd Gam_cd (-1)^|k| E'_cd, k[1..3] the same with the derivatives of E'.
template <class GT, bool DYN, class Tab>
__device__ __forceinline__ void ket_rows(const Tab& tab, const double* gam, const double* __restrict__ e,
                                         const double* __restrict__ r, double* k) {
  using K = typename GT::K;
  constexpr int U = DYN ? 1 : 64;
#pragma unroll U
  for (int h = 0; h < GT::HQ; ++h) {
    double s[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll U
    for (int q = tab.first[h]; q < tab.first[h + 1]; ++q) {
      const double w = gam[tab.cd[q]];
      const int t = tab.term[q];
      s[0] = fma(w, __ldg(e + t), s[0]);
#pragma unroll
      for (int d = 0; d < 3; ++d) s[d + 1] = fma(w, __ldg(r + d * K::NNZ + t), s[d + 1]);
    }
#pragma unroll
    for (int d = 0; d < 4; ++d) k[d * GT::HQ + h] = flip_sign(s[d], tab.odd[h]);
  }
}

// ------------------------------------------------------------------ two-electron terms
// Every unique function quartet counts once, with the degeneracy of cython/fock.pyx:60-70
// and the density factor 2 P_ij P_kl - (P_ik P_jl + P_il P_jk) / 2 (the exchange term
// averaged over the quartet's permutations).  With the ket rows k above and the Hermite
// integrals R of a primitive quartet, per bra component pair ab
//     x_k = sum_h E'_h R_{h+k}:   dP_d += k0[k - 1_d] x_k,   dS_d += k_d[k] x_k
//     y_h = sum_k k0[k] R_{h+k}:  dR_d += (dE'_h/d(A-B)_d) y_h
// give the derivatives with respect to P, C - D and A - B; centres A, B, C, D follow from
// the chain rule above and translational invariance.
//
// 2^lg lanes share a shell quartet: first its primitive pairs, then its bra component
// pairs (R is then recomputed by every lane: the long high-L quartets are few and their
// chain is what a launch waits for).  Buckets and lanes as in k_tensor; quartets with
// Q_ab Q_cd below qtol are skipped (inside a bucket the lists are sorted by Q).  Classes up
// to L = 2 are unrolled, their tables folded away; the others run their loops over tables in
// shared memory with R and the ket rows in local memory: an FP64 warp instruction holds
// its pipe for 64 cycles, so the index work and L1 traffic around it are nearly free.  The
// kernel before this one (a warp per quartet, every lane the whole recursion, each function
// quartet its own sums) took 103 of a gradient's 119 ms on (H2O)2 6-31G**; the whole
// gradient is 2.7 ms now, bound by the chains of the d classes (lanes per quartet up to
// 32, 128, 256: 4.5, 3.1, 3.0 ms; those classes launched first: 2.7).
constexpr int kGradThreads = 128;
constexpr int kGradMaxLg = 8;     // up to 256 lanes (eight warps) per shell quartet
constexpr int kGradStore = 400;   // ket rows kept over the bra primitives up to this many doubles

template <int LA, int LB, int LC, int LD>
__global__ void __launch_bounds__(kGradThreads) k_grad_two(GradArgs a, Geometry g, ClassLaunch cl, TensorBuckets tb,
                                                           unsigned long long* work) {
  using GT = GradTab<LA, LB, LC, LD>;
  using B = typename GT::B;
  using K = typename GT::K;
  constexpr int M = GT::M, HQ = GT::HQ, HQ1 = GT::HQ1, NAB = B::NAB, NCD = K::NAB;
  constexpr bool DYN = B::L + K::L > 2;
  constexpr int U = DYN ? 1 : 256;
  constexpr bool STORE = NAB * 4 * HQ <= kGradStore;
  __shared__ BucketPlan<unsigned long long> plan;
  __shared__ typename GT::Data s_tab;
  static constexpr typename GT::Data ctab = GT::make();
  if constexpr (DYN)
    for (int x = threadIdx.x; x < (int)sizeof(s_tab) / 4; x += kGradThreads)
      reinterpret_cast<unsigned*>(&s_tab)[x] = reinterpret_cast<const unsigned*>(&ctab)[x];
  const int nkeys = tb.nbg * tb.nkg;
  plan_buckets(plan, nkeys, 1, (long long)gridDim.x * kGradThreads,
               [&](int k) { return bucket_quartets(tb, cl.same, k); },
               [&](int k) { return tb.bw[k / tb.nkg] * tb.kw[k % tb.nkg] * (DYN ? NAB : 1); }, kGradMaxLg);
  const auto& tab = [&]() -> const typename GT::Data& {
    if constexpr (DYN) return s_tab;
    else return ctab;
  }();
  const int lane = threadIdx.x & 31;
  double* grad = a.grad + (long long)(blockIdx.x % kGradCopies) * 3 * a.natom;
  const int N = a.N;
  int x = 0;
  for (;;) {
    unsigned long long base = 0;
    if (lane == 0) base = atomicAdd(work, 32ull);
    base = __shfl_sync(0xffffffffu, base, 0);
    if (base >= plan.pre[nkeys]) break;  // (kept in a register, it cost the d classes spills)
    const unsigned long long r = base + lane;
    while (r >= plan.pre[x + 1]) ++x;
    const int lg = plan.lg[x], key = nkeys - 1 - x, wl = min(lg, 5);  // wl: the group's lanes in this warp
    const unsigned long long slot = (r - plan.pre[x]) >> lg;
    if (slot >= bucket_quartets(tb, cl.same, key)) continue;
    int ib, jk;
    bucket_slot(tb, cl.same, key, slot, ib, jk);
    const int bp = __ldg(cl.bra + ib), kp = __ldg(cl.ket + jk);
    if (a.Qpair && (double)__ldg(a.Qpair + bp) * (double)__ldg(a.Qpair + kp) < a.qtol) continue;
    const int sa = __ldg(a.pa + bp), sb = __ldg(a.pb + bp), sc = __ldg(a.pa + kp), sd = __ldg(a.pb + kp);
    // ---- this lane's share
    const int nb = __ldg(a.prc + bp), nk = __ldg(a.prc + kp);
    const int lgb = min(lg, 31 - __clz(nb)), lgk = min(lg - lgb, 31 - __clz(nk)), lga = lg - lgb - lgk;
    const int sub = (int)((unsigned)(r - plan.pre[x]) & ((1u << lg) - 1u));
    const int s0 = sub & ((1 << lgb) - 1), s1 = (sub >> lgb) & ((1 << lgk) - 1), s2 = sub >> (lgb + lgk);
    const int step = DYN ? 1 << lga : 1, ab0 = DYN ? s2 : 0;
    const int i0 = (s0 * nb) >> lgb, i1 = ((s0 + 1) * nb) >> lgb;
    const int j0 = (s1 * nk) >> lgk, j1 = !DYN && s2 > 0 ? j0 : ((s1 + 1) * nk) >> lgk;
    // ---- density weights of one bra component pair's unique function quartets (0: not
    // counted here), kept where the ket rows are
    double gam[STORE ? NAB * NCD : NCD];
    auto weights = [&](int ab, double* w) {
      const int ca = ab / B::NB, cb = ab - ca * B::NB;
      const int f0 = __ldg(a.func + sa * kMaxComp + ca), f1 = __ldg(a.func + sb * kMaxComp + cb);
#pragma unroll U
      for (int cd = 0; cd < NCD; ++cd) {
        const int cc = cd / K::NB, ce = cd - cc * K::NB;
        int i = f0, j = f1, k = __ldg(a.func + sc * kMaxComp + cc), l = __ldg(a.func + sd * kMaxComp + ce);
        const bool skip = (sa == sb && ca < cb) || (sc == sd && cc < ce) || (bp == kp && ab < cd) ||
                          (i | j | k | l) < 0;
        w[cd] = 0.0;
        if (skip) continue;
        if (i < j) { const int t = i; i = j; j = t; }
        if (k < l) { const int t = k; k = l; l = t; }
        if (i < k || (i == k && j < l)) {
          int t = i; i = k; k = t;
          t = j; j = l; l = t;
        }
        const double* Pm = a.P;
        const double dir = __ldg(Pm + (long long)i * N + j) * __ldg(Pm + (long long)k * N + l);
        const double ex = fma(__ldg(Pm + (long long)i * N + k), __ldg(Pm + (long long)j * N + l),
                              __ldg(Pm + (long long)i * N + l) * __ldg(Pm + (long long)j * N + k));
        const int deg = (i != j) + (k != l) + !(i == k && j == l);
        w[cd] = __hiloint2double((1023 + deg) << 20, 0) * fma(-0.5, ex, 2.0 * dir);
      }
    };
    if constexpr (STORE) {
#pragma unroll U
      for (int ab = ab0; ab < NAB; ab += step) weights(ab, gam + (DYN ? ab >> lga : ab) * NCD);
    }
    double gA[3] = {0, 0, 0}, gP[3] = {0, 0, 0}, gC[3] = {0, 0, 0};
    const int b0 = __ldg(a.prb + bp), k0 = __ldg(a.prb + kp);
    const long long eb = __ldg(a.eoff + bp), ek = __ldg(a.eoff + kp);
    double krow[STORE ? NAB * 4 * HQ : 4 * HQ];
    for (int j = j0; j < j1; ++j) {
      const double* __restrict__ ke = a.E64 + ek + (long long)j * K::NNZ;
      const double* __restrict__ kr = a.ER + 3 * (ek + (long long)j * K::NNZ);
      if (STORE) {
#pragma unroll U
        for (int ab = ab0; ab < NAB; ab += step)
          ket_rows<GT, DYN>(tab, gam + (DYN ? ab >> lga : ab) * NCD, ke, kr, krow + (DYN ? ab >> lga : ab) * 4 * HQ);
      }
      const double4_32a qb = g.pP[k0 + j];
      const double fc = __ldg(a.frac + k0 + j);
      for (int i = i0; i < i1; ++i) {
        double Rn[M + 1], X, Y, Z, R[GT::HM];
        hermite_r0_grad<M>(g, g.pP[b0 + i], qb, Rn, X, Y, Z);
        R[0] = Rn[M];
#pragma unroll U
        for (int s = 1; s <= M; ++s) {
#pragma unroll U
          for (int q = hcount(s) - 1; q > 0; q -= 4) {  // four at a time: every source is read before a write
            double v[4];
#pragma unroll
            for (int z = 0; z < 4; ++z) {
              if (q - z <= 0) continue;
              const int c = tab.rd[q - z], m = tab.rc[q - z];
              v[z] = (c == 0 ? X : (c == 1 ? Y : Z)) * R[tab.r1[q - z]];
              if (m > 0) v[z] = fma(a.small[m], R[tab.r2[q - z]], v[z]);
            }
#pragma unroll
            for (int z = 0; z < 4; ++z)
              if (q - z > 0) R[q - z] = v[z];
          }
          R[0] = Rn[M - s];
        }
        const double* __restrict__ be = a.E64 + eb + (long long)i * B::NNZ;
        const double* __restrict__ br = a.ER + 3 * (eb + (long long)i * B::NNZ);
        double tP[3] = {0, 0, 0}, tR[3] = {0, 0, 0}, tS[3] = {0, 0, 0};
#pragma unroll U
        for (int ab = ab0; ab < NAB; ab += step) {
          double* kq = STORE ? krow + (DYN ? ab >> lga : ab) * 4 * HQ : krow;
          if constexpr (!STORE) {
            weights(ab, gam);
            ket_rows<GT, DYN>(tab, gam, ke, kr, kq);
          }
          const int t0 = tab.bra.off[ab], t1 = tab.bra.off[ab + 1];
#pragma unroll U
          for (int k = 0; k < GT::CS; k += 4) {
            double xk[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll U
            for (int t = t0; t < t1; ++t) {
              const double e = __ldg(be + t);
              const unsigned char* row = tab.comb + tab.bra.h[t] * GT::CS + k;
#pragma unroll
              for (int z = 0; z < 4; ++z) xk[z] = fma(e, R[row[z]], xk[z]);
            }
#pragma unroll
            for (int z = 0; z < 4; ++z) {
              if (k + z >= HQ1) continue;
#pragma unroll
              for (int d = 0; d < 3; ++d) {
                const int low = tab.down[d * HQ1 + k + z];
                if (low != 255) tP[d] = fma(kq[low], xk[z], tP[d]);
                if (k + z < HQ) tS[d] = fma(kq[(d + 1) * HQ + k + z], xk[z], tS[d]);
              }
            }
          }
#pragma unroll U
          for (int t = t0; t < t1; ++t) {
            const unsigned char* row = tab.comb + tab.bra.h[t] * GT::CS;
            double y0 = 0.0, y1 = 0.0;
#pragma unroll U
            for (int k = 0; k + 1 < HQ; k += 2) {
              y0 = fma(kq[k], R[row[k]], y0);
              y1 = fma(kq[k + 1], R[row[k + 1]], y1);
            }
            if (HQ & 1) y0 = fma(kq[HQ - 1], R[row[HQ - 1]], y0);
            const double yh = y0 + y1;
#pragma unroll
            for (int d = 0; d < 3; ++d) tR[d] = fma(__ldg(br + d * B::NNZ + t), yh, tR[d]);
          }
        }
        const double fa = __ldg(a.frac + b0 + i);
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          gP[d] += tP[d];
          gA[d] += fma(fa, tP[d], tR[d]);
          gC[d] += fma(-fc, tP[d], tS[d]);
        }
      }
    }
    // ---- sums over the group's lanes in this warp, then the four centres
    const unsigned mask = (wl == 5 ? 0xffffffffu : ((1u << (1 << wl)) - 1u)) << (lane & ~((1 << wl) - 1));
    for (int o = 1; o < (1 << wl); o <<= 1)
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        gA[d] += __shfl_xor_sync(mask, gA[d], o);
        gP[d] += __shfl_xor_sync(mask, gP[d], o);
        gC[d] += __shfl_xor_sync(mask, gC[d], o);
      }
    if ((sub & ((1 << wl) - 1)) == 0) {
      const int at[4] = {__ldg(a.shell_atom + sa), __ldg(a.shell_atom + sb), __ldg(a.shell_atom + sc),
                         __ldg(a.shell_atom + sd)};
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        atomicAdd(grad + 3 * at[0] + d, gA[d]);
        atomicAdd(grad + 3 * at[1] + d, gP[d] - gA[d]);
        atomicAdd(grad + 3 * at[2] + d, gC[d]);
        atomicAdd(grad + 3 * at[3] + d, -(gP[d] + gC[d]));
      }
    }
  }
}

// ------------------------------------------------------------------ one-electron terms
// Nuclear attraction of the pairs of one class: one warp per shell pair, its lanes over
// (primitive pair, nucleus).  The Hermite density of the primitive pair, D_h = sum_ab
// P_ab E'_h, and its derivatives meet R_h(p, P - C): d/dP on the pair and with the
// opposite sign on the nucleus (its Hellmann-Feynman term), d/d(A-B) on the centres.
template <int LA, int LB>
__global__ void __launch_bounds__(kGradThreads) k_grad_nuclei(GradArgs a, Geometry g, const int* list, int n) {
  using B = PairTab<LA, LB>;
  constexpr int M = B::L + 1, HP = B::HP;
  constexpr typename B::Data tab = B::make();
  const int w = (int)((blockIdx.x * (long long)kGradThreads + threadIdx.x) >> 5), lane = threadIdx.x & 31;
  if (w >= n) return;
  const int pr = list[w], sa = a.pa[pr], sb = a.pb[pr];
  const int count = a.prc[pr], first = a.prb[pr];
  double* grad = a.grad + (long long)(blockIdx.x % kGradCopies) * 3 * a.natom;
  double gA[3] = {0, 0, 0}, gP[3] = {0, 0, 0};
  // attraction -Z (2 pi / p) K E ... from E' = sqrt(2 pi^{5/2}) K p^{-3/2} E ...; both orders of two
  // different shells, and 2 P_ij
  const double pre = -2.0 * kPi / kSqrtTwoPi52 * 2.0 * (sa == sb ? 1.0 : 2.0);
  for (int it = lane; it < count * a.natom; it += 32) {
    const int k = it / a.natom, c = it - k * a.natom;
    const long long o = a.eoff[pr] + (long long)k * B::NNZ;
    const double* __restrict__ e = a.E64 + o;
    const double* __restrict__ er = a.ER + 3 * o;
    double D[4][HP];
#pragma unroll
    for (int h = 0; h < HP; ++h) D[0][h] = D[1][h] = D[2][h] = D[3][h] = 0.0;
#pragma unroll
    for (int ab = 0; ab < B::NAB; ++ab) {
      const int i = __ldg(a.func + sa * kMaxComp + ab / B::NB), j = __ldg(a.func + sb * kMaxComp + ab % B::NB);
      const double p = (i | j) < 0 ? 0.0 : __ldg(a.P + (long long)i * a.N + j);
#pragma unroll
      for (int t = tab.off[ab]; t < tab.off[ab + 1]; ++t) {
        D[0][tab.h[t]] = fma(p, __ldg(e + t), D[0][tab.h[t]]);
#pragma unroll
        for (int d = 0; d < 3; ++d) D[d + 1][tab.h[t]] = fma(p, __ldg(er + d * B::NNZ + t), D[d + 1][tab.h[t]]);
      }
    }
    const double4_32a pp = g.pP[first + k];
    const double pe = 1.0 / pp.x;  // p
    const double X = pp.y - a.xyz[3 * c], Y = pp.z - a.xyz[3 * c + 1], Z = pp.w - a.xyz[3 * c + 2];
    double F[M + 1], R[hcount(M)];
    boys_eval<M>(g.boys64, pe * fma(X, X, fma(Y, Y, Z * Z)), F);
    double f = pre * sqrt(pe) * a.Z[c];
#pragma unroll
    for (int m = 0; m <= M; ++m) {
      F[m] *= f;
      f *= -2.0 * pe;
    }
    R[0] = F[M];
#pragma unroll
    for (int s = 1; s <= M; ++s) {
#pragma unroll
      for (int t = s; t >= 0; --t)
#pragma unroll
        for (int u = s - t; u >= 0; --u)
#pragma unroll
          for (int v = s - t - u; v >= 0; --v) {
            double val;
            if (t > 0) val = X * R[hidx(t - 1, u, v)] + (t > 1 ? (t - 1) * R[hidx(t - 2, u, v)] : 0.0);
            else if (u > 0) val = Y * R[hidx(0, u - 1, v)] + (u > 1 ? (u - 1) * R[hidx(0, u - 2, v)] : 0.0);
            else if (v > 0) val = Z * R[hidx(0, 0, v - 1)] + (v > 1 ? (v - 1) * R[hidx(0, 0, v - 2)] : 0.0);
            else val = F[M - s];
            R[hidx(t, u, v)] = val;
          }
    }
    double tP[3] = {0, 0, 0}, tR[3] = {0, 0, 0};
#pragma unroll
    for (int t = 0; t <= B::L; ++t)
#pragma unroll
      for (int u = 0; u <= B::L - t; ++u)
#pragma unroll
        for (int v = 0; v <= B::L - t - u; ++v) {
          const int h = hidx(t, u, v);
          tP[0] = fma(D[0][h], R[hidx(t + 1, u, v)], tP[0]);
          tP[1] = fma(D[0][h], R[hidx(t, u + 1, v)], tP[1]);
          tP[2] = fma(D[0][h], R[hidx(t, u, v + 1)], tP[2]);
#pragma unroll
          for (int d = 0; d < 3; ++d) tR[d] = fma(D[d + 1][h], R[h], tR[d]);
        }
    const double fa = a.frac[first + k];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      gP[d] += tP[d];
      gA[d] += fma(fa, tP[d], tR[d]);
      atomicAdd(grad + 3 * c + d, -tP[d]);
    }
  }
  const int atA = a.shell_atom[sa], atB = a.shell_atom[sb];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    for (int o = 16; o > 0; o >>= 1) {
      gA[d] += __shfl_xor_sync(0xffffffffu, gA[d], o);
      gP[d] += __shfl_xor_sync(0xffffffffu, gP[d], o);
    }
    if (lane == 0) {
      atomicAdd(grad + 3 * atA + d, gA[d]);
      atomicAdd(grad + 3 * atB + d, gP[d] - gA[d]);
    }
  }
}

// 1D Hermite expansion coefficients E[i][j][t] of G_i(x; a, A) G_j(x; b, B) for
// i <= imax, j <= jmax (cython/util.pxi:13-28 recursion; the Gaussian factor is
// applied by the caller)
struct E1 {
  double v[kEi][kEj][kEt];
};

__device__ void hermite_1d(E1& E, int imax, int jmax, double p, double XPA, double XPB) {
  const double i2p = 0.5 / p;
  for (int i = 0; i <= imax; ++i)
    for (int j = 0; j <= jmax; ++j)
      for (int t = 0; t < kEt; ++t) E.v[i][j][t] = 0.0;
  E.v[0][0][0] = 1.0;
  for (int i = 0; i < imax; ++i)
    for (int t = 0; t <= i + 1; ++t) {
      double v = XPA * E.v[i][0][t];
      if (t > 0) v += i2p * E.v[i][0][t - 1];
      if (t + 1 <= i) v += (t + 1) * E.v[i][0][t + 1];
      E.v[i + 1][0][t] = v;
    }
  for (int j = 0; j < jmax; ++j)
    for (int i = 0; i <= imax; ++i)
      for (int t = 0; t <= i + j + 1 && t < kEt; ++t) {
        double v = XPB * E.v[i][j][t];
        if (t > 0) v += i2p * E.v[i][j][t - 1];
        if (t + 1 <= i + j) v += (t + 1) * E.v[i][j][t + 1];
        E.v[i][j + 1][t] = v;
      }
}

// Overlap and kinetic terms (d/dB = -d/dA): one warp per shell pair, its lanes over the
// primitive pairs (one thread per pair was a chain of up to 36 of them).
__global__ void __launch_bounds__(64) k_grad_one(GradArgs a) {
  const int pr = (int)((blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
  if (pr >= a.npair) return;
  const int sa = a.pa[pr], sb = a.pb[pr];
  const int la = a.L[sa], lb = a.L[sb];
  const int Ka = a.nprim[sa], Kb = a.nprim[sb];
  const double A[3] = {a.center[3 * sa], a.center[3 * sa + 1], a.center[3 * sa + 2]};
  const double B[3] = {a.center[3 * sb], a.center[3 * sb + 1], a.center[3 * sb + 2]};
  const double fac = sa == sb ? 1.0 : 2.0;  // (i, j) and (j, i) of two different shells
  const int nca = ncart(la), ncb = ncart(lb);
  double gA[3] = {0, 0, 0};
  E1 E[3];
  for (int kk = lane; kk < Ka * Kb; kk += 32) {
    const int ka = kk / Kb, kb = kk - ka * Kb;
    const double ea = a.exps[a.poff[sa] + ka], eb = a.exps[a.poff[sb] + kb];
    const double p = ea + eb, mu = ea * eb / p;
    double AB2 = 0.0;
    for (int d = 0; d < 3; ++d) AB2 += (A[d] - B[d]) * (A[d] - B[d]);
    const double K = exp(-mu * AB2) * a.coefs[a.poff[sa] + ka] * a.coefs[a.poff[sb] + kb];
    if (K == 0.0) continue;
    const double sq = sqrt(kPi / p);
    for (int d = 0; d < 3; ++d)
      hermite_1d(E[d], la + 1, lb + 2, p, -(eb / p) * (A[d] - B[d]), (ea / p) * (A[d] - B[d]));
    for (int ca = 0; ca < nca; ++ca) {
      const int fi = a.func[sa * kGradMaxComp + ca];
      if (fi < 0) continue;
      const int ia[3] = {comp_x(la, ca), comp_y(la, ca), la - comp_x(la, ca) - comp_y(la, ca)};
      for (int cb = 0; cb < ncb; ++cb) {
        const int fj = a.func[sb * kGradMaxComp + cb];
        if (fj < 0) continue;
        const int jb[3] = {comp_x(lb, cb), comp_y(lb, cb), lb - comp_x(lb, cb) - comp_y(lb, cb)};
        const double nrm = comp_norm(ia[0]) * comp_norm(ia[1]) * comp_norm(ia[2]) * comp_norm(jb[0]) *
                           comp_norm(jb[1]) * comp_norm(jb[2]);
        const double Pij = a.P[(long long)fi * a.N + fj], Wij = a.W[(long long)fi * a.N + fj];
        // 1D overlap S(i, j) and kinetic T(i, j) (cython/onee.pyx:103-133 decomposition)
        auto S1 = [&](int d, int i, int j) { return (i < 0 || j < 0) ? 0.0 : E[d].v[i][j][0] * sq; };
        auto T1 = [&](int d, int i, int j) {
          if (i < 0) return 0.0;
          double t = eb * (2 * j + 1) * S1(d, i, j) - 2.0 * eb * eb * S1(d, i, j + 2);
          if (j >= 2) t -= 0.5 * j * (j - 1) * S1(d, i, j - 2);
          return t;
        };
        for (int d = 0; d < 3; ++d) {
          // derivative in direction d of the bra: 2a f(i+1) - i f(i-1)
          double Sd[3], Td[3];
          for (int e = 0; e < 3; ++e) {
            if (e == d) {
              Sd[e] = 2.0 * ea * S1(e, ia[e] + 1, jb[e]) - ia[e] * S1(e, ia[e] - 1, jb[e]);
              Td[e] = 2.0 * ea * T1(e, ia[e] + 1, jb[e]) - ia[e] * T1(e, ia[e] - 1, jb[e]);
            } else {
              Sd[e] = S1(e, ia[e], jb[e]);
              Td[e] = T1(e, ia[e], jb[e]);
            }
          }
          const double dS = Sd[0] * Sd[1] * Sd[2];
          const double dT = Td[0] * Sd[1] * Sd[2] + Sd[0] * Td[1] * Sd[2] + Sd[0] * Sd[1] * Td[2];
          gA[d] += fac * K * nrm * (2.0 * Pij * dT - 2.0 * Wij * dS);
        }
      }
    }
  }
  double* grad = a.grad + (long long)(blockIdx.x % kGradCopies) * 3 * a.natom;
  const int atA = a.shell_atom[sa], atB = a.shell_atom[sb];
  for (int d = 0; d < 3; ++d) {
    for (int o = 16; o > 0; o >>= 1) gA[d] += __shfl_xor_sync(0xffffffffu, gA[d], o);
    if (lane == 0) {
      atomicAdd(grad + 3 * atA + d, gA[d]);
      atomicAdd(grad + 3 * atB + d, -gA[d]);
    }
  }
}

// the copies added into the first
__global__ void k_grad_sum(double* grad, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double s = 0.0;
  for (int c = 0; c < kGradCopies; ++c) s += grad[(long long)c * n + i];
  grad[i] = s;
}

template <int LA, int LB, int LC, int LD>
cudaError_t launch_two(const GradArgs& a, const Geometry& g, const ClassLaunch& cl, const TensorBuckets& tb,
                       unsigned long long* work, cudaStream_t st) {
  auto k = k_grad_two<LA, LB, LC, LD>;
  k<<<persistent_blocks(k, 0, 0, kGradThreads), kGradThreads, 0, st>>>(a, g, cl, tb, work);
  return cudaGetLastError();
}

}  // namespace

// Pair data and tables, then every term on its own kernel; the two-electron classes run on
// the nstreams side streams (one class's tail beside the next), joined into st at the end.
cudaError_t mmdg_launch_rhf_gradient(const GradArgs& a, const Geometry& g, const GradList* lists, int nstreams,
                                     const cudaStream_t* side, cudaEvent_t fork, const cudaEvent_t* join,
                                     cudaStream_t st) {
#define GRAD_TRY(x)                       \
  do {                                    \
    const cudaError_t e_ = (x);           \
    if (e_ != cudaSuccess) return e_;     \
  } while (0)
  if (a.npair <= 0) return cudaSuccess;
  GRAD_TRY(cudaMemsetAsync(a.grad, 0, sizeof(double) * 3 * a.natom * kGradCopies, st));
  GRAD_TRY(cudaMemsetAsync(a.work, 0, sizeof(unsigned long long) * kGradClasses, st));
  if (a.nprimpair > 0) {
    k_grad_pairs<<<(a.nprimpair + 63) / 64, 64, 0, st>>>(a);
    GRAD_TRY(cudaGetLastError());
  }
  if (nstreams > 1) {
    GRAD_TRY(cudaEventRecord(fork, st));
    for (int k = 0; k < nstreams; ++k) GRAD_TRY(cudaStreamWaitEvent(side[k], fork, 0));
  }
  // highest angular momentum first: its few quartets are the longest chains
  int ci = 0;
#define GRAD_CLASS(LA, LB, LC, LD)                                                                              \
  [&]() -> cudaError_t {                                                                                                             \
    const GradList &b = lists[LA * (LA + 1) / 2 + LB], &k = lists[LC * (LC + 1) / 2 + LD];                      \
    if (b.n && k.n) {                                                                                           \
      TensorBuckets tb;                                                                                         \
      tb.nbg = b.ngroup;                                                                                        \
      tb.nkg = k.ngroup;                                                                                        \
      for (int x = 0; x <= b.ngroup; ++x) tb.bstart[x] = b.start[x];                                            \
      for (int x = 0; x <= k.ngroup; ++x) tb.kstart[x] = k.start[x];                                            \
      for (int x = 0; x < b.ngroup; ++x) tb.bw[x] = b.prims[x];                                                 \
      for (int x = 0; x < k.ngroup; ++x) tb.kw[x] = k.prims[x];                                                 \
      const ClassLaunch cl{b.list, k.list, b.n, k.n, LA == LC && LB == LD};                  \
      return launch_two<LA, LB, LC, LD>(a, g, cl, tb, a.work + ci, nstreams > 1 ? side[ci % nstreams] : st);    \
    }                                                                                                           \
    return cudaSuccess;                                                                                         \
  },
  const std::function<cudaError_t()> classes[] = {MMDG_FOR_EACH_CLASS(GRAD_CLASS)};
#undef GRAD_CLASS
  for (ci = kGradClasses - 1; ci >= 0; --ci) GRAD_TRY(classes[ci]());
  k_grad_one<<<(unsigned)((a.npair * 32LL + 63) / 64), 64, 0, st>>>(a);
  GRAD_TRY(cudaGetLastError());
#define GRAD_NUCLEI(LA, LB)                                                                                 \
  {                                                                                                         \
    const GradList& b = lists[LA * (LA + 1) / 2 + LB];                                                      \
    if (b.n) {                                                                                              \
      k_grad_nuclei<LA, LB><<<(unsigned)((b.n * 32LL + kGradThreads - 1) / kGradThreads), kGradThreads, 0, st>>>( \
          a, g, b.list, b.n);                                                                               \
      GRAD_TRY(cudaGetLastError());                                                                         \
    }                                                                                                       \
  }
  GRAD_NUCLEI(0, 0) GRAD_NUCLEI(1, 0) GRAD_NUCLEI(1, 1) GRAD_NUCLEI(2, 0) GRAD_NUCLEI(2, 1) GRAD_NUCLEI(2, 2)
#undef GRAD_NUCLEI
  if (nstreams > 1)
    for (int k = 0; k < nstreams; ++k) {
      GRAD_TRY(cudaEventRecord(join[k], side[k]));
      GRAD_TRY(cudaStreamWaitEvent(st, join[k], 0));
    }
  k_grad_sum<<<(3 * a.natom + 127) / 128, 128, 0, st>>>(a.grad, 3 * a.natom);
  return cudaGetLastError();
#undef GRAD_TRY
}
