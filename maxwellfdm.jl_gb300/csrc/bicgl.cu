// BiCGStab(ℓ) (Sleijpen & Fokkema, ETNA 1, 1993), ℓ ≤ 4, for the same
// systems as BiCGSTAB: ℓ BiCG steps followed by a minimal-residual
// polynomial of degree ℓ.  On the FDFD operator, whose spectrum has large
// imaginary parts, the degree-1 polynomial of BiCGSTAB stalls where the
// degree-ℓ one does not; it needs markedly fewer operator applications in
// both precisions, for about 1.3× the vector traffic per application.
//
// One cycle = 4ℓ + 2 kernels, all reading their scalars from device memory
// (so a batch of cycles replays as one CUDA graph):
//   for j = 0 … ℓ−1:
//     u_j = r_j − β u_j                              k_bl_step
//     u_{j+1} = A u_j, γ = (r̂, u_{j+1}), α = ρ/γ     operator, EPI_DOT_SHD + FIN_ALPHA
//     r_j −= α u_{j+1}                               k_bl_step
//     r_{j+1} = A r_j [, ρ₁ = (r̂, r_{j+1}), β]       operator, EPI_DOT_SHD + FIN_BL_RHO
// r̂ is the generated shadow vector (shadow() in krylov_fin.cuh): no
// memory traffic for it.
//   Gram matrix of r_0 … r_ℓ and, in its last block, the
//   minimal-residual coefficients γ from it                   k_bl_gram
//   x, r_0, u_0 closing update, (r̂, r_0), ‖r_0‖², stop tests  k_bl_fin + FIN_BL_CYCLE
// Only the operator's inputs u_j and r_j are updated as the cycle goes.  The
// lower vectors' updates of step j — u_i = r_i − β_j u_i, x += α_j u_0,
// r_i −= α_j u_{i+1} for i < j — are never stored: k_bl_gram and k_bl_fin
// read those vectors anyway and replay the steps in registers from the saved
// α_j and β_j (Replay below; only r_0, u_0 and x outlive the cycle).  A
// cycle of ℓ = 4 makes 46 vector passes instead of the 73 that storing them
// took (96³ complex64: the solve 1.29× faster).  In complex128 a complex
// product costs more than three vector passes (FP64 pipe), so there k_bl_gram
// stores the replayed vectors and x, and k_bl_fin does not replay them again:
// 55 passes.
// Vectors and products are in the solve's inner precision; every sum
// across threads and blocks is double-float FP32 (complex64) or FP64
// (complex128), in a fixed order.
// The grid-stride vector kernels run one full wave (SM count × the
// kernel's resident blocks per SM), so none ends on a partial wave.
#include <algorithm>
#include <mutex>
#include <unordered_map>

#include "krylov_fin.cuh"

namespace fdfd {

namespace {

constexpr int VB = 256;
constexpr int RED_BLOCKS = 152 * 4;
constexpr int LMAX = 4;

template <typename C>
struct VSet {
  C *v[LMAX + 1];
};

__device__ __forceinline__ double2 conjd(double2 a) { return make_double2(a.x, -a.y); }
__device__ __forceinline__ double2 subd(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double2 scd(double2 a, double s) { return make_double2(a.x * s, a.y * s); }

// y + s·v and y − s·v as four fused multiply-adds: six instructions as a
// product and a sum, and complex128 vectors are bound by the FP64 pipe.
// (32³ box, FP64, per launch: Gram kernel 54.8 → 37.9 µs, closing update
// 28.2 → 22.3, step 5.2 → 4.5; an application with its share of them 31.0 → 27.2.)
__device__ __forceinline__ float fmar(float a, float b, float c) { return fmaf(a, b, c); }
__device__ __forceinline__ double fmar(double a, double b, double c) { return fma(a, b, c); }
template <typename C>
__device__ __forceinline__ C addsv(C y, C s, C v) {
  return mk(fmar(-s.y, v.y, fmar(s.x, v.x, y.x)), fmar(s.y, v.x, fmar(s.x, v.y, y.y)));
}
template <typename C>
__device__ __forceinline__ C subsv(C y, C s, C v) {
  return mk(fmar(s.y, v.y, fmar(-s.x, v.x, y.x)), fmar(-s.y, v.x, fmar(-s.x, v.y, y.y)));
}

template <typename R>
__device__ __forceinline__ long long vstride() { return (long long)gridDim.x * VB; }

// Two consecutive complex elements per access (16-byte loads for complex64).
template <typename C> struct Pair { C a, b; };
__device__ __forceinline__ Pair<float2> ldp(const float2 *__restrict__ p, long long q) {
  const float4 v = reinterpret_cast<const float4 *>(p)[q];
  return {make_float2(v.x, v.y), make_float2(v.z, v.w)};
}
__device__ __forceinline__ Pair<double2> ldp(const double2 *__restrict__ p, long long q) {
  return {p[2 * q], p[2 * q + 1]};
}
__device__ __forceinline__ void stp(float2 *p, long long q, Pair<float2> v) {
  reinterpret_cast<float4 *>(p)[q] = make_float4(v.a.x, v.a.y, v.b.x, v.b.y);
}
__device__ __forceinline__ void stp(double2 *p, long long q, Pair<double2> v) {
  p[2 * q] = v.a;
  p[2 * q + 1] = v.b;
}

// Grid-stride visit of the n elements: complex64 in pairs (an odd tail
// element by block 0 thread 0), complex128 — 16 bytes each, and bound by the
// FP64 pipe on small systems, where pairs leave some threads one pair more
// than others — singly.
template <typename R, typename F2, typename F1>
__device__ __forceinline__ void visit(long long n, F2 f2, F1 f1) {
  if constexpr (sizeof(R) == 8) {
    for (long long e = blockIdx.x * (long long)VB + threadIdx.x; e < n; e += (long long)gridDim.x * VB) f1(e);
  } else {
    const long long np = n >> 1;
    for (long long q = blockIdx.x * (long long)VB + threadIdx.x; q < np; q += (long long)gridDim.x * VB) f2(q);
    if ((n & 1) && blockIdx.x == 0 && threadIdx.x == 0) f1(n - 1);
  }
}

// v −= s·w, the form of both BiCG updates: u_j = r_j − β u_j (out = u_j)
// and r_j −= α u_{j+1} (out = r_j).  Bound by HBM (3 vectors); saves the
// scalar for the cycle's end.
template <typename R>
__global__ void __launch_bounds__(VB) k_bl_step(const typename CT<R>::C *v, const typename CT<R>::C *w,
                                                typename CT<R>::C *out, long long n, int beta, int j, KScalars *sc) {
  using C = typename CT<R>::C;
  if (sc->done) return;
  C s1[1];
  scalars<R>([&](int) { return beta ? sc->beta : sc->alpha; }, s1);
  const C s = s1[0];
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    (beta ? sc->beta_j : sc->alpha_j)[j] = beta ? sc->beta : sc->alpha;
    sc->bl_steps = beta ? j : j + 1;
  }
  visit<R>(
      n,
      [&](long long q) {
        const Pair<C> a = ldp(v, q), b = ldp(w, q);
        stp(out, q, Pair<C>{subsv(a.a, s, b.a), subsv(a.b, s, b.b)});
      },
      [&](long long e) { out[e] = subsv(v[e], s, w[e]); });
}

// α_1 … α_{L−1} (index 0 … L−2), β_1 … β_{L−1}, then α_0, in one array
template <int L>
struct Hist {
  static constexpr int N = 2 * (L - 1) + 1;
  static __device__ __forceinline__ double2 at(const KScalars *sc, int i) {
    return i < L - 1 ? sc->alpha_j[i + 1] : i < 2 * (L - 1) ? sc->beta_j[i - (L - 1) + 1] : sc->alpha_j[0];
  }
};

// The steps j = 1 … L−1 of one element: r[0 … L−1] and u[0 … L−1] hold each
// vector as the operator read it (r_j, u_j of step j) and end as they stand
// after step L−1.  With X also x += Σ_j α_j u_0; without it u_0 is not used.
template <int L, bool X, typename C>
__device__ __forceinline__ void replay(C *r, C *u, C &x, const C *hist) {
  if (X) x = addsv(x, hist[2 * (L - 1)], u[0]);
#pragma unroll
  for (int j = 1; j < L; ++j) {
    const C al = hist[j - 1], be = hist[L - 1 + j - 1];
#pragma unroll
    for (int i = X ? 0 : 1; i < j; ++i) u[i] = subsv(r[i], be, u[i]);
    if (X) x = addsv(x, al, u[0]);
#pragma unroll
    for (int i = 0; i < j; ++i) r[i] = subsv(r[i], al, u[i + 1]);
  }
}

constexpr int pow2_at_least(int k) { return k <= 1 ? 1 : 2 * pow2_at_least((k + 1) / 2); }

// The minimal-residual step of a cycle from the Gram sums (gram: (r_i, r_j),
// 1 ≤ i ≤ j ≤ L, then (r_i, r_0), as (re, im) pairs): γ = argmin
// ‖r_0 − Σ γ_k r_k‖ by G = Tᴴ D T (T unit upper triangular — the modified
// Gram–Schmidt coefficients), T γ = D⁻¹ T⁻ᴴ g.  Written with the original
// r_k, the cycle's closing update is x += Σ γ_k r_{k−1}, r_0 −= Σ γ_k r_k,
// u_0 −= Σ γ_k u_k.  One warp, an entry (a, b) of the factorisation per
// lane: every FP64 instruction costs its 64 cycles for all entries at once
// (one thread working through them took 13.5 µs and a launch of its own: with it a
// BiCGStab(4) cycle of the 32³ box in FP64 took 36 µs more).
template <int L>
__device__ __forceinline__ void bl_mr(const double *gram, KScalars *sc) {
  const int lane = threadIdx.x & 31;
  // lane (a, b), 0 ≤ a < L, a ≤ b ≤ L (column L: the right-hand side);
  // lanes beyond hold a copy of entry (L−1, L)
  constexpr int NE = L * (L + 1) / 2 + L;
  int la = L - 1, lb = L;
  {
    int e = 0;
#pragma unroll
    for (int a = 0; a < L; ++a)
#pragma unroll
      for (int b = a; b <= L; ++b, ++e)
        if (lane == e) {
          la = a;
          lb = b;
        }
  }
  auto lane_of = [](int a, int b) { return a * (L + 1) - a * (a - 1) / 2 + (b - a); };
  double2 v;
  {
    const int q = lb < L ? lb * (lb + 1) / 2 + la : L * (L + 1) / 2 + la;
    v = make_double2(gram[2 * q], gram[2 * q + 1]);
  }
  auto from = [&](double2 t, int src) {
    return make_double2(__shfl_sync(0xffffffffu, t.x, src), __shfl_sync(0xffffffffu, t.y, src));
  };
  double2 tau = make_double2(0.0, 0.0);  // row a scaled: τ_ab, and γ' in column L
#pragma unroll
  for (int p = 0; p < L; ++p) {
    const double s = __shfl_sync(0xffffffffu, v.x, lane_of(p, p));
    if (!(s > 0.0) || !isfinite(s)) {
      if (lane == 0) {
        sc->done = 1;
        sc->reason = isfinite(s) ? 3 : 4;
      }
      return;
    }
    const double inv = 1.0 / s;
    if (la == p) tau = scd(v, inv);
    if (p + 1 < L) {
      // v_ab −= conj(v_pa) τ_pb for the rows below
      const double2 va = from(v, lane_of(p, la > p ? la : p));
      const double2 tb = from(tau, lane_of(p, lb > p ? lb : p));
      if (la > p) v = subd(v, dcmul(conjd(va), tb));
    }
  }
  // back substitution: γ_a = γ'_a − Σ_{b>a} τ_ab γ_b, kept in column L
  double2 gam = from(tau, lane_of(la, L));
#pragma unroll
  for (int p = L - 1; p >= 1; --p) {
    const double2 gp = from(gam, lane_of(p, L));
    const double2 t = from(tau, lane_of(la, la < p ? p : L));
    if (la < p) gam = subd(gam, dcmul(t, gp));
  }
  if (lb == L && lane < NE) {
    sc->gam[la] = gam;
    if (la == L - 1) sc->omega = gam;
  }
}

// Gram matrix of r_0 … r_L — (r_i, r_j) for 1 ≤ i ≤ j ≤ L, then (r_i, r_0)
// for 1 ≤ i ≤ L — and, in the last block, the minimal-residual coefficients
// from it.
template <typename R, int L>
__global__ void __launch_bounds__(VB, 2) k_bl_gram(VSet<typename CT<R>::C> r, VSet<typename CT<R>::C> u,
                                                   typename CT<R>::C *x, long long n, RedBuf red, KScalars *sc) {
  constexpr bool KEEP = sizeof(R) == 8;  // complex128: the replayed vectors are stored
  using C = typename CT<R>::C;
  constexpr int NV = L * (L + 1) / 2 + L;
  if (sc->done) return;
  C hist[Hist<L>::N];
  scalars<R>([&](int i) { return Hist<L>::at(sc, i); }, hist);
  R ar[NV], ai[NV];
#pragma unroll
  for (int q = 0; q < NV; ++q) ar[q] = ai[q] = R(0);
  // adds the products of one element (complex128), or of a pair of elements
  // (complex64, a zero one for an odd tail): a pair's products are summed
  // first, so that the plain FP32 chains have one term per pair
  auto add = [&](int q, const C &a, const C &b, const C &a2, const C &b2, bool real) {
    if constexpr (sizeof(R) == 8) {
      ar[q] = fma(a.y, b.y, fma(a.x, b.x, ar[q]));
      if (!real) ai[q] = fma(-a.y, b.x, fma(a.x, b.y, ai[q]));
    } else {
      const C d = cadd(cdotc(a, b), cdotc(a2, b2));
      ar[q] += d.x;
      ai[q] += d.y;
    }
  };
  auto two = [&](const C (&v)[L + 1], const C (&w)[L + 1]) {
    int q = 0;
#pragma unroll
    for (int j = 1; j <= L; ++j)
#pragma unroll
      for (int i = 1; i <= j; ++i, ++q) add(q, v[i], v[j], w[i], w[j], i == j);  // (r_i, r_i) is real
#pragma unroll
    for (int i = 1; i <= L; ++i, ++q) add(q, v[i], v[0], w[i], w[0], false);
  };
  visit<R>(
      n,
      [&](long long q) {
        C va[L + 1], vb[L + 1], ua[L], ub[L];
#pragma unroll
        for (int i = 0; i <= L; ++i) {
          const Pair<C> p = ldp(r.v[i], q);
          va[i] = p.a;
          vb[i] = p.b;
        }
#pragma unroll
        for (int i = 1; i < L; ++i) {
          const Pair<C> p = ldp(u.v[i], q);
          ua[i] = p.a;
          ub[i] = p.b;
        }
        C none = czero<C>();
        replay<L, false>(va, ua, none, hist);
        replay<L, false>(vb, ub, none, hist);
        two(va, vb);
      },
      [&](long long e) {
        C v[L + 1], ue[L], xe = czero<C>();
        if (KEEP) xe = x[e];
#pragma unroll
        for (int i = 0; i <= L; ++i) v[i] = r.v[i][e];
#pragma unroll
        for (int i = KEEP ? 0 : 1; i < L; ++i) ue[i] = u.v[i][e];
        replay<L, KEEP>(v, ue, xe, hist);
        if (KEEP) {
          x[e] = xe;
#pragma unroll
          for (int i = 0; i + 1 < L; ++i) {
            r.v[i][e] = v[i];
            u.v[i][e] = ue[i];
          }
        }
        const C nil[L + 1] = {};
        two(v, nil);
      });
  if (KEEP && blockIdx.x == 0 && threadIdx.x == 0) sc->bl_steps = 0;  // x holds this cycle's steps
  if constexpr (sizeof(R) == 4) {
    constexpr int K = pow2_at_least(2 * NV);
    DF v[K];
#pragma unroll
    for (int q = 0; q < K; ++q) v[q] = DF{0.f, 0.f};
#pragma unroll
    for (int q = 0; q < NV; ++q) {
      v[2 * q].hi = ar[q];
      v[2 * q + 1].hi = ai[q];
    }
    __shared__ double tot[2 * NV];
    if (!df_block_sums_last<VB, K, 2 * NV>(v, red, tot)) return;
    if (threadIdx.x < 32) bl_mr<L>(tot, sc);
  } else {
    constexpr int K = pow2_at_least(2 * NV);
    double v[K];
#pragma unroll
    for (int q = 0; q < K; ++q) v[q] = 0.0;
#pragma unroll
    for (int q = 0; q < NV; ++q) {
      v[2 * q] = (double)ar[q];
      v[2 * q + 1] = (double)ai[q];
    }
    __shared__ double tot[2 * NV];
    if (!d_block_sums_last<VB, K, 2 * NV>(v, red, tot)) return;
    if (threadIdx.x < 32) bl_mr<L>(tot, sc);
  }
}

// The replayed steps (complex64; k_bl_gram has stored them in complex128),
// then x += Σ γ_k r_{k−1} ; r_0 −= Σ γ_k r_k ;
// u_0 −= Σ γ_k u_k ; then (r̂, r_0) and ‖r_0‖² → FIN_BL_CYCLE.
template <typename R, int L>
__global__ void __launch_bounds__(VB, sizeof(R) == 4 ? 3 : 2) k_bl_fin(VSet<typename CT<R>::C> r, VSet<typename CT<R>::C> u,
                                                  typename CT<R>::C *x, long long n, RedBuf red, KScalars *sc) {
  using C = typename CT<R>::C;
  if (sc->done) return;
  C cs[L + Hist<L>::N];
  scalars<R>([&](int i) { return i < L ? sc->gam[i] : Hist<L>::at(sc, i - L); }, cs);
  const C *hist = cs + L;
  Acc<R> a0r, a0i, a1;
  visit<R>(
      n,
      [&](long long q) {
        C ra[L + 1], rb[L + 1], ua[L + 1], ub[L + 1];
#pragma unroll
        for (int k = 0; k <= L; ++k) {
          const Pair<C> pr = ldp(r.v[k], q), pu = ldp(u.v[k], q);
          ra[k] = pr.a;
          rb[k] = pr.b;
          ua[k] = pu.a;
          ub[k] = pu.b;
        }
        Pair<C> xv = ldp(x, q);
        const Pair<C> hv{shadow<R>(2 * q), shadow<R>(2 * q + 1)};
        if (sizeof(R) == 4) {
          replay<L, true>(ra, ua, xv.a, hist);
          replay<L, true>(rb, ub, xv.b, hist);
        }
        C r0a = ra[0], r0b = rb[0], u0a = ua[0], u0b = ub[0];
#pragma unroll
        for (int k = 1; k <= L; ++k) {
          xv.a = addsv(xv.a, cs[k - 1], ra[k - 1]);
          xv.b = addsv(xv.b, cs[k - 1], rb[k - 1]);
          r0a = subsv(r0a, cs[k - 1], ra[k]);
          r0b = subsv(r0b, cs[k - 1], rb[k]);
          u0a = subsv(u0a, cs[k - 1], ua[k]);
          u0b = subsv(u0b, cs[k - 1], ub[k]);
        }
        stp(x, q, xv);
        stp(r.v[0], q, Pair<C>{r0a, r0b});
        stp(u.v[0], q, Pair<C>{u0a, u0b});
        const C da = cdotc(hv.a, r0a), db = cdotc(hv.b, r0b);
        a0r.add(da.x + db.x);
        a0i.add(da.y + db.y);
        a1.add((r0a.x * r0a.x + r0a.y * r0a.y) + (r0b.x * r0b.x + r0b.y * r0b.y));
      },
      [&](long long e) {
        C rk[L + 1], uk[L + 1];
#pragma unroll
        for (int k = 0; k <= L; ++k) {
          rk[k] = r.v[k][e];
          uk[k] = u.v[k][e];
        }
        C xe = x[e];
        if (sizeof(R) == 4) replay<L, true>(rk, uk, xe, hist);
        C r0 = rk[0], u0 = uk[0];
#pragma unroll
        for (int k = 1; k <= L; ++k) {
          xe = addsv(xe, cs[k - 1], rk[k - 1]);
          r0 = subsv(r0, cs[k - 1], rk[k]);
          u0 = subsv(u0, cs[k - 1], uk[k]);
        }
        x[e] = xe;
        r.v[0][e] = r0;
        u.v[0][e] = u0;
        const C d = cdotc(shadow<R>(e), r0);
        a0r.add(d.x);
        a0i.add(d.y);
        a1.add(r0.x * r0.x + r0.y * r0.y);
      });
  sum_finalise<VB>(a0r, a0i, a1, red, FIN_BL_CYCLE, sc);
}

// A cycle that broke down after `steps` completed BiCG steps: x += Σ α_j u_0
// over them (replay() cut short), so that the restart keeps their progress.
template <typename R>
__global__ void __launch_bounds__(VB) k_bl_fold(VSet<typename CT<R>::C> r, VSet<typename CT<R>::C> u,
                                                typename CT<R>::C *x, long long n, int steps, const KScalars *sc) {
  using C = typename CT<R>::C;
  for (long long e = blockIdx.x * (long long)VB + threadIdx.x; e < n; e += (long long)gridDim.x * VB) {
    C rv[LMAX], uv[LMAX];
#pragma unroll
    for (int i = 0; i < LMAX; ++i)
      if (i < steps) {
        rv[i] = r.v[i][e];
        uv[i] = u.v[i][e];
      }
    C xe = cadd(x[e], cmul(tocr<R>(sc->alpha_j[0]), uv[0]));
#pragma unroll
    for (int j = 1; j < LMAX; ++j)
      if (j < steps) {
        const C al = tocr<R>(sc->alpha_j[j]), be = tocr<R>(sc->beta_j[j]);
#pragma unroll
        for (int i = 0; i < j; ++i) uv[i] = subsv(rv[i], be, uv[i]);
        xe = addsv(xe, al, uv[0]);
#pragma unroll
        for (int i = 0; i < j; ++i) rv[i] = subsv(rv[i], al, uv[i + 1]);
      }
    x[e] = xe;
  }
}

// (r̂, r_0) with the generated shadow vector: FIN_BL_REDO after a replaced
// residual, FIN_NONE (into dot0) for the first ρ of a (re)started solve
template <typename R>
__global__ void __launch_bounds__(VB) k_bl_redo(const typename CT<R>::C *__restrict__ r0, long long n, RedBuf red,
                                                int fin, KScalars *sc) {
  using C = typename CT<R>::C;
  Acc<R> a0r, a0i;
  for (long long e = blockIdx.x * (long long)VB + threadIdx.x; e < n; e += vstride<R>()) {
    const C d = cdotc(shadow<R>(e), r0[e]);
    a0r.add(d.x);
    a0i.add(d.y);
  }
  sum_finalise<VB>(a0r, a0i, red, fin, sc);
}

}  // namespace

template <typename R>
static VSet<typename CT<R>::C> vset(typename CT<R>::C *const *v, int count) {
  VSet<typename CT<R>::C> s{};
  for (int i = 0; i < count && i <= LMAX; ++i) s.v[i] = v[i];
  return s;
}

// Blocks for one full wave of a grid-stride kernel: SM count × its resident
// blocks per SM (cached per kernel and device), at most `cap`.
static int wave_blocks(const void *kern, int cap) {
  static std::mutex mu;
  static std::unordered_map<const void *, int> cache[16];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 16) {
    cudaGetLastError();
    return std::min(RED_BLOCKS, cap);
  }
  std::lock_guard<std::mutex> lock(mu);
  const auto it = cache[dev].find(kern);
  if (it != cache[dev].end()) return std::min(it->second, cap);
  int sms = 0, per = 0;
  int b = RED_BLOCKS;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess &&
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kern, VB, 0) == cudaSuccess && sms * per > 0)
    b = sms * per;
  else
    cudaGetLastError();
  cache[dev].emplace(kern, b);
  return std::min(b, cap);
}

// Blocks for a reducing kernel over n elements: at most RED_BLOCKS, and at
// least two element pairs per thread down to one block per SM — below that
// the block and grid sums cost more than the elements (a warp's share of the
// Gram matrix's sums is 31 additions; at n = 98304 the FP64 Gram kernel took
// 68 µs on two blocks per SM with butterfly sums).
static int red_cap(long long n) {
  const long long b = (n / 2 + 2 * VB - 1) / (2 * VB);
  return (int)std::min<long long>(RED_BLOCKS, std::max<long long>(b, 152));
}

// Launch a grid-stride vector kernel on one full wave.
template <typename... P, typename... A>
static void launch_wave(fdfd_handle *h, void (*kern)(P...), int cap, A... args) {
  kern<<<wave_blocks(reinterpret_cast<const void *>(kern), cap), VB, 0, h->stream>>>(args...);
  h->launches++;
}

template <typename R, int L>
static int bl_cycle_t(fdfd_handle *h, typename CT<R>::C *x, typename CT<R>::C *const *r, typename CT<R>::C *const *u,
                      long long n, KScalars *sc, bool tr) {
  const VSet<typename CT<R>::C> rs = vset<R>(r, L + 1), us = vset<R>(u, L + 1);
  constexpr int NOCAP = 1 << 30;
  int rc;
  for (int j = 0; j < L; ++j) {
    launch_wave(h, k_bl_step<R>, NOCAP, (const typename CT<R>::C *)r[j], (const typename CT<R>::C *)u[j], u[j], n, 1, j, sc);
    if ((rc = cuda_check(h, cudaGetLastError(), "k_bl_step"))) return rc;
    if ((rc = launch_apply_fin<R>(h, u[j], u[j + 1], EPI_DOT_SHD, nullptr, FIN_ALPHA, sc, tr))) return rc;
    launch_wave(h, k_bl_step<R>, NOCAP, (const typename CT<R>::C *)r[j], (const typename CT<R>::C *)u[j + 1], r[j], n, 0, j, sc);
    if ((rc = cuda_check(h, cudaGetLastError(), "k_bl_step"))) return rc;
    if (j + 1 < L) rc = launch_apply_fin<R>(h, r[j], r[j + 1], EPI_DOT_SHD, nullptr, FIN_BL_RHO, sc, tr);
    else rc = launch_apply_fin<R>(h, r[j], r[j + 1], EPI_STORE, nullptr, FIN_NONE, sc, tr);
    if (rc) return rc;
  }
  // the reducing kernels keep ≤ RED_BLOCKS blocks: 8·RED_BLOCKS partial
  // slots hold the Gram matrix's L(L+1)/2 + L ≤ 14 values per block
  if ((rc = ensure_red(h, 8 * RED_BLOCKS))) return rc;
  launch_wave(h, k_bl_gram<R, L>, red_cap(n), rs, us, x, n, h->red, sc);
  if ((rc = cuda_check(h, cudaGetLastError(), "k_bl_gram"))) return rc;
  launch_wave(h, k_bl_fin<R, L>, red_cap(n), rs, us, x, n, h->red, sc);
  return cuda_check(h, cudaGetLastError(), "k_bl_fin");
}

// One BiCGStab(ℓ) cycle (2ℓ operator applications).
template <typename R>
int bl_cycle(fdfd_handle *h, typename CT<R>::C *x, typename CT<R>::C *const *r, typename CT<R>::C *const *u,
             long long n, int ell, KScalars *sc, bool tr) {
  switch (ell) {
    case 1: return bl_cycle_t<R, 1>(h, x, r, u, n, sc, tr);
    case 2: return bl_cycle_t<R, 2>(h, x, r, u, n, sc, tr);
    case 3: return bl_cycle_t<R, 3>(h, x, r, u, n, sc, tr);
    case 4: return bl_cycle_t<R, 4>(h, x, r, u, n, sc, tr);
  }
  return set_error(h, FDFD_ERR_ARG, "BiCGStab(l) needs 1 <= l <= 4");
}

// Fold the completed steps of a broken-down cycle into x (see k_bl_fold).
template <typename R>
int bl_fold(fdfd_handle *h, typename CT<R>::C *x, typename CT<R>::C *const *r, typename CT<R>::C *const *u, long long n,
            int ell, int steps, KScalars *sc) {
  if (steps < 1) return FDFD_OK;
  steps = std::min(steps, ell);
  k_bl_fold<R><<<RED_BLOCKS, VB, 0, h->stream>>>(vset<R>(r, ell + 1), vset<R>(u, ell + 1), x, n, steps, sc);
  h->launches++;
  return cuda_check(h, cudaGetLastError(), "k_bl_fold");
}

template <typename R>
int bl_redo(fdfd_handle *h, const typename CT<R>::C *r0, long long n, int fin, KScalars *sc) {
  int rc = ensure_red(h, RED_BLOCKS);
  if (rc) return rc;
  k_bl_redo<R><<<RED_BLOCKS, VB, 0, h->stream>>>(r0, n, h->red, fin, sc);
  h->launches++;
  return cuda_check(h, cudaGetLastError(), "k_bl_redo");
}

template int bl_cycle<float>(fdfd_handle *, float2 *, float2 *const *, float2 *const *, long long, int, KScalars *,
                             bool);
template int bl_cycle<double>(fdfd_handle *, double2 *, double2 *const *, double2 *const *, long long, int,
                              KScalars *, bool);
template int bl_fold<float>(fdfd_handle *, float2 *, float2 *const *, float2 *const *, long long, int, int, KScalars *);
template int bl_fold<double>(fdfd_handle *, double2 *, double2 *const *, double2 *const *, long long, int, int,
                             KScalars *);
template int bl_redo<float>(fdfd_handle *, const float2 *, long long, int, KScalars *);
template int bl_redo<double>(fdfd_handle *, const double2 *, long long, int, KScalars *);

}  // namespace fdfd
