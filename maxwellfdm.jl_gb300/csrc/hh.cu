// The H-field formulation (ft = HH in create_A / create_b,
// src/model/model.jl:238-240, 266-268):
//     y = A_H h,   A_H = Cₑ·(Pε \ Cₘ) − ω²·Pμ     (Pμ = I here)
// applied matrix-free on the same Yee grid and boundaries as the E operator:
// E' = ε⁻¹ ⊙ (Cₘ h) by backward differences of H (Bloch axes wrap with the
// phase; what a symmetry wall's ghost H(−1) would enter is pinned), then the
// forward differences of Cₑ back onto the H samples, with E' = 0 on the
// pinned tangential samples of the low walls and on the PEC ghost plane N.
// Like the reference (whose Pε \ Cₘ needs a diagonal Pε), this path takes a
// diagonal ε only.
//
// Kernel: the mirror image of the second E operator kernel (stencil2.cuh).  A
// CTA owns a 32 × TYT (x, y) tile, warp w rows RW·w …, lane = x, and marches
// along z over a ring of H planes filled by cp.async (any Nx, periodic
// axes).  Each thread keeps its cells' H and E' of two planes in registers:
// E'(q) reads only the i−1 and (first row of a warp) j−1 neighbours of H from
// shared memory, y(q−1) the j+1 and i+1 neighbours of E'(q−1) by registers,
// shuffles and — across warps — an exchange buffer double-buffered by plane
// parity.  Two warps compute the E' of tile row TYT and column 32 that no
// thread owns.  One barrier per plane.  The reciprocal of ε is recomputed
// only on planes where ε changes for some lane of the warp.
// 96³ complex64 (in a stream of overlapping launches): 69.6 → 17 µs; the
// earlier kernel loaded each plane synchronously between two barriers with
// 64-bit index arithmetic per element.
#include <cuda_runtime.h>

#include <algorithm>

#include "cp_ring.cuh"
#include "krylov_fin.cuh"
#include "operator_common.cuh"
#include "pair_math.cuh"

namespace fdfd {

namespace {

template <typename R, int RW>
struct HG {
  using C = typename CT<R>::C;
  static constexpr int NW = 8, NT = NW * 32, NS = 4;
  static constexpr int TYT = NW * RW;
  static constexpr int XOFF = sizeof(R) == 4 ? 2 : 1;
  static constexpr int XW = sizeof(R) == 4 ? TX + 4 : TX + 2;
  static constexpr int BY = TYT + 2;
  static constexpr int SLOT = (XW * BY * 3 * (int)sizeof(C) + 127) / 128 * 128;
  // exchange, per plane parity: E'_x, E'_z of each warp's first row ([w]) and
  // of tile row TYT ([NW]); E'_y, E'_z of column i0+32 per tile row
  struct Exch {
    C ex[NW + 1][TX], ez[NW + 1][TX];
    C eyh[TYT], ezh[TYT];
  };
  static constexpr int EXCH_OFF = NS * SLOT;
  static constexpr int XT_OFF = EXCH_OFF + 2 * (int)sizeof(Exch);
  static constexpr int YT_OFF = XT_OFF + 2 * (TX + 1) * (int)sizeof(C);   // cm, ce of columns 0 … TX
  static constexpr int ZT_OFF = YT_OFF + 2 * (TYT + 1) * (int)sizeof(C);  // cm, ce of rows 0 … TYT
  static constexpr int ZN = KCMAX + 1;                                    // planes k0 … k1
  static constexpr int SMEM = ZT_OFF + 2 * ZN * (int)sizeof(C);
  static_assert(SMEM <= 113 * 1024, "two CTAs per SM");
};

}  // namespace

// W2R (complex128): ω² is real.  A branch on it inside the plane loop
// becomes predicated FP64 instructions, which take the pipe all the same.
template <typename R, int EPI, int RW, bool W2R>
__global__ void __launch_bounds__(HG<R, RW>::NT, 2)
    k_apply_hh(OpArgs<R> a, Extra<R> ex, const typename CT<R>::C *__restrict__ x, typename CT<R>::C *__restrict__ y,
               const typename CT<R>::C *__restrict__ aux0, RedBuf red, int fin, KScalars *sc) {
  using G = HG<R, RW>;
  using C = typename CT<R>::C;
  using X = typename G::Exch;
  constexpr int NW = G::NW, NS = G::NS, TYT = G::TYT;
  extern __shared__ __align__(128) unsigned char sm[];
  X *xch = reinterpret_cast<X *>(sm + G::EXCH_OFF);
  C *xt = reinterpret_cast<C *>(sm + G::XT_OFF);
  C *yt = reinterpret_cast<C *>(sm + G::YT_OFF);
  C *zt = reinterpret_cast<C *>(sm + G::ZT_OFF);
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int i0 = blockIdx.x * TX, j0 = blockIdx.y * TYT;
  const int k0 = blockIdx.z * ex.kchunk, k1 = min(k0 + ex.kchunk, a.N[2]);
  const bool bx = a.bloch[0], by = a.bloch[1], bz = a.bloch[2];
  const int gi = i0 + lane, jw = RW * w;
  if (sc != nullptr && sc->done) return;

  // planes k0−1 … k0+2 on their way, one group each; plane q in slot (q − k0 + 1) mod NS
  CpRing<R, NW, G::BY, G::XW, G::XOFF> ring;
  ring.init(a, ex, x, i0, j0, w, lane);
  for (int p = 0; p < NS; ++p) {
    if (k0 - 1 + p <= k1) ring.copy(a, sm + p * G::SLOT, k0 - 1 + p);
    cp_async_commit();
  }
  if (tid >= 64 && tid < 64 + TX + 1) {
    const int t = tid - 64, c = cidx(a, 0, i0 + t);
    xt[t] = a.cm[0][c];
    xt[TX + 1 + t] = a.ce[0][c];
  }
  if (tid >= 128 && tid < 128 + TYT + 1) {
    const int t = tid - 128, c = cidx(a, 1, j0 + t);
    yt[t] = a.cm[1][c];
    yt[TYT + 1 + t] = a.ce[1][c];
  }
  if (tid >= 160 && tid - 160 <= k1 - k0) {
    const int t = tid - 160, c = cidx(a, 2, k0 + t);
    zt[t] = a.cm[2][c];
    zt[G::ZN + t] = a.ce[2][c];
  }
  auto hv = [&](int s, int c, int jj, int ii) -> C {
    return reinterpret_cast<const C *>(sm + s * G::SLOT)[((jj + 1) * G::XW + ii + G::XOFF) * 3 + c];
  };
  // warp-uniform: every coefficient this warp's cells use is real
  const bool rxy = i0 >= a.rlo[0] && i0 + TX <= a.rhi[0] && j0 + jw >= a.rlo[1] && j0 + jw + RW <= a.rhi[1];
  // E' samples: pinned on the low symmetry walls, 0 past the high ones
  const bool pin_i = !bx && gi == 0, out_i = !bx && gi >= a.N[0];
  bool pin_j[RW], out_j[RW], act[RW];
  long long cell[RW];      // output cell at plane k0
  long long ecell[RW];     // ε index of the E' sample in plane 0 (wrapped on periodic axes)
  const long long plane = (long long)a.N[0] * a.N[1];
  const int ei = gi >= a.N[0] ? (gi == a.N[0] && bx ? 0 : a.N[0] - 1) : gi;
#pragma unroll
  for (int r = 0; r < RW; ++r) {
    const int gj = j0 + jw + r;
    pin_j[r] = !by && gj == 0;
    out_j[r] = !by && gj >= a.N[1];
    act[r] = gi < a.N[0] && gj < a.N[1];
    cell[r] = gi + (long long)a.N[0] * gj + plane * k0;
    const int ej = gj >= a.N[1] ? (gj == a.N[1] && by ? 0 : a.N[1] - 1) : gj;
    ecell[r] = ei + (long long)a.N[0] * ej;
  }
  const C zero = czero<C>();
  // ε of plane q at the warp's samples; inv = 1/ε, kept while ε stays the same
  R eps[RW][3], inv[RW][3], epre[RW][3];
  auto load_eps = [&](R (&e)[RW][3], int q) {
    const int qz = q < a.N[2] ? q : bz ? q - a.N[2] : a.N[2] - 1;
#pragma unroll
    for (int r = 0; r < RW; ++r)
#pragma unroll
      for (int c = 0; c < 3; ++c) e[r][c] = a.eps[c * a.ncell + ecell[r] + plane * qz];
  };
  load_eps(epre, k0);
#pragma unroll
  for (int r = 0; r < RW; ++r)
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      eps[r][c] = epre[r][c];
      inv[r][c] = R(1) / epre[r][c];
    }

  cp_async_wait<2>();  // planes k0−1, k0
  if (ring.phased())
    for (int p = 0; p < 2; ++p) ring.phase(a, ex, sm + p * G::SLOT, k0 - 1 + p);
  __syncthreads();
  C hp[RW][3];             // H(q−1) at the thread's cells
  C eo[RW][3];             // E'(q−1)
#pragma unroll
  for (int r = 0; r < RW; ++r)
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      hp[r][c] = hv(0, c, jw + r, lane);
      eo[r][c] = zero;
    }
  const C cmx = xt[lane], cex = xt[TX + 1 + lane];
  RowAcc<R, RW> a0r, a0i, a1r;

  int sm1 = 0, s0 = 1;  // slots of planes q−1 and q
  for (int q = k0; q <= k1; ++q) {
    const int t = q - k0;
    X &xq = xch[q & 1], &xk = xch[(q - 1) & 1];
    const C cez = zt[G::ZN + t];
    const bool zpin = !bz && q == 0, zout = !bz && q >= a.N[2];
    const bool rq = rxy && q >= a.rlo[2] && q <= a.rhi[2];
    // 1/ε of this plane, then the next plane's ε on its way
    {
      bool same = true;
#pragma unroll
      for (int r = 0; r < RW; ++r)
#pragma unroll
        for (int c = 0; c < 3; ++c) same = same && epre[r][c] == eps[r][c];
      if (!__all_sync(0xffffffffu, same)) {
#pragma unroll
        for (int r = 0; r < RW; ++r)
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            eps[r][c] = epre[r][c];
            inv[r][c] = R(1) / epre[r][c];
          }
      }
      if (q < k1) load_eps(epre, q + 1);
    }
    C aux[RW][3];
    if ((EPI == EPI_RESID || EPI == EPI_DOT_AUX) && q > k0) {
#pragma unroll
      for (int r = 0; r < RW; ++r)
#pragma unroll
        for (int c = 0; c < 3; ++c)
          if (act[r]) aux[r][c] = aux0[3 * cell[r] + c];
    }
    // ---- E'(q) at the thread's cells
    C hq[RW][3], en[RW][3];
#pragma unroll
    for (int r = 0; r < RW; ++r)
#pragma unroll
      for (int c = 0; c < 3; ++c) hq[r][c] = hv(s0, c, jw + r, lane);
    auto curl_h = [&](auto rc_tag) {
      constexpr bool RC = decltype(rc_tag)::value;
#pragma unroll
      for (int r = 0; r < RW; ++r) {
        const int jj = jw + r;
        const C cey = yt[TYT + 1 + jj];
        const C hyi = hv(s0, 1, jj, lane - 1), hzi = hv(s0, 2, jj, lane - 1);
        const C hxj = r > 0 ? hq[r - 1][0] : hv(s0, 0, jj - 1, lane);
        const C hzj = r > 0 ? hq[r - 1][2] : hv(s0, 2, jj - 1, lane);
        en[r][0] = pdiff<RC>(cey, psub(hq[r][2], hzj), cez, psub(hq[r][1], hp[r][1]));
        en[r][1] = pdiff<RC>(cez, psub(hq[r][0], hp[r][0]), cex, psub(hq[r][2], hzi));
        en[r][2] = pdiff<RC>(cex, psub(hq[r][1], hyi), cey, psub(hq[r][0], hxj));
      }
    };
    if (rq) curl_h(std::true_type{});
    else curl_h(std::false_type{});
#pragma unroll
    for (int r = 0; r < RW; ++r) {
      const bool o = out_i || out_j[r] || zout;
      en[r][0] = zif(o || pin_j[r] || zpin, cscale(en[r][0], inv[r][0]));
      en[r][1] = zif(o || pin_i || zpin, cscale(en[r][1], inv[r][1]));
      en[r][2] = zif(o || pin_i || pin_j[r], cscale(en[r][2], inv[r][2]));
    }
    // ---- y(q−1) from E'(q−1) and E'(q)
    if (q > k0) {
      const C cmz = zt[t - 1];
      const bool rk = rxy && q - 1 >= a.rlo[2] && q - 1 <= a.rhi[2];
      C yv[RW][3];
      auto curl_e = [&](auto rc_tag) {
        constexpr bool RC = decltype(rc_tag)::value;
#pragma unroll
        for (int r = 0; r < RW; ++r) {
          const int jj = jw + r;
          const C cmy = yt[jj];
          C eyi = shfl_down1(eo[r][1]), ezi = shfl_down1(eo[r][2]);
          if (lane == TX - 1) {
            eyi = xk.eyh[jj];
            ezi = xk.ezh[jj];
          }
          C exj, ezj;
          if (r + 1 < RW) {
            exj = eo[r + 1][0];
            ezj = eo[r + 1][2];
          } else {
            exj = xk.ex[w + 1][lane];
            ezj = xk.ez[w + 1][lane];
          }
          yv[r][0] = pdiff<RC>(cmy, psub(ezj, eo[r][2]), cmz, psub(en[r][1], eo[r][1]));
          yv[r][1] = pdiff<RC>(cmz, psub(en[r][0], eo[r][0]), cmx, psub(ezi, eo[r][2]));
          yv[r][2] = pdiff<RC>(cmx, psub(eyi, eo[r][1]), cmy, psub(exj, eo[r][0]));
        }
      };
      if (rk) curl_e(std::true_type{});
      else curl_e(std::false_type{});
#pragma unroll
      for (int r = 0; r < RW; ++r) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          if (W2R || (sizeof(R) == 4 && a.w2.y == R(0))) yv[r][c] = pfma(hp[r][c], -a.w2.x, yv[r][c]);
          else yv[r][c] = csub(yv[r][c], cmul(a.w2, hp[r][c]));
        }
        if (!act[r]) continue;
        C *v = yv[r];
        if (EPI == EPI_RESID) {
#pragma unroll
          for (int c = 0; c < 3; ++c) v[c] = csub(aux[r][c], v[c]);
          a0r.add(r, v[0].x * v[0].x + v[0].y * v[0].y + v[1].x * v[1].x + v[1].y * v[1].y + v[2].x * v[2].x +
                  v[2].y * v[2].y);
        } else if (EPI == EPI_DOT_AUX || EPI == EPI_DOT_TS || EPI == EPI_DOT_SHD) {
          C d[3];
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            if (EPI == EPI_DOT_AUX) d[c] = cdotc(aux[r][c], v[c]);
            else if (EPI == EPI_DOT_TS) d[c] = cdotc(v[c], hp[r][c]);
            else d[c] = cdotc(shadow<R>(3 * cell[r] + c), v[c]);
          }
          a0r.add(r, d[0].x + d[1].x + d[2].x);
          a0i.add(r, d[0].y + d[1].y + d[2].y);
          if (EPI == EPI_DOT_TS)
            a1r.add(r, v[0].x * v[0].x + v[0].y * v[0].y + v[1].x * v[1].x + v[1].y * v[1].y + v[2].x * v[2].x +
                    v[2].y * v[2].y);
        }
        C *yo = y + 3 * cell[r];
        yo[0] = v[0];
        yo[1] = v[1];
        yo[2] = v[2];
      }
      a0r.end_plane();
      a0i.end_plane();
      a1r.end_plane();
#pragma unroll
      for (int r = 0; r < RW; ++r) cell[r] += plane;
    }
    // ---- publish E'(q) for the neighbours' y(q)
    if (q < k1) {
      xq.ex[w][lane] = en[0][0];
      xq.ez[w][lane] = en[0][2];
      const int qz = q < a.N[2] ? q : bz ? q - a.N[2] : a.N[2] - 1;
      if (w == 0) {
        // tile row TYT
        const int jj = TYT, gj = j0 + TYT;
        C e0 = zero, e2 = zero;
        const bool o = (!by && gj >= a.N[1]) || out_i || gj > a.N[1];
        if (!o) {
          const long long ec = ei + (long long)a.N[0] * (gj == a.N[1] ? 0 : gj) + plane * qz;
          const C cey = yt[TYT + 1 + jj];
          if (!zpin)
            e0 = cscale(csub(cmul(cey, csub(hv(s0, 2, jj, lane), hv(s0, 2, jj - 1, lane))),
                             cmul(cez, csub(hv(s0, 1, jj, lane), hv(sm1, 1, jj, lane)))),
                        R(1) / a.eps[ec]);
          if (!pin_i)
            e2 = cscale(csub(cmul(cex, csub(hv(s0, 1, jj, lane), hv(s0, 1, jj, lane - 1))),
                             cmul(cey, csub(hv(s0, 0, jj, lane), hv(s0, 0, jj - 1, lane)))),
                        R(1) / a.eps[2 * a.ncell + ec]);
        }
        xq.ex[NW][lane] = e0;
        xq.ez[NW][lane] = e2;
      } else if (w == 1 && lane < TYT) {
        // column i0+32, tile row `lane`
        const int jj = lane, ii = TX, gj = j0 + jj, gx = i0 + TX;
        C e1 = zero, e2 = zero;
        const bool o = (!bx && gx >= a.N[0]) || (!by && gj >= a.N[1]) || gx > a.N[0] || gj > a.N[1];
        if (!o) {
          const long long ec =
              (gx == a.N[0] ? 0 : gx) + (long long)a.N[0] * (gj == a.N[1] ? 0 : gj) + plane * qz;
          const C cxh = xt[TX + 1 + TX], cey = yt[TYT + 1 + jj];
          if (!zpin)
            e1 = cscale(csub(cmul(cez, csub(hv(s0, 0, jj, ii), hv(sm1, 0, jj, ii))),
                             cmul(cxh, csub(hv(s0, 2, jj, ii), hv(s0, 2, jj, ii - 1)))),
                        R(1) / a.eps[a.ncell + ec]);
          if (by || gj > 0)
            e2 = cscale(csub(cmul(cxh, csub(hv(s0, 1, jj, ii), hv(s0, 1, jj, ii - 1))),
                             cmul(cey, csub(hv(s0, 0, jj, ii), hv(s0, 0, jj - 1, ii)))),
                        R(1) / a.eps[2 * a.ncell + ec]);
        }
        xq.eyh[jj] = e1;
        xq.ezh[jj] = e2;
      }
    }
#pragma unroll
    for (int r = 0; r < RW; ++r)
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        hp[r][c] = hq[r][c];
        eo[r][c] = en[r][c];
      }
    // plane q+1 has landed (q+2 may be in flight); after the barrier every
    // thread sees it, E'(q) is published and plane q−1 is read no more
    const int s1 = s0 + 1 == NS ? 0 : s0 + 1;
    cp_async_wait<1>();
    if (ring.phased() && q + 1 <= k1) ring.phase(a, ex, sm + s1 * G::SLOT, q + 1);
    __syncthreads();
    if (q - 1 + NS <= k1) ring.copy(a, sm + sm1 * G::SLOT, q - 1 + NS);
    cp_async_commit();
    sm1 = s0;
    s0 = s1;
  }
  cp_async_wait<0>();
  if (EPI != EPI_STORE) {
    __syncthreads();
    sum_finalise<G::NT>(a0r.acc, a0i.acc, a1r.acc, red, fin, sc);
  }
}

// z-chunk length: the one whose waves of thread blocks (two per SM), each
// taking its planes plus about two planes' worth of prologue, end first.
// Against chunks of 1 … 64 planes forced one by one, on one stream: in complex64
// the fastest at 48³ (1 plane, 8.4 µs; 2: 10.4), 96³ (6, 20.6 µs; 4: 26.4, 8:
// 24.8), 33×65×129 (5, 20.2; 8: 26.8), 200×16×200, 192×208×64 (6, 58.8; 4:
// 67.0) and 256×256×128 (19, 153; 12: 161); in complex128, where a chunk's
// FP64 time is less even, within 10 % of it (33×65×129: 9 planes 158 µs, 8:
// 144), at 96³ the fastest (12, 208 µs; 6: 213).
static int hh_chunk(const fdfd_handle *h, int tiles) {
  if (h->kc_force > 0) return std::min(h->kc_force, KCMAX);
  int best = 1;
  long long best_cost = 1ll << 62;
  for (int kc = 1; kc <= std::min(KCMAX, h->N[2]); ++kc) {
    const long long blocks = (long long)tiles * ((h->N[2] + kc - 1) / kc);
    const long long cost = (blocks + 303) / 304 * (kc + 2);
    if (cost < best_cost) {
      best_cost = cost;
      best = kc;
    }
  }
  return best;
}

// Thread blocks of a launch, and the larger of the two precisions'.
template <typename R>
static constexpr int hh_rows() { return sizeof(R) == 4 ? 2 : 1; }  // rows per warp
template <typename R>
static dim3 hh_grid(const fdfd_handle *h, int *kchunk) {
  constexpr int TYT = HG<R, hh_rows<R>()>::TYT;
  dim3 grid((h->N[0] + TX - 1) / TX, (h->N[1] + TYT - 1) / TYT, 1);
  *kchunk = hh_chunk(h, (int)(grid.x * grid.y));
  grid.z = (h->N[2] + *kchunk - 1) / *kchunk;
  return grid;
}
int hh_blocks(const fdfd_handle *h) {
  int kc;
  const dim3 a = hh_grid<float>(h, &kc), b = hh_grid<double>(h, &kc);
  return (int)std::max(a.x * a.y * a.z, b.x * b.y * b.z);
}

template <typename R, int EPI, bool W2R>
static int launch_hh_t(fdfd_handle *h, const typename CT<R>::C *x, typename CT<R>::C *y,
                       const typename CT<R>::C *aux0, int fin, KScalars *sc) {
  constexpr int RW = hh_rows<R>();
  using G = HG<R, RW>;
  const auto kern = k_apply_hh<R, EPI, RW, W2R>;
  Extra<R> ex = make_extra<R>(h);
  const dim3 grid = hh_grid<R>(h, &ex.kchunk);
  if (EPI != EPI_STORE) {
    int rc = ensure_red(h, (int)(grid.x * grid.y * grid.z));
    if (rc) return rc;
  }
  static DevFlags attr;
  if (!attr.done(h->dev)) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, G::SMEM);
    if (e != cudaSuccess) return cuda_check(h, e, "cudaFuncSetAttribute(k_apply_hh)");
    e = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
    if (e != cudaSuccess) return cuda_check(h, e, "cudaFuncSetAttribute(carveout)");
    attr.set(h->dev);
  }
  const OpArgs<R> a = op_args<R>(h);
  kern<<<grid, G::NT, G::SMEM, h->stream>>>(a, ex, x, y, aux0, h->red, fin, sc);
  h->launches++;
  return cuda_check(h, cudaGetLastError(), "k_apply_hh launch");
}

template <typename R, int EPI>
static int launch_hh_e(fdfd_handle *h, const typename CT<R>::C *x, typename CT<R>::C *y,
                       const typename CT<R>::C *aux0, int fin, KScalars *sc) {
  if constexpr (sizeof(R) == 8) {
    if (h->w2[1] == 0.0) return launch_hh_t<R, EPI, true>(h, x, y, aux0, fin, sc);
  }
  return launch_hh_t<R, EPI, false>(h, x, y, aux0, fin, sc);
}

template <typename R>
int launch_apply_hh(fdfd_handle *h, const typename CT<R>::C *x, typename CT<R>::C *y, int epi,
                    const typename CT<R>::C *aux0, int fin, KScalars *sc) {
  if (h->has_off) return set_error(h, FDFD_ERR_UNSUPPORTED, "the H formulation needs a diagonal ε (Pε \\ Cₘ)");
  switch (epi) {
    case EPI_STORE: return launch_hh_e<R, EPI_STORE>(h, x, y, aux0, fin, sc);
    case EPI_RESID: return launch_hh_e<R, EPI_RESID>(h, x, y, aux0, fin, sc);
    case EPI_DOT_AUX: return launch_hh_e<R, EPI_DOT_AUX>(h, x, y, aux0, fin, sc);
    case EPI_DOT_TS: return launch_hh_e<R, EPI_DOT_TS>(h, x, y, aux0, fin, sc);
    case EPI_DOT_SHD: return launch_hh_e<R, EPI_DOT_SHD>(h, x, y, aux0, fin, sc);
  }
  return set_error(h, FDFD_ERR_UNSUPPORTED, "this reduction is not available for the H formulation");
}
template int launch_apply_hh<float>(fdfd_handle *, const float2 *, float2 *, int, const float2 *, int, KScalars *);
template int launch_apply_hh<double>(fdfd_handle *, const double2 *, double2 *, int, const double2 *, int, KScalars *);

}  // namespace fdfd
