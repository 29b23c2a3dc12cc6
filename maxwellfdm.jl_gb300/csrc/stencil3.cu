// Matrix-free y = A x, A = Cₘ·Cₑ − ω²·Pε (create_A, src/model/model.jl:225-246),
// complex64 on PEC walls: the second operator kernel's march (stencil2.cuh)
// with two helper warps.
//
// In stencil2.cuh every warp forms the off-diagonal (corner) terms of its own
// strip, and every warp waits at the plane's barrier for the slowest.  Corner
// terms exist on interfaces only — 2.4 % of the corners at 320³ with 400
// spheres, but in a third of the tile-planes and a fifth of the strips — so
// most of a strip's 64 lanes of corner arithmetic were zeros, and it cost
// 80 µs of 415 (vacuum: 333 µs, 87 % of the measured copy rate).
//   * The non-zero corners are kept as lists per (32×16 tile, plane), built
//     when ε is set (16 bytes each: position and the three values), with a
//     bit mask of their positions.  Both come to shared memory by cp.async
//     two planes ahead.
//   * Warps 0-7 own two rows each and do curls, the diagonal term and the
//     outputs.  Warps 8 and 9, the helpers, take 32 corners each of the
//     plane's list, a corner per lane, compute the H values that no thread of
//     the tile owns (row j0−1, column i0−1) and refill the ring.  A corner
//     beyond the first 64 goes to a main warp, 32 at a time: with all of them
//     left to the helpers a large sphere's cap (over 200 corners on a
//     tile-plane) held the block up, 446 µs at 320³ and 842 instead of 506
//     with 20 spheres of radius 65.
//   * Each corner's three terms (half of them, as every output averages two
//     corners) are stored in shared memory; where its strip is flagged, an
//     output adds the terms of its two corners per component that the mask
//     has — so nothing is cleared and no two lanes add to one place.  (Adding
//     into per-output sums, six read-modify-write rounds a corner, took
//     490 µs.)  x- and y-directed terms live in two buffers by plane parity,
//     z-directed ones, formed a plane ahead, in three.
// One barrier per plane, as before.  320 threads at 96 registers, two CTAs
// per SM.  (Four helpers, which 80 registers a thread at launch and setmaxnreg
// allow, took 452 µs.)  What bounds it: vacuum the memory (331 µs at 320³,
// 88 % of the copy rate); with corners the plane's barrier, which waits for
// the corner arithmetic.  Against the second kernel's best layout, back to
// back: 320³ with 400 spheres 415 → 392 µs, 96³ with 40 spheres 18.6 → 16.5,
// 128×128×96 in vacuum 54 → 50 and with 60 spheres 73 → 60.
//
// The lists are worth their build (8 µs of a 96³ re-smoothing) only for this
// kernel, so they are made when it is in use or about to be timed by the
// autotuner, which keeps it (layout 5) where it is 3 % faster than the
// second kernel: with odd Nx and corners on most planes it is not (95×89×83
// with 30 spheres: 18.3 µs against 21.2).
#include <cuda.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <type_traits>

#include "cp_ring.cuh"
#include "krylov_fin.cuh"
#include "operator_common.cuh"
#include "pair_math.cuh"
#include "tma_util.cuh"

namespace fdfd {

PFN_cuTensorMapEncodeTiled_v12000 tensor_encode_fn();

namespace {

struct V3 {
  using R = float;
  using C = float2;
  using K = Coef<float>;
  static constexpr int RW = 2, NW = 8, NH = 2, NB = 4, NT = (NW + NH) * 32, NS = 4;
  static constexpr int TYT = NW * RW;
  static constexpr int XOFF = 2, XW = TX + 4, BY = TYT + 2;
  static constexpr int PLANE_BYTES = XW * BY * 3 * (int)sizeof(C);
  static constexpr int SLOT = (PLANE_BYTES + 127) / 128 * 128;
  static constexpr int KC2 = KCMAX + 2;
  // exchange, per plane parity: H_x, H_z of the row below each warp ([0]: tile
  // row j0−1, [w+1]: warp w's last row), H at column i0−1 per tile row
  struct Exch {
    C hx[NW + 1][TX], hz[NW + 1][TX];
    C hyh[TYT], hzh[TYT];
  };
  // half the off-diagonal terms at the corners of a plane: x- and y-directed
  // (two planes' worth), z-directed (three), and the masks of the corners
  // that have any, row by row (on their way or in use: five planes', in a
  // ring of eight)
  struct XTerm { C v[TYT][TX + 1]; };
  struct YTerm { C v[TYT + 1][TX]; };
  struct ZTerm { C v[TYT][TX]; };
  struct Mask { unsigned long long row[TYT + 2]; };
  static constexpr int EXCH_OFF = NS * SLOT;
  static constexpr int XC_OFF = EXCH_OFF + 2 * (int)sizeof(Exch);
  static constexpr int YC_OFF = XC_OFF + 2 * (int)sizeof(XTerm);
  static constexpr int ZC_OFF = YC_OFF + 2 * (int)sizeof(YTerm);
  static constexpr int MK_OFF = ZC_OFF + 3 * (int)sizeof(ZTerm);
  static constexpr int IT_OFF = MK_OFF + 8 * (int)sizeof(Mask);  // list entries on their way, 3 planes'
  static constexpr int XT_OFF = IT_OFF + 3 * NB * 32 * 16;  // cm, wm, wp of columns −1 … TX
  static constexpr int YK_OFF = XT_OFF + 3 * (TX + 2) * (int)sizeof(C);
  static constexpr int ZK_OFF = YK_OFF + 2 * (TYT + 2) * (int)sizeof(K);
  static constexpr int YT_OFF = ZK_OFF + 2 * KC2 * (int)sizeof(K);
  static constexpr int ZT_OFF = YT_OFF + 2 * (TYT + 2) * (int)sizeof(C);
  static constexpr int ZL_OFF = ZT_OFF + 2 * KC2 * (int)sizeof(C);   // corner lists: (start, count) per plane
  static constexpr int ZF_OFF = ZL_OFF + KC2 * (int)sizeof(int2);    // strip flags
  static constexpr int BAR_OFF = (ZF_OFF + KC2 * NW + 15) / 16 * 16;
  static constexpr int SMEM = BAR_OFF + NS * 8;
  static_assert(EXCH_OFF % 128 == 0 && XC_OFF % 8 == 0 && MK_OFF % 16 == 0 && IT_OFF % 16 == 0 && YK_OFF % 16 == 0, "alignment");
  static_assert(2 * (SMEM + 1024) <= 228 * 1024, "two CTAs per SM");
};

}  // namespace

// The block's barrier, reached by the helpers and by the main warps from
// different places: barrier 0 counts the block's threads wherever they
// arrive from (each warp arrives as a whole).
__device__ __forceinline__ void bar_all() {
  asm volatile("barrier.sync.aligned 0, %0;" ::"n"(V3::NT) : "memory");
}
__device__ __forceinline__ bool bar_any(bool p) {
  uint32_t r;
  asm volatile(
      "{\n .reg .pred p, q;\n setp.ne.u32 p, %1, 0;\n barrier.red.or.pred.aligned q, 0, %2, p;\n"
      " selp.u32 %0, 1, 0, q;\n}"
      : "=r"(r)
      : "r"((uint32_t)p), "n"(V3::NT)
      : "memory");
  return r != 0;
}

// CPA: the ring is filled by cp.async (odd Nx), else by TMA.  OFF: ε has
// off-diagonal entries.
template <int EPI, bool CPA, bool OFF>
__device__ __forceinline__ void apply_v3(const CUtensorMap &tmap, const OpArgs<float> &a, const Extra<float> &ex,
                                         const float2 *__restrict__ x, float2 *__restrict__ y,
                                         const float2 *__restrict__ aux0, RedBuf red, int fin, KScalars *sc,
                                         int *errflag) {
  using G = V3;
  using R = float;
  using C = float2;
  using K = G::K;
  constexpr int RW = G::RW, NW = G::NW, NS = G::NS, TYT = G::TYT, KC2 = G::KC2;
  extern __shared__ __align__(128) unsigned char sm[];
  G::Exch *xch = reinterpret_cast<G::Exch *>(sm + G::EXCH_OFF);
  G::XTerm *xc_ = reinterpret_cast<G::XTerm *>(sm + G::XC_OFF);
  G::YTerm *yc_ = reinterpret_cast<G::YTerm *>(sm + G::YC_OFF);
  G::ZTerm *zc_ = reinterpret_cast<G::ZTerm *>(sm + G::ZC_OFF);
  int4 *its = reinterpret_cast<int4 *>(sm + G::IT_OFF);
  G::Mask *mk_ = reinterpret_cast<G::Mask *>(sm + G::MK_OFF);
  C *xt = reinterpret_cast<C *>(sm + G::XT_OFF);
  K *yk = reinterpret_cast<K *>(sm + G::YK_OFF);
  K *zk = reinterpret_cast<K *>(sm + G::ZK_OFF);
  C *yt = reinterpret_cast<C *>(sm + G::YT_OFF);
  C *zt = reinterpret_cast<C *>(sm + G::ZT_OFF);
  int2 *zl = reinterpret_cast<int2 *>(sm + G::ZL_OFF);
  unsigned char *zf = sm + G::ZF_OFF;
  uint64_t *bars = reinterpret_cast<uint64_t *>(sm + G::BAR_OFF);

  // (the shuffle tells the compiler that w is the same for the whole warp)
  const int tid = threadIdx.x, lane = tid & 31, w = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const bool helper = w >= NW;
  int bx = blockIdx.x, by = blockIdx.y, k0 = blockIdx.z * ex.kchunk, k1;
  if (ex.work != nullptr) {
    const int4 wk = ex.work[blockIdx.x];
    bx = wk.x;
    by = wk.y;
    k0 = wk.z;
    k1 = wk.w;
  } else {
    k1 = min(k0 + ex.kchunk, a.N[2]);
  }
  const int tiles_x = (a.N[0] + TX - 1) / TX, strips_y = (a.N[1] + RW - 1) / RW;
  const int i0 = bx * TX, j0 = by * TYT, kfirst = k0 - 1;
  const int gi = i0 + lane, jw = RW * w;
  const int cx = 6 * (i0 - G::XOFF), cy = j0 - 1;

  if (!CPA && (smem_u32(sm) & 127u) != 0u) {  // TMA destinations (the declared alignment gives it)
    if (tid == 0) atomicExch(errflag, 2);
    return;
  }
  if (!CPA && tid == NW * 32) {
    for (int s = 0; s < NS; ++s) mbar_init(smem_u32(&bars[s]), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmap)) : "memory");
  }
  pdl_wait();
  if (sc != nullptr && sc->done) return;  // every thread, before any copy is issued
  auto issue = [&](int q, int s) {  // plane q into slot s (one thread)
    const uint32_t bar = smem_u32(&bars[s]);
    mbar_expect(bar, (uint32_t)G::PLANE_BYTES);
    tma_copy3d(smem_u32(sm + s * G::SLOT), &tmap, cx, cy, q, bar);
  };
  bool ok = true;
  CpRing<R, NW, G::BY, G::XW, G::XOFF> ring;
  if constexpr (CPA) {
    if (!helper) {
      ring.init(a, ex, x, i0, j0, w, lane);
      for (int p = 0; p < NS; ++p) {
        if (kfirst + p <= k1) ring.copy(a, sm + p * G::SLOT, kfirst + p);
        cp_async_commit();
      }
    }
  } else if (tid == NW * 32) {
    for (int p = 0; p < NS; ++p)
      if (kfirst + p <= k1) issue(kfirst + p, p);
    // waits that may not wait at all (for tests): the first one happens here,
    // where the copy cannot have landed by the time the tables are filled
    if (ex.wait_limit <= 0) ok = mbar_wait(smem_u32(&bars[0]), 0, 0);
  }
  if (tid < TX + 2) {
    const int c = cidx(a, 0, i0 + tid - 1);
    xt[tid] = a.cm[0][c];
    xt[(TX + 2) + tid] = a.wm[0][c];
    xt[2 * (TX + 2) + tid] = a.wp[0][c];
  }
  if (tid >= 64 && tid < 64 + TYT + 2) {
    const int t = tid - 64, c = cidx(a, 1, j0 + t - 1);
    yk[t] = coef_of(a.cm[1][c]);
    yk[(TYT + 2) + t] = coef_of(a.ce[1][c]);
    yt[t] = a.wm[1][c];
    yt[(TYT + 2) + t] = a.wp[1][c];
  }
  // z coefficients, corner lists and strip flags over planes kfirst … k1 (k1 − kfirst ≤ KCMAX + 1)
  if (tid >= 128 && tid < 128 + KC2 && kfirst + tid - 128 <= k1) {
    const int t = tid - 128, q = kfirst + t, c = cidx(a, 2, q);
    zk[t] = coef_of(a.cm[2][c]);
    zk[KC2 + t] = coef_of(a.ce[2][c]);
    zt[t] = a.wm[2][c];
    zt[KC2 + t] = a.wp[2][c];
    const bool in = OFF && q >= 0 && q < a.N[2];
    zl[t] = in ? ex.corner_list[(bx + (long long)tiles_x * by) * a.N[2] + q] : make_int2(0, 0);
#pragma unroll
    for (int s = 0; s < NW; ++s) {
      const int tr = j0 / RW + s;
      zf[t * NW + s] = in && tr < strips_y ? ex.oflag_w[(bx + (long long)tiles_x * tr) * a.N[2] + q] : 0;
    }
  }
  const int cxi = cidx(a, 0, gi);
  const K cmx = coef_of(a.cm[0][cxi]), cex = coef_of(a.ce[0][cxi]);
  // where the curl coefficients are real: the warp's own cells
  const int gj0 = j0 + jw;
  const bool rxy = i0 >= a.rlo[0] && min(i0 + TX, a.N[0]) - 1 <= a.rhi[0] && gj0 >= a.rlo[1] &&
                   min(gj0 + RW, a.N[1]) - 1 <= a.rhi[1];
  __syncthreads();

  const int plane = a.N[0] * a.N[1];  // 3·Ncell < 2³¹ (checked at launch)
  const int nc = (int)a.ncell;
  const C zero = czero<C>();
  const bool wall_i = i0 == 0, wall_j = j0 == 0;
  // E component c of the cell di columns and dj rows from the one at byte offset b
  auto ev = [&](int b, int c, int dj, int di) -> C {
    return *reinterpret_cast<const C *>(sm + b + ((dj * G::XW + di) * 3 + c) * (int)sizeof(C));
  };
  auto at = [&](int jj, int ii) { return ((jj + 1) * G::XW + ii + G::XOFF) * 3 * (int)sizeof(C); };  // in a slot

  // slots of planes k−1, k, k+1
  int sm1 = 0, s0 = 1, s1 = 2;
  // x and y averages of E onto the lane's corner (tile column ii, row jj)
  // of the plane in slot s; on: not the z wall plane
  auto ax_ay = [&](int ii, int jj, int s, bool on, C &ax, C &ay) {
    const int b = at(jj, ii) + s * G::SLOT;
    C x0 = ev(b, 0, 0, 0), xm = ev(b, 0, 0, -1), y0 = ev(b, 1, 0, 0), ym = ev(b, 1, -1, 0);
    if (!on || (wall_j && jj == 0)) x0 = xm = zero;
    if (!on || (wall_i && ii == 0)) y0 = ym = zero;
    ax = wsum<false>(xt[(TX + 2) + ii + 1], xm, xt[2 * (TX + 2) + ii + 1], x0);
    ay = wsum<false>(yt[jj + 1], ym, yt[(TYT + 2) + jj + 1], y0);
  };
  // z-directed terms of plane q (slot s); ax, ay are kept for the plane's
  // x- and y-directed terms
  auto z_terms = [&](int4 e, int s, int q, C &ax, C &ay) {
    const int p = max(e.x, 0), ii = p & 63, jj = p >> 6;
    ax_ay(ii, jj, s, q > 0, ax, ay);
    const C v = cscale(cadd(cscale(ax, __int_as_float(e.w)), cscale(ay, __int_as_float(e.z))), 0.5f);
    if (e.x >= 0 && ii < TX && jj < TYT) zc_[q % 3].v[jj][ii] = v;
  };
  auto xy_terms = [&](int4 e, int k, C ax, C ay, C wmz, C wpz) {
    const int p = max(e.x, 0), ii = p & 63, jj = p >> 6;
    C z_0 = ev(at(jj, ii) + s0 * G::SLOT, 2, 0, 0), z_m = ev(at(jj, ii) + sm1 * G::SLOT, 2, 0, 0);
    if ((wall_i && ii == 0) || (wall_j && jj == 0)) z_0 = z_m = zero;
    const C az = wsum<false>(wmz, z_m, wpz, z_0);
    const float exy = __int_as_float(e.y), eyz = __int_as_float(e.z), ezx = __int_as_float(e.w);
    const C vx = cscale(cadd(cscale(ay, exy), cscale(az, ezx)), 0.5f);
    const C vy = cscale(cadd(cscale(ax, exy), cscale(az, eyz)), 0.5f);
    if (e.x >= 0 && jj < TYT) xc_[k & 1].v[jj][ii] = vx;
    if (e.x >= 0 && ii < TX) yc_[k & 1].v[jj][ii] = vy;
  };
  const int hw = w - NW;  // helper warp 0 or 1
  // Plane q's mask (warp 8, a row per lane) and the helper's half of
  // its first NB rounds of entries start their way to shared memory two planes
  // before their first use there.
  const int lp = (bx + tiles_x * by) * a.N[2];
  auto fetch = [&](int q) {
    if (OFF && q <= k1) {
      const int2 l = zl[q - kfirst];
#pragma unroll
      for (int n = 0; n < G::NB; n += G::NH) {
        const int i = (n + hw) * 32 + lane;
        if (i < l.y) cp_async<16>(smem_u32(&its[q % 3 * (G::NB * 32) + i]), ex.corners + l.x + i, true);
      }
      if (hw == 0 && lane <= TYT) {
        if (q < a.N[2])
          cp_async<8>(smem_u32(&mk_[q & 7].row[lane]), ex.corner_mask + (long long)(lp + q) * (TYT + 1) + lane, true);
        else
          mk_[q & 7].row[lane] = 0;
      }
    }
    cp_async_commit();
  };
  // round n's entry for this lane of plane q; position < 0: none.  Rounds from
  // NB on come from global memory.
  auto entry = [&](int q, int n) -> int4 {
    const int i = n * 32 + lane;
    const int2 l = zl[q - kfirst];
    if (i >= l.y) return make_int4(-1, 0, 0, 0);
    return n < G::NB ? its[q % 3 * (G::NB * 32) + i] : ex.corners[l.x + i];
  };
  auto rounds = [&](int t) { return OFF ? (zl[t].y + 31) >> 5 : 0; };
  RowAcc<R, RW> acr, aci, ac1;
  int kstop = k0;
  bool run = true;
  if (helper) {
    fetch(k0);
    fetch(k0 + 1);
    cp_async_wait<0>();
  }
  if constexpr (CPA) {
    if (!helper) cp_async_wait<1>();  // planes k0−1 … k0+1 have landed
    bar_all();
  } else {
    ok = ok && mbar_wait_sleep(smem_u32(&bars[0]), 0, ex.wait_limit, 100000u);
    ok = ok && mbar_wait_sleep(smem_u32(&bars[1]), 0, ex.wait_limit, 100000u);
    run = !bar_any(!ok);
  }
  // the phase parity expected next in each slot
  unsigned phase = 0x3u;  // slots 0 and 1 have completed phase 0

  if (helper) {
    // ------------------------------------------------------------ helper warps
    int4 ecur = make_int4(-1, 0, 0, 0);  // the lane's corner on plane k and the averages there
    C axk = zero, ayk = zero;
    if (run && hw < rounds(1)) {
      ecur = entry(k0, hw);
      z_terms(ecur, 1, k0, axk, ayk);
    }
    const K cmh = coef_of(xt[0]);
    for (int k = k0; run && k < k1; ++k) {
      const int t = k - kfirst;
      const bool z0 = k == 0;
      fetch(k + 2);
      // corners of plane k: x- and y-directed terms
      if (hw < rounds(t)) {
        const C wmz = zt[t], wpz = zt[KC2 + t];
        xy_terms(ecur, k, axk, ayk, wmz, wpz);
      }
      if (!CPA) {
        ok = mbar_wait_sleep(smem_u32(&bars[s1]), (phase >> s1) & 1u, ex.wait_limit, 100000u);
        phase ^= 1u << s1;
      }
      G::Exch &xc = xch[k & 1];
      const K cmz = zk[t];
      if (hw == 0) {
        // H of the tile row j0−1 (its values reach only outputs of pinned DOFs
        // when j0 = 0)
        const int b0 = at(0, lane) + s0 * G::SLOT, b1 = at(0, lane) + s1 * G::SLOT;
        const K cmy = yk[0];
        C mx = ev(b0, 0, -1, 0), my = ev(b0, 1, -1, 0), mz = ev(b0, 2, -1, 0), ex0 = ev(b0, 0, 0, 0),
          ez0 = ev(b0, 2, 0, 0);
        C myk = ev(b1, 1, -1, 0), myi = ev(b0, 1, -1, 1);
        if (wall_i && lane == 0) my = mz = myk = ez0 = zero;
        if (wall_j) ex0 = ez0 = zero;
        if (z0) mx = my = myi = ex0 = zero;
        xc.hx[0][lane] = csum<false, false>(cmy, psub(ez0, mz), cmz, psub(my, myk));
        xc.hz[0][lane] = csum<false, false>(cmx, psub(myi, my), cmy, psub(mx, ex0));
      }
      if (hw == 1) {
        // H of the column i0−1 (reaches only pinned outputs when i0 = 0), one
        // component of one tile row per lane: H_y = cmz (E_x(k+1) − E_x) +
        // cmh (E_z(−1) − E_z(0)), H_z = cmh (E_y(0) − E_y(−1)) + cmy (E_x − E_x(j+1))
        const bool hzl = lane >= TYT;
        const int jj = hzl ? lane - TYT : lane;
        const int b0 = at(jj, -1) + s0 * G::SLOT, b1 = at(jj, -1) + s1 * G::SLOT;
        C p = hzl ? ev(b0, 1, 0, 1) : ev(b1, 0, 0, 0);
        C q = hzl ? ev(b0, 1, 0, 0) : ev(b0, 0, 0, 0);
        C u = hzl ? ev(b0, 0, 0, 0) : ev(b0, 2, 0, 0);
        C v = hzl ? ev(b0, 0, 1, 0) : ev(b0, 2, 0, 1);
        if (wall_i) {  // E_y, E_z of column 0
          if (hzl) p = zero;
          else v = zero;
        }
        if (wall_j && jj == 0) {  // E_x, E_z of row 0
          if (!hzl) p = q = v = zero;
          u = zero;
        }
        if (z0) {  // E_x, E_y of plane 0
          if (hzl) p = u = v = zero;
          q = zero;
        }
        const K ca = hzl ? cmh : cmz, cb = hzl ? yk[jj + 1] : cmh;
        (hzl ? xc.hzh : xc.hyh)[jj] = csum<false, false>(ca, psub(p, q), cb, psub(u, v));
      }
      if (OFF) {
        // corners of plane k+1: z-directed terms
        if (hw < rounds(t + 1)) {
          ecur = entry(k + 1, hw);
          z_terms(ecur, s1, k + 1, axk, ayk);
        }
      }
      cp_async_wait<0>();  // plane k+2's entries and mask: all warps see them after the barrier
      if constexpr (CPA) {
        bar_all();
      } else {
        if (bar_any(!ok)) {
          run = false;
          kstop = k;
          break;
        }
        if (hw == 0 && lane == 0 && k - 1 + NS <= k1) {
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          issue(k - 1 + NS, sm1);
        }
        __syncwarp();
      }
      sm1 = s0;
      s0 = s1;
      s1 = s1 + 1 == NS ? 0 : s1 + 1;
    }
    cp_async_wait<0>();
  } else {
    // ------------------------------------------------------------ main warps
    const int b_own = at(jw, lane);
    const bool pj0 = wall_j && w == 0;  // row 0 of warp 0 lies on the y wall
    const bool pw = wall_i || pj0;
    const bool pin_i = wall_i && lane == 0;  // PEC x wall: E_y, E_z at i = 0 are pinned
    // zero the pinned entries of own-cell values of a plane other than the z wall
    auto pin_own = [&](C (&v)[RW][3]) {
#pragma unroll
      for (int r = 0; r < RW; ++r) {
        const bool pj = pj0 && r == 0;
        v[r][0] = zif(pj, v[r][0]);
        v[r][1] = zif(pin_i, v[r][1]);
        v[r][2] = zif(pin_i || pj, v[r][2]);
      }
    };
    C eo[RW][3];         // E(k), pinned DOFs zeroed
    C hxp[RW], hyp[RW];  // H_x, H_y at k−1
    bool act[RW];
    int off[RW];         // the cell in its plane
#pragma unroll
    for (int r = 0; r < RW; ++r) {
      act[r] = gi < a.N[0] && gj0 + r < a.N[1];
      off[r] = gi + a.N[0] * (gj0 + r);
    }
    {
      const int bm = b_own, b0 = b_own + G::SLOT;
      C em[RW][3], mzi[RW], mzj[RW];
#pragma unroll
      for (int r = 0; r < RW; ++r) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          eo[r][c] = ev(b0, c, r, 0);
          em[r][c] = ev(bm, c, r, 0);
        }
        mzi[r] = ev(bm, 2, r, 1);
        mzj[r] = ev(bm, 2, r + 1, 0);
      }
      if (pw) {
        pin_own(eo);
        pin_own(em);
#pragma unroll
        for (int r = 0; r < RW; ++r) {
          mzi[r] = zif(pj0 && r == 0, mzi[r]);
          mzj[r] = zif(pin_i, mzj[r]);
        }
      }
      if (k0 <= 1) {
#pragma unroll
        for (int r = 0; r < RW; ++r)
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            if (k0 == 0) eo[r][c] = zero;
            else em[r][c] = zero;
          }
      }
      const K cmzm = zk[0];
#pragma unroll
      for (int r = 0; r < RW; ++r) {
        const K cmy = yk[jw + r + 1];
        hxp[r] = csum<false, false>(cmy, psub(mzj[r], em[r][2]), cmzm, psub(em[r][1], eo[r][1]));
        hyp[r] = csum<false, false>(cmzm, psub(eo[r][0], em[r][0]), cmx, psub(em[r][2], mzi[r]));
      }
    }
    // rounds of corners beyond the helpers': one per warp
    if (OFF && run) {
      C ax, ay;
#pragma unroll 1
      for (int n = G::NH + w; n < rounds(1); n += NW) z_terms(entry(k0, n), 1, k0, ax, ay);
    }
    const R *ek = a.eps + (long long)plane * k0;  // the plane's ε and outputs (uniform addresses)
    C *yp = y + 3ll * plane * k0;
    for (int k = k0; run && k < k1; ++k) {
      const int t = k - kfirst;
      G::Exch &xc = xch[k & 1];
      const bool z0 = k == 0;
      // rounds of corners beyond the helpers': here, where few registers are
      // live (the wait for plane k+1 is repeated below, where it costs nothing)
      if (OFF) {
        const int nr = max(rounds(t), rounds(t + 1));
        if (nr > G::NH + w) {
          // (a wait that gave up is reported here: carried to the barrier below,
          // it cost a live register, 384 → 390 µs at 320³)
          if (!CPA && !mbar_wait_sleep(smem_u32(&bars[s1]), (phase >> s1) & 1u, ex.wait_limit, 100000u))
            atomicExch(errflag, 1);
#pragma unroll 1
          for (int n = G::NH + w; n < nr; n += NW) {
            const int4 e = entry(k, n), e1 = entry(k + 1, n);
            C ax, ay;
            ax_ay(max(e.x, 0) & 63, max(e.x, 0) >> 6, s0, !z0, ax, ay);
            xy_terms(e, k, ax, ay, zt[t], zt[KC2 + t]);
            z_terms(e1, s1, k + 1, ax, ay);
          }
        }
      }
      // diagonal ε and the epilogue operand at plane k: their latency overlaps
      // this plane's curls
      R epk[RW][3];
      C aux[RW][3];
#pragma unroll
      for (int r = 0; r < RW; ++r) {
        if (act[r]) {
          epk[r][0] = ek[off[r]];
          epk[r][1] = (ek + nc)[off[r]];
          epk[r][2] = (ek + 2ll * nc)[off[r]];
        }
        if (EPI == EPI_RESID || EPI == EPI_DOT_AUX) {
          if (act[r]) {
            const C *ap = aux0 + 3ll * plane * k + 3 * off[r];
            aux[r][0] = ap[0];
            aux[r][1] = ap[1];
            aux[r][2] = ap[2];
          }
        }
      }
      if (!CPA) {
        ok = mbar_wait_sleep(smem_u32(&bars[s1]), (phase >> s1) & 1u, ex.wait_limit, 100000u);
        phase ^= 1u << s1;
      }
      const int b0 = b_own + s0 * G::SLOT, b1 = b_own + s1 * G::SLOT;
      const K cmz = zk[t], cez = zk[KC2 + t];
      const bool rc = rxy && k >= a.rlo[2] && k <= a.rhi[2];
      const bool offd = OFF && zf[t * NW + w] != 0;
      // E(k+1) at the thread's cells and E(k) at their i+1 and j+1 neighbours
      C en[RW][3], eyi[RW], ezi[RW], exj, ezj;
#pragma unroll
      for (int r = 0; r < RW; ++r) {
#pragma unroll
        for (int c = 0; c < 3; ++c) en[r][c] = ev(b1, c, r, 0);
        eyi[r] = ev(b0, 1, r, 1);
        ezi[r] = ev(b0, 2, r, 1);
      }
      exj = ev(b0, 0, RW, 0);
      ezj = ev(b0, 2, RW, 0);
      if (pw) {
        pin_own(en);
        ezi[0] = zif(pj0, ezi[0]);
        ezj = zif(pin_i, ezj);
      }
      if (z0) {
#pragma unroll
        for (int r = 0; r < RW; ++r) eyi[r] = zero;
        exj = zero;
      }
      // ---- H(k) at the thread's cells
      C hx[RW], hy[RW], hz[RW];
      by_axis<false>(rc, true, true, [&](auto rt, auto, auto) {
        constexpr bool RC = decltype(rt)::value;
#pragma unroll
        for (int r = 0; r < RW; ++r) {
          const K cmy = yk[jw + r + 1];
          const C xj = r + 1 < RW ? eo[r + 1 < RW ? r + 1 : r][0] : exj, zj = r + 1 < RW ? eo[r + 1 < RW ? r + 1 : r][2] : ezj;
          hx[r] = csum<RC, RC>(cmy, psub(zj, eo[r][2]), cmz, psub(eo[r][1], en[r][1]));
          hy[r] = csum<RC, RC>(cmz, psub(en[r][0], eo[r][0]), cmx, psub(eo[r][2], ezi[r]));
          hz[r] = csum<RC, RC>(cmx, psub(eyi[r], eo[r][1]), cmy, psub(eo[r][0], xj));
        }
      });
      // last row's H_x, H_z for the warp above
      xc.hx[w + 1][lane] = hx[RW - 1];
      xc.hz[w + 1][lane] = hz[RW - 1];
      // ---- all H(k) and corner sums written; plane k−1 is read no more
      if constexpr (CPA) {
        cp_async_wait<0>();  // plane k+2 has landed; every thread sees it after the barrier
        bar_all();
        if (k - 1 + NS <= k1) ring.copy(a, sm + sm1 * G::SLOT, k - 1 + NS);
        cp_async_commit();
      } else if (bar_any(!ok)) {
        run = false;
        break;
      }
      // ---- outputs y(k)
      C yv[RW][3];
      {
        const C hzj0 = xc.hz[w][lane], hxj0 = xc.hx[w][lane];
        C hzim[RW], hyim[RW];
#pragma unroll
        for (int r = 0; r < RW; ++r) {
          hzim[r] = shfl_up1(hz[r]);
          hyim[r] = shfl_up1(hy[r]);
          if (lane == 0) {
            hzim[r] = xc.hzh[jw + r];
            hyim[r] = xc.hyh[jw + r];
          }
        }
        by_axis<false>(rc, true, true, [&](auto rt, auto, auto) {
          constexpr bool RC = decltype(rt)::value;
#pragma unroll
          for (int r = 0; r < RW; ++r) {
            const K cey = yk[(TYT + 2) + jw + r + 1];
            const C hzjm = r > 0 ? hz[r > 0 ? r - 1 : 0] : hzj0, hxjm = r > 0 ? hx[r > 0 ? r - 1 : 0] : hxj0;
            yv[r][0] = csum<RC, RC>(cey, psub(hz[r], hzjm), cez, psub(hyp[r], hy[r]));
            yv[r][1] = csum<RC, RC>(cez, psub(hx[r], hxp[r]), cex, psub(hzim[r], hz[r]));
            yv[r][2] = csum<RC, RC>(cex, psub(hy[r], hyim[r]), cey, psub(hxjm, hx[r]));
          }
        });
      }
      // Pε E at the cell: the diagonal with the true E (eo holds 0 at pinned
      // DOFs; the ring slot of plane k still has them) plus the corner terms
      C tv[RW][3], dv[RW][3];
#pragma unroll
      for (int r = 0; r < RW; ++r)
#pragma unroll
        for (int c = 0; c < 3; ++c) tv[r][c] = eo[r][c];
      if (pw || z0) {  // pinned outputs: −ω²ε E alone
#pragma unroll
        for (int r = 0; r < RW; ++r) {
          const bool pj = pj0 && r == 0;
          const bool pn[3] = {pj || z0, pin_i || z0, pin_i || pj};
#pragma unroll
          for (int c = 0; c < 3; ++c)
            if (pn[c]) {
              tv[r][c] = ev(b0, c, r, 0);
              yv[r][c] = zero;
            }
        }
      }
      if (offd) {
        const int zb = k % 3, zb1 = zb == 2 ? 0 : zb + 1;
#pragma unroll
        for (int r = 0; r < RW; ++r) {
          const int jj = jw + r;
          const unsigned long long m0 = mk_[k & 7].row[jj], m1 = mk_[k & 7].row[jj + 1], mz = mk_[(k + 1) & 7].row[jj];
          C o[3] = {zero, zero, zero};
          if ((m0 >> lane) & 1) {
            o[0] = xc_[k & 1].v[jj][lane];
            o[1] = yc_[k & 1].v[jj][lane];
            o[2] = zc_[zb].v[jj][lane];
          }
          if ((m0 >> (lane + 1)) & 1) o[0] = cadd(o[0], xc_[k & 1].v[jj][lane + 1]);
          if ((m1 >> lane) & 1) o[1] = cadd(o[1], yc_[k & 1].v[jj + 1][lane]);
          if ((mz >> lane) & 1) o[2] = cadd(o[2], zc_[zb1].v[jj][lane]);
          if (pw || z0) {
            const bool pj = pj0 && r == 0;
            if (pj || z0) o[0] = zero;
            if (pin_i || z0) o[1] = zero;
            if (pin_i || pj) o[2] = zero;
          }
#pragma unroll
          for (int c = 0; c < 3; ++c) dv[r][c] = pfma(tv[r][c], epk[r][c], o[c]);
        }
      } else {
#pragma unroll
        for (int r = 0; r < RW; ++r)
#pragma unroll
          for (int c = 0; c < 3; ++c) dv[r][c] = cscale(tv[r][c], epk[r][c]);
      }
      if (a.w2.y == R(0)) {
#pragma unroll
        for (int r = 0; r < RW; ++r)
#pragma unroll
          for (int c = 0; c < 3; ++c) yv[r][c] = pfma(dv[r][c], -a.w2.x, yv[r][c]);
      } else {
#pragma unroll
        for (int r = 0; r < RW; ++r)
#pragma unroll
          for (int c = 0; c < 3; ++c) yv[r][c] = csub(yv[r][c], cmul(a.w2, dv[r][c]));
      }
#pragma unroll
      for (int r = 0; r < RW; ++r) {
        if (!act[r]) continue;
        C *v = yv[r];
        if (EPI == EPI_RESID) {
#pragma unroll
          for (int c = 0; c < 3; ++c) v[c] = csub(aux[r][c], v[c]);
          acr.add(r, v[0].x * v[0].x + v[0].y * v[0].y + v[1].x * v[1].x + v[1].y * v[1].y + v[2].x * v[2].x +
                  v[2].y * v[2].y);
        } else if (EPI == EPI_DOT_AUX || EPI == EPI_DOT_TS) {
          // (r̂, y), or (t, s) with the true input s
          const C q0 = EPI == EPI_DOT_AUX ? cdotc(aux[r][0], v[0]) : cdotc(v[0], tv[r][0]);
          const C q1 = EPI == EPI_DOT_AUX ? cdotc(aux[r][1], v[1]) : cdotc(v[1], tv[r][1]);
          const C q2 = EPI == EPI_DOT_AUX ? cdotc(aux[r][2], v[2]) : cdotc(v[2], tv[r][2]);
          acr.add(r, q0.x + q1.x + q2.x);
          aci.add(r, q0.y + q1.y + q2.y);
          if (EPI == EPI_DOT_TS)
            ac1.add(r, v[0].x * v[0].x + v[0].y * v[0].y + v[1].x * v[1].x + v[1].y * v[1].y + v[2].x * v[2].x +
                    v[2].y * v[2].y);
        } else if (EPI == EPI_DOT_SHD) {
          const int ce = 3 * (plane * k + off[r]);
          const C q = pdot3(shadow<R>(ce), v[0], shadow<R>(ce + 1), v[1], shadow<R>(ce + 2), v[2]);
          acr.add(r, q.x);
          aci.add(r, q.y);
        }
        C *yo = yp + 3 * off[r];
        yo[0] = v[0];
        yo[1] = v[1];
        yo[2] = v[2];
      }
      acr.end_plane();
      aci.end_plane();
      ac1.end_plane();
      // ---- advance to plane k+1
#pragma unroll
      for (int r = 0; r < RW; ++r) {
        hxp[r] = hx[r];
        hyp[r] = hy[r];
#pragma unroll
        for (int c = 0; c < 3; ++c) eo[r][c] = en[r][c];
      }
      ek += plane;
      yp += 3ll * plane;
      sm1 = s0;
      s0 = s1;
      s1 = s1 + 1 == NS ? 0 : s1 + 1;
    }
    if (CPA) cp_async_wait<0>();
  }
  if (!CPA && w == NW && !run && lane == 0) {
    // a bounded wait gave up: report it and wait (with the full limit) for
    // the last copy issued into each slot — planes up to min(k1, kstop+NS−2),
    // plane q in slot (q − kfirst) mod NS as phase (q − kfirst) / NS — so no
    // copy lands in this block's shared memory after it exits
    atomicExch(errflag, 1);
    const int qlast = min(k1, kstop + NS - 2);
    for (int q = max(kfirst, qlast - NS + 1); q <= qlast; ++q)
      mbar_wait(smem_u32(&bars[(q - kfirst) % NS]), ((q - kfirst) / NS) & 1);
  }
  __syncthreads();
  if (EPI != EPI_STORE) sum_finalise<G::NT>(acr.acc, aci.acc, ac1.acc, red, fin, sc);
}

template <int EPI, bool OFF>
__global__ void __launch_bounds__(V3::NT, 2)
    k_apply_v3(const __grid_constant__ CUtensorMap tmap, OpArgs<float> a, Extra<float> ex, const float2 *__restrict__ x,
               float2 *__restrict__ y, const float2 *__restrict__ aux0, RedBuf red, int fin, KScalars *sc,
               int *errflag) {
  apply_v3<EPI, false, OFF>(tmap, a, ex, x, y, aux0, red, fin, sc, errflag);
}

template <int EPI, bool OFF>
__global__ void __launch_bounds__(V3::NT, 2)
    k_apply_v3cp(OpArgs<float> a, Extra<float> ex, const float2 *__restrict__ x, float2 *__restrict__ y,
                 const float2 *__restrict__ aux0, RedBuf red, int fin, KScalars *sc) {
  apply_v3<EPI, true, OFF>(CUtensorMap{}, a, ex, x, y, aux0, red, fin, sc, nullptr);
}

// ------------------------------------------------------------ corner lists
// One warp per (tile, plane) whose strips are flagged: the masks of its 17
// corner rows from ballots, a place for its entries from one atomic add, then
// the entries row by row (the order of the lists among each other does not
// matter).  Reading ε once per flagged tile-plane, with no counting pass and
// no atomic per corner, took the rebuild at 96³ from 48 to 8 µs.
__global__ void __launch_bounds__(256)
    k_corner_lists(const float *__restrict__ eoff, const uint8_t *__restrict__ flag, long long ncell, int N0, int N1,
                   int N2, int tiles_x, int tiles_y, int2 *list, int4 *items, unsigned cap, unsigned long long *mask,
                   unsigned *next) {
  constexpr int ROWS = V3::TYT + 1;
  const int lane = threadIdx.x & 31, strips_y = (N1 + V3::RW - 1) / V3::RW;
  const long long n = (long long)tiles_x * tiles_y * N2;
  for (long long tp = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5; tp < n;
       tp += (gridDim.x * (long long)blockDim.x) >> 5) {
    const int col = (int)(tp / N2), k = (int)(tp - (long long)col * N2), by = col / tiles_x, bx = col - by * tiles_x;
    const int tr = by * V3::NW + lane;
    const bool f = lane < V3::NW && tr < strips_y && flag[(bx + (long long)tiles_x * tr) * N2 + k];
    if (!__any_sync(~0u, f)) {
      if (lane < ROWS) mask[tp * ROWS + lane] = 0;
      if (lane == 0) list[tp] = make_int2(0, 0);
      continue;
    }
    const int i0 = bx * TX, j0 = by * V3::TYT;
    const float *e = eoff + (long long)k * N0 * N1;
    // the tile's corners, a row of each component per load, all in flight at once
    float v[ROWS][3], u[3];
    auto load = [&](int jj, int ii, bool in, float (&o)[3]) {
      in = in && i0 + ii < N0 && j0 + jj < N1;
      const float *p = e + (long long)(j0 + jj) * N0 + i0 + ii;
#pragma unroll
      for (int q = 0; q < 3; ++q) o[q] = in ? p[q * ncell] : 0.f;
    };
#pragma unroll
    for (int jj = 0; jj < ROWS; ++jj) load(jj, lane, true, v[jj]);
    load(lane, TX, lane < ROWS, u);
    unsigned row[ROWS];
#pragma unroll
    for (int jj = 0; jj < ROWS; ++jj)
      row[jj] = __ballot_sync(~0u, v[jj][0] != 0.f || v[jj][1] != 0.f || v[jj][2] != 0.f);
    const unsigned last = __ballot_sync(~0u, u[0] != 0.f || u[1] != 0.f || u[2] != 0.f);  // column 32, a row per bit
    int c = __popc(last);
#pragma unroll
    for (int jj = 0; jj < ROWS; ++jj) {
      c += __popc(row[jj]);
      if (lane == jj) mask[tp * ROWS + jj] = row[jj] | (unsigned long long)((last >> jj) & 1) << TX;
    }
    unsigned base = 0;
    if (lane == 0) {
      base = c ? atomicAdd(next, (unsigned)c) : 0u;
      list[tp] = make_int2((int)base, c);
    }
    base = __shfl_sync(~0u, base, 0);
    if (base + c > cap) continue;  // the host runs again with room for all
    auto put = [&](unsigned q, int jj, int ii, const float (&o)[3]) {
      items[q] = make_int4(ii | (jj << 6), __float_as_int(o[0]), __float_as_int(o[1]), __float_as_int(o[2]));
    };
    const unsigned below = (1u << lane) - 1;
#pragma unroll
    for (int jj = 0; jj < ROWS; ++jj) {
      if ((row[jj] >> lane) & 1) put(base + __popc(row[jj] & below), jj, lane, v[jj]);
      base += __popc(row[jj]);
    }
    if ((last >> lane) & 1) put(base + __popc(last & below), lane, TX, u);
  }
}

// Whether the layout in use, or the tuner that is about to run, may take the
// lists (the grid's share of v3_serves).
static bool lists_wanted(const fdfd_handle *h) {
  return !h->bloch[0] && !h->bloch[1] && !h->bloch[2] && (h->op_variant == 5 || h->tuned_off == 0) &&
         3 * h->ncell < (1ll << 31);
}

// next: a word of device memory holding 0, left holding the number of corners
static int launch_corner_lists(fdfd_handle *h, unsigned *next) {
  const int tiles_x = (h->N[0] + TX - 1) / TX, tiles_y = (h->N[1] + V3::TYT - 1) / V3::TYT;
  k_corner_lists<<<152 * 4, 256, 0, h->stream>>>(h->eoff32, h->oflag_rows[V3::RW - 1], h->ncell, h->N[0], h->N[1],
                                                 h->N[2], tiles_x, tiles_y, h->corner_list, h->corners,
                                                 (unsigned)h->corner_cap, h->corner_mask, next);
  return cuda_check(h, cudaGetLastError(), "k_corner_lists");
}

// Launch the rebuild where an earlier one left the memory for it; the caller
// reads the count with what else it reads and hands it to build_corner_lists.
int queue_corner_lists(fdfd_handle *h, unsigned *next, bool *queued) {
  *queued = lists_wanted(h) && h->corner_mask && h->corners;
  return *queued ? launch_corner_lists(h, next) : FDFD_OK;
}

// Rebuild the corner lists from eoff32 and the strip flags on the handle's
// stream (queued: the count where they were rebuilt already).  Where there is
// no memory for them the third kernel is not used.
int build_corner_lists(fdfd_handle *h, const unsigned *queued) {
  const long long nl = (long long)((h->N[0] + TX - 1) / TX) * ((h->N[1] + V3::TYT - 1) / V3::TYT) * h->N[2];
  const bool was_ok = h->corner_ok;
  const int4 *const was = h->corners;
  // captured solver graphs hold the lists' addresses and the kernel chosen
  auto unused = [&]() -> int {
    cudaGetLastError();
    h->corner_ok = false;
    if (was_ok) drop_graphs(h);
    return FDFD_OK;
  };
  if (!h->has_off || !lists_wanted(h)) return unused();
  if (!h->corner_mask) {
    if (!h->corner_list && dev_malloc(&h->corner_list, (nl + 1) * sizeof(int2)) != cudaSuccess) {
      h->corner_list = nullptr;
      return unused();
    }
    if (dev_malloc(&h->corner_mask, nl * (V3::TYT + 1) * sizeof(unsigned long long)) != cudaSuccess) {
      h->corner_mask = nullptr;
      return unused();
    }
  }
  unsigned *next = reinterpret_cast<unsigned *>(h->corner_list + nl);
  unsigned n = queued != nullptr ? *queued : 0;
  for (bool have = queued != nullptr;; have = false) {  // twice at most: the second time with room for all
    if (!have) {
      int rc = cuda_check(h, cudaMemsetAsync(next, 0, sizeof(unsigned), h->stream), "memset corner count");
      if (rc || (rc = launch_corner_lists(h, next))) return rc;
      if ((rc = cuda_check(h, cudaMemcpyAsync(&n, next, sizeof(n), cudaMemcpyDeviceToHost, h->stream), "D2H corner count")))
        return rc;
      if ((rc = cuda_check(h, cudaStreamSynchronize(h->stream), "stream sync"))) return rc;
    }
    if (n <= h->corner_cap) break;
    cudaFree(h->corners);
    h->corners = nullptr;
    h->corner_cap = 0;
    const size_t cap = (size_t)n + n / 8;
    if (dev_malloc(&h->corners, cap * sizeof(int4)) != cudaSuccess) {
      h->corners = nullptr;
      return unused();
    }
    h->corner_cap = cap;
  }
  h->corner_ok = true;
  if (!was_ok || was != h->corners) drop_graphs(h);
  return FDFD_OK;
}

// ------------------------------------------------------------ launch
template <int EPI, bool OFF>
static int launch_v3_t(fdfd_handle *h, const float2 *x, float2 *y, const float2 *aux0, int fin, KScalars *sc, int kc,
                       bool tma) {
  using G = V3;
  Extra<float> ex = make_extra<float>(h);
  ex.kchunk = kc;
  dim3 grid((h->N[0] + TX - 1) / TX, (h->N[1] + G::TYT - 1) / G::TYT, (h->N[2] + kc - 1) / kc);
  if (h->nwork[1] > 0) {  // the balanced schedule (built for this layout's tile rows)
    ex.work = h->work[1];
    grid = dim3((unsigned)h->nwork[1], 1, 1);
  }
  if (EPI != EPI_STORE) {
    int rc = ensure_red(h, (int)(grid.x * grid.y * grid.z));
    if (rc) return rc;
  }
  static DevFlags attr;
  if (!attr.done(h->dev)) {
    const void *ks[2] = {reinterpret_cast<const void *>(k_apply_v3<EPI, OFF>), reinterpret_cast<const void *>(k_apply_v3cp<EPI, OFF>)};
    for (const void *kern : ks) {
      cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, G::SMEM);
      if (e != cudaSuccess) return cuda_check(h, e, "cudaFuncSetAttribute(k_apply_v3)");
      e = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
      if (e != cudaSuccess) return cuda_check(h, e, "cudaFuncSetAttribute(carveout)");
    }
    attr.set(h->dev);
  }
  if (OFF) {
    ex.oflag_w = h->oflag_rows[G::RW - 1];
    ex.corners = h->corners;
    ex.corner_list = h->corner_list;
    ex.corner_mask = h->corner_mask;
  }
  const OpArgs<float> a = op_args<float>(h);
  cudaError_t e;
  if (tma) {
    CUtensorMap map;
    const cuuint64_t dims[3] = {(cuuint64_t)6 * h->N[0], (cuuint64_t)h->N[1], (cuuint64_t)h->N[2]};
    const cuuint64_t strides[2] = {(cuuint64_t)24 * h->N[0], (cuuint64_t)24 * h->N[0] * h->N[1]};
    const cuuint32_t box[3] = {(cuuint32_t)(6 * G::XW), (cuuint32_t)G::BY, 1u};
    const cuuint32_t estr[3] = {1u, 1u, 1u};
    if (tensor_encode_fn()(&map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, const_cast<float2 *>(x), dims, strides, box, estr,
                           CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                           CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return set_error(h, FDFD_ERR_CUDA, "cuTensorMapEncodeTiled (third operator kernel) failed");
    e = launch_k(h, k_apply_v3<EPI, OFF>, grid, dim3(G::NT, 1, 1), (size_t)G::SMEM, map, a, ex, x, y, aux0, h->red, fin, sc,
                 h->dev_err);
  } else {
    e = launch_k(h, k_apply_v3cp<EPI, OFF>, grid, dim3(G::NT, 1, 1), (size_t)G::SMEM, a, ex, x, y, aux0, h->red, fin, sc);
  }
  h->launches++;
  return cuda_check(h, e, "k_apply_v3 launch");
}

// Launch through this kernel when it serves the call (PEC walls; tma: by TMA,
// else by cp.async), FDFD_ERR_UNSUPPORTED otherwise.
template <int EPI>
static int launch_v3_e(fdfd_handle *h, const float2 *x, float2 *y, const float2 *aux0, int fin, KScalars *sc, int kc,
                       bool tma) {
  return h->has_off ? launch_v3_t<EPI, true>(h, x, y, aux0, fin, sc, kc, tma)
                    : launch_v3_t<EPI, false>(h, x, y, aux0, fin, sc, kc, tma);
}

bool v3_serves(const fdfd_handle *h) {
  return !h->bloch[0] && !h->bloch[1] && !h->bloch[2] && (!h->has_off || h->corner_ok);
}

int launch_apply_v3(fdfd_handle *h, const float2 *x, float2 *y, int epi, const float2 *aux0, int fin, KScalars *sc,
                    int kc, bool tma) {
  if (!v3_serves(h)) return FDFD_ERR_UNSUPPORTED;
  switch (epi) {
    case EPI_STORE: return launch_v3_e<EPI_STORE>(h, x, y, aux0, fin, sc, kc, tma);
    case EPI_RESID: return launch_v3_e<EPI_RESID>(h, x, y, aux0, fin, sc, kc, tma);
    case EPI_DOT_AUX: return launch_v3_e<EPI_DOT_AUX>(h, x, y, aux0, fin, sc, kc, tma);
    case EPI_DOT_TS: return launch_v3_e<EPI_DOT_TS>(h, x, y, aux0, fin, sc, kc, tma);
    case EPI_DOT_SHD: return launch_v3_e<EPI_DOT_SHD>(h, x, y, aux0, fin, sc, kc, tma);
  }
  return FDFD_ERR_UNSUPPORTED;
}

}  // namespace fdfd
