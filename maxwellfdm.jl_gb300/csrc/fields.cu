// Field post-processing on the device:
//   * h_from_e — H = (i/ω)·Pμ⁻¹·(Cₑ e + jₘ)        (src/model/model.jl:276-279,
//     Pμ = I): the forward-difference curl E→H of the operator, one pass;
//   * e_from_h — E = (−i/ω)·Pε⁻¹·(Cₘ h − jₑ)       (model.jl:281-284) for a
//     diagonal Pε: the backward-difference curl H→E of the operator (ghost
//     H(−1) mirrors H(0) on a symmetry wall, Bloch axes wrap with the phase),
//     divided by ε at each E sample, one pass;
//   * corner means — the create_Mcs interpolation (model.jl:287-306):
//     Mcₑ averages E_w backward along w onto the primal voxel corners with
//     weights s∆lₘ and 1/s∆lₑ (isfwdₑ = boundft .!= EE = false);
//     Mcₘ averages H_w forward along w onto the dual corners with weights
//     s∆lₑ and 1/s∆lₘ (isfwdₘ = boundft .!= HH = true):
//         Ec_w[j] = (s∆lₘ[j−1]·E_w[j−1] + s∆lₘ[j]·E_w[j]) / (2·s∆lₑ[j])
//         Hc_w[j] = (s∆lₑ[j]·H_w[j] + s∆lₑ[j+1]·H_w[j+1]) / (2·s∆lₘ[j]).
//     Ghosts: E_w[−1] mirrors E_w[0] (weight s∆lₘ[0]) on a symmetry wall,
//     H_w[N] = 0 there (normal H on the PEC plane); Bloch axes wrap with the
//     phase e^{∓ikL}.  These are the same two-point means the ε tensor's
//     off-diagonal averaging uses.
#include <cuda_runtime.h>

#include <algorithm>

#include "operator_common.cuh"
#include "pair_math.cuh"

namespace fdfd {

// The two kernels below are bound by the FP64 pipe (a warp's FP64
// instruction holds its scheduler's pipe for 64 cycles however few lanes are
// active: 0.63·10¹² lane FMAs/s on the chip at its top clock, 0.53 to 0.63
// measured), so they are laid out to issue
// few FP64 instructions:
//   * threads run over the flattened cells of an x-y plane, so ragged Nx
//     leaves no idle lanes, and march along z keeping what the next plane
//     needs in registers;
//   * a coefficient that is real for the whole warp (outside that axis' PML)
//     multiplies as a real number, axis by axis.
// 128×128×64, cold: k_h_from_e 192 → 84 µs, each k_corner_mean 271 → 43 µs
// (HBM alone would take 22 and 15 µs; the FP64 pipe is busy 75-78 % of the
// launch).
constexpr int FB = 256;

// acc ± c·d and c·d, with a real c when RC
template <bool NEG, bool RC>
__device__ __forceinline__ void axpy_c(double2 &acc, double2 c, double2 d) {
  const double cx = NEG ? -c.x : c.x;
  acc.x = fma(cx, d.x, acc.x);
  acc.y = fma(cx, d.y, acc.y);
  if (!RC) {
    const double cy = NEG ? -c.y : c.y;
    acc.x = fma(-cy, d.y, acc.x);
    acc.y = fma(cy, d.x, acc.y);
  }
}
template <bool RC>
__device__ __forceinline__ double2 mul_c(double2 c, double2 d) {
  double2 r = mk(c.x * d.x, c.x * d.y);
  if (!RC) {
    r.x = fma(-c.y, d.y, r.x);
    r.y = fma(c.y, d.x, r.y);
  }
  return r;
}

// by_axis (pair_math.cuh) branches once per cell to a body that holds only
// the FP64 instructions it needs; with the tests inside the body they became
// predicated instructions, which take the pipe too: 131 µs against 84 for
// k_h_from_e at 128×128×64.

// The thread's cell p of the plane and its planes [k0, k1), and whether it
// stores (a lane that does not repeats a cell).  zs > 1 (planes of at most 16
// cells): one warp per block, which takes zs z-chunks side by side.  k0 < 0:
// the whole warp lies past the plane.
__device__ __forceinline__ bool plane_thread(int plane, int nz, int kc, int zs, int &p, int &k0, int &k1) {
  bool act;
  if (zs > 1) {
    int sub = threadIdx.x / plane;
    p = threadIdx.x - sub * plane;
    act = sub < zs && (blockIdx.y * zs + sub) * kc < nz;
    k0 = (blockIdx.y * zs + (act ? sub : 0)) * kc;
  } else {
    const int p0 = blockIdx.x * FB + threadIdx.x;
    act = p0 < plane;
    p = act ? p0 : plane - 1;
    k0 = (p0 & ~31) < plane ? (int)blockIdx.y * kc : -1;
  }
  k1 = min(k0 + kc, nz);
  return act;
}

// REALW: ω is real, so i/ω = i·s and s is folded into the curl coefficients.
// BL: some axis is periodic.
template <bool REALW, bool BL>
__global__ void __launch_bounds__(FB) k_h_from_e(OpArgs<double> a, Extra<double> ex, const double2 *__restrict__ e,
                                                 const double2 *__restrict__ jm, double2 *__restrict__ hout,
                                                 double2 iow, int kc, int zs) {
  const int plane = a.N[0] * a.N[1];
  int p, k0, k1;
  const bool act = plane_thread(plane, a.N[2], kc, zs, p, k0, k1);
  if (k0 < 0) return;
  const int i = p % a.N[0], j = p / a.N[0];
  const bool blx = BL && a.bloch[0], bly = BL && a.bloch[1], blz = BL && a.bloch[2];
  const bool pi = !blx && i == 0, pj = !bly && j == 0;
  const double sc = REALW ? iow.y : 1.0;
  const double2 cx = cscale(a.cm[0][i], sc), cy = cscale(a.cm[1][j], sc);
  const bool xr = __all_sync(0xffffffffu, cx.y == 0.0), yr = __all_sync(0xffffffffu, cy.y == 0.0);
  // the +x and +y neighbours: offset in cells, factor (1, or the Bloch phase), present or a PEC ghost
  const bool xin = i + 1 < a.N[0], yin = j + 1 < a.N[1];
  const bool xok = xin || blx, yok = yin || bly;
  const long long dx = xin ? 1 : 1 - a.N[0], dy = yin ? a.N[0] : a.N[0] - plane;
  const double2 zero = czero<double2>();
  const double2 *c0 = e + 3 * ((long long)plane * k0 + p);
  double2 v0 = c0[0], v1 = c0[1], v2 = c0[2];
  for (int k = k0; k < k1; ++k) {
    const long long cell = (long long)plane * k + p;
    const double2 *ec = e + 3 * cell;
    const bool z0 = !blz && k == 0;
    double2 n0 = zero, n1 = zero, n2 = zero;
    if (k + 1 < a.N[2]) {
      const double2 *en = ec + 3ll * plane;
      n0 = en[0];
      n1 = en[1];
      n2 = en[2];
    } else if (blz) {
      n0 = cmul(e[3ll * p], ex.ph[2]);
      n1 = cmul(e[3ll * p + 1], ex.ph[2]);
    }
    double2 eyx = zero, ezx = zero, exy = zero, ezy = zero;
    if (xok) {
      eyx = ec[3 * dx + 1];
      ezx = ec[3 * dx + 2];
      if (BL && !xin) {
        eyx = cmul(eyx, ex.ph[0]);
        ezx = cmul(ezx, ex.ph[0]);
      }
    }
    if (yok) {
      exy = ec[3 * dy];
      ezy = ec[3 * dy + 2];
      if (BL && !yin) {
        exy = cmul(exy, ex.ph[1]);
        ezy = cmul(ezy, ex.ph[1]);
      }
    }
    // tangential E on the low PEC walls is pinned
    const double2 ex0 = (pj || z0) ? zero : v0, ey0 = (pi || z0) ? zero : v1, ez0 = (pi || pj) ? zero : v2;
    if (z0) eyx = exy = zero;
    if (pj) ezx = zero;
    if (pi) ezy = zero;
    const double2 exz = pj ? zero : n0, eyz = pi ? zero : n1;
    const double2 cz = cscale(a.cm[2][k], sc);
    const bool zr = cz.y == 0.0;
    double2 h[3];
    const double2 dzy = csub(ezy, ez0), dyz = csub(eyz, ey0), dxz = csub(exz, ex0), dzx = csub(ezx, ez0),
                  dyx = csub(eyx, ey0), dxy = csub(exy, ex0);
    by_axis(xr, yr, zr, [&](auto tx, auto ty, auto tz) {
      constexpr bool XR = decltype(tx)::value, YR = decltype(ty)::value, ZR = decltype(tz)::value;
      h[0] = mul_c<YR>(cy, dzy);
      axpy_c<true, ZR>(h[0], cz, dyz);
      h[1] = mul_c<ZR>(cz, dxz);
      axpy_c<true, XR>(h[1], cx, dzx);
      h[2] = mul_c<XR>(cx, dyx);
      axpy_c<true, YR>(h[2], cy, dxy);
    });
    if (act) {
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        double2 m = zero;
        if (jm) m = jm[3 * cell + c];
        if (REALW) hout[3 * cell + c] = mk(fma(-sc, m.y, -h[c].y), fma(sc, m.x, h[c].x));
        else hout[3 * cell + c] = cmul(iow, cadd(h[c], m));
      }
    }
    v0 = n0;
    v1 = n1;
    v2 = n2;
  }
}

// H_c at the cell one step back along w from `cell` (t: the cell's index
// along w, stride: the cell stride along w).
__device__ __forceinline__ double2 h_back(const double2 *__restrict__ hin, const OpArgs<double> &a,
                                          const Extra<double> &ex, long long cell, int t, int w, long long stride,
                                          int c) {
  if (t > 0) return hin[3 * (cell - stride) + c];
  if (a.bloch[w]) return cmul(hin[3 * (cell + (long long)(a.N[w] - 1) * stride) + c], ex.phinv[w]);
  return hin[3 * cell + c];  // mirror: H(−1) = H(0)
}

__global__ void k_e_from_h(OpArgs<double> a, Extra<double> ex, const double2 *__restrict__ hin,
                           const double2 *__restrict__ je, double2 *__restrict__ eout, double2 miow) {
  const long long nc = a.ncell;
  const long long sy = a.N[0], sz = (long long)a.N[0] * a.N[1];
  for (long long cell = blockIdx.x * (long long)blockDim.x + threadIdx.x; cell < nc;
       cell += (long long)gridDim.x * blockDim.x) {
    const int i = (int)(cell % a.N[0]), j = (int)((cell / a.N[0]) % a.N[1]), k = (int)(cell / sz);
    const double2 cex = a.ce[0][i], cey = a.ce[1][j], cez = a.ce[2][k];
    const double2 hx = hin[3 * cell], hy = hin[3 * cell + 1], hz = hin[3 * cell + 2];
    const double2 hzj = h_back(hin, a, ex, cell, j, 1, sy, 2), hyk = h_back(hin, a, ex, cell, k, 2, sz, 1);
    const double2 hxk = h_back(hin, a, ex, cell, k, 2, sz, 0), hzi = h_back(hin, a, ex, cell, i, 0, 1, 2);
    const double2 hyi = h_back(hin, a, ex, cell, i, 0, 1, 1), hxj = h_back(hin, a, ex, cell, j, 1, sy, 0);
    double2 e[3];
    e[0] = csub(cmul(cey, csub(hz, hzj)), cmul(cez, csub(hy, hyk)));
    e[1] = csub(cmul(cez, csub(hx, hxk)), cmul(cex, csub(hz, hzi)));
    e[2] = csub(cmul(cex, csub(hy, hyi)), cmul(cey, csub(hx, hxj)));
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      if (je) e[c] = csub(e[c], je[3 * cell + c]);
      eout[3 * cell + c] = cscale(cmul(miow, e[c]), 1.0 / a.eps[c * nc + cell]);
    }
  }
}

// Weights of a two-point mean along each axis, per index t: own[w][t] of the
// value at t and nb[w][t] of its neighbour (t − 1 for E, t + 1 for H).
struct MeanW {
  const double2 *own[3], *nb[3];
};

template <bool HF, bool BL>
__global__ void __launch_bounds__(FB) k_corner_mean(OpArgs<double> a, Extra<double> ex, MeanW wt,
                                                    const double2 *__restrict__ in, double2 *__restrict__ out, int kc, int zs) {
  const int plane = a.N[0] * a.N[1];
  int p, k0, k1;
  const bool act = plane_thread(plane, a.N[2], kc, zs, p, k0, k1);
  if (k0 < 0) return;
  const int i = p % a.N[0], j = p / a.N[0];
  const double2 ox = wt.own[0][i], nx = wt.nb[0][i], oy = wt.own[1][j], ny = wt.nb[1][j];
  const bool xr = __all_sync(0xffffffffu, ox.y == 0.0 && nx.y == 0.0);
  const bool yr = __all_sync(0xffffffffu, oy.y == 0.0 && ny.y == 0.0);
  // neighbour along x and y: in the grid, wrapped with the Bloch phase, or a
  // symmetry wall (E mirrors its own value, H is 0)
  const bool xin = HF ? i + 1 < a.N[0] : i > 0, yin = HF ? j + 1 < a.N[1] : j > 0;
  const long long dx = HF ? (xin ? 1 : 1 - a.N[0]) : (xin ? -1 : a.N[0] - 1);
  const long long dy = HF ? (yin ? a.N[0] : a.N[0] - plane) : (yin ? -a.N[0] : plane - a.N[0]);
  const double2 zero = czero<double2>();
  const double2 phx = HF ? ex.ph[0] : ex.phinv[0], phy = HF ? ex.ph[1] : ex.phinv[1];
  // z: the value at k carried from plane to plane (E: the previous one, H: the next)
  const bool blx = BL && a.bloch[0], bly = BL && a.bloch[1], blz = BL && a.bloch[2];
  double2 carry = zero;
  if (HF) carry = in[3 * ((long long)plane * k0 + p) + 2];
  else if (k0 > 0) carry = in[3 * ((long long)plane * (k0 - 1) + p) + 2];
  for (int k = k0; k < k1; ++k) {
    const long long cell = (long long)plane * k + p;
    const double2 *ic = in + 3 * cell;
    const double2 s0 = ic[0], s1 = ic[1];
    double2 b0 = HF ? zero : s0, b1 = HF ? zero : s1;
    if (xin || blx) b0 = ic[3 * dx];
    if (yin || bly) b1 = ic[3 * dy + 1];
    if (BL) {
      if (!xin && blx) b0 = cmul(b0, phx);
      if (!yin && bly) b1 = cmul(b1, phy);
    }
    double2 s2, b2;
    if (HF) {
      s2 = carry;
      b2 = zero;
      if (k + 1 < a.N[2]) b2 = carry = ic[3ll * plane + 2];
      else if (blz) b2 = cmul(in[3ll * p + 2], ex.ph[2]);
    } else {
      s2 = ic[2];
      b2 = carry;
      if (k == 0) b2 = blz ? cmul(in[3 * ((long long)plane * (a.N[2] - 1) + p) + 2], ex.phinv[2]) : s2;
      carry = s2;
    }
    const double2 oz = wt.own[2][k], nz = wt.nb[2][k];
    const bool zr = oz.y == 0.0 && nz.y == 0.0;
    double2 r0, r1, r2;
    by_axis(xr, yr, zr, [&](auto tx, auto ty, auto tz) {
      constexpr bool XR = decltype(tx)::value, YR = decltype(ty)::value, ZR = decltype(tz)::value;
      r0 = mul_c<XR>(ox, s0);
      r1 = mul_c<YR>(oy, s1);
      r2 = mul_c<ZR>(oz, s2);
      axpy_c<false, XR>(r0, nx, b0);
      axpy_c<false, YR>(r1, ny, b1);
      axpy_c<false, ZR>(r2, nz, b2);
    });
    if (act) {
      out[3 * cell] = r0;
      out[3 * cell + 1] = r1;
      out[3 * cell + 2] = r2;
    }
  }
}

// 2D slices (TE/TM): host vectors carry only the components in `mask`
// (bit c = component c), component-fastest per cell.
__global__ void k_unpack(const double2 *__restrict__ src, double2 *__restrict__ dst, int mask, long long ncell) {
  const int nc = __popc(mask);
  for (long long cell = blockIdx.x * (long long)blockDim.x + threadIdx.x; cell < ncell;
       cell += (long long)gridDim.x * blockDim.x) {
    int q = 0;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      double2 v = make_double2(0.0, 0.0);
      if (mask & (1 << c)) v = src[nc * cell + q++];
      dst[3 * cell + c] = v;
    }
  }
}

__global__ void k_pack(const double2 *__restrict__ src, double2 *__restrict__ dst, int mask, long long ncell) {
  const int nc = __popc(mask);
  for (long long cell = blockIdx.x * (long long)blockDim.x + threadIdx.x; cell < ncell;
       cell += (long long)gridDim.x * blockDim.x) {
    int q = 0;
#pragma unroll
    for (int c = 0; c < 3; ++c)
      if (mask & (1 << c)) dst[nc * cell + q++] = src[3 * cell + c];
  }
}

__global__ void k_pack_real(const double *__restrict__ src, double *__restrict__ dst, int mask, long long ncell) {
  const int nc = __popc(mask);
  for (long long cell = blockIdx.x * (long long)blockDim.x + threadIdx.x; cell < ncell;
       cell += (long long)gridDim.x * blockDim.x) {
    int q = 0;
#pragma unroll
    for (int c = 0; c < 3; ++c)
      if (mask & (1 << c)) dst[nc * cell + q++] = src[3 * cell + c];
  }
}

int field_mask(const fdfd_handle *h, bool hfield) {
  if (h->slice2d == FDFD_SLICE_TE) return hfield ? 4 : 3;
  if (h->slice2d == FDFD_SLICE_TM) return hfield ? 3 : 4;
  return 7;
}

static int ensure_stage(fdfd_handle *h) {
  if (h->stage64) return FDFD_OK;
  if (dev_malloc(&h->stage64, 3 * (size_t)h->ncell * sizeof(double2)) != cudaSuccess) {
    cudaGetLastError();
    h->stage64 = nullptr;
    return set_error(h, FDFD_ERR_NOMEM, "cudaMalloc(2D staging) failed");
  }
  return FDFD_OK;
}

int h2d_field(fdfd_handle *h, const double *src, double2 *dst, int mask) {
  const long long nc = h->ncell;
  if (mask == 7)
    return cuda_check(h, cudaMemcpyAsync(dst, src, 3 * nc * sizeof(double2), cudaMemcpyHostToDevice, h->stream),
                      "H2D field");
  int rc = ensure_stage(h);
  if (rc) return rc;
  const int n = __builtin_popcount(mask);
  if ((rc = cuda_check(h, cudaMemcpyAsync(h->stage64, src, n * nc * sizeof(double2), cudaMemcpyHostToDevice, h->stream),
                       "H2D field")))
    return rc;
  k_unpack<<<152 * 4, 256, 0, h->stream>>>(h->stage64, dst, mask, nc);
  h->launches++;
  return cuda_check(h, cudaGetLastError(), "k_unpack");
}

int d2h_field(fdfd_handle *h, const double2 *src, double *dst, int mask) {
  const long long nc = h->ncell;
  if (mask == 7)
    return cuda_check(h, cudaMemcpyAsync(dst, src, 3 * nc * sizeof(double2), cudaMemcpyDeviceToHost, h->stream),
                      "D2H field");
  int rc = ensure_stage(h);
  if (rc) return rc;
  const int n = __builtin_popcount(mask);
  k_pack<<<152 * 4, 256, 0, h->stream>>>(src, h->stage64, mask, nc);
  h->launches++;
  if ((rc = cuda_check(h, cudaGetLastError(), "k_pack"))) return rc;
  return cuda_check(h, cudaMemcpyAsync(dst, h->stage64, n * nc * sizeof(double2), cudaMemcpyDeviceToHost, h->stream),
                    "D2H field");
}

int d2h_real(fdfd_handle *h, const double *src, double *dst, int mask) {
  const long long nc = h->ncell;
  if (mask == 7)
    return cuda_check(h, cudaMemcpyAsync(dst, src, 3 * nc * sizeof(double), cudaMemcpyDeviceToHost, h->stream),
                      "D2H values");
  int rc = ensure_stage(h);
  if (rc) return rc;
  const int n = __builtin_popcount(mask);
  double *st = reinterpret_cast<double *>(h->stage64);
  k_pack_real<<<152 * 4, 256, 0, h->stream>>>(src, st, mask, nc);
  h->launches++;
  if ((rc = cuda_check(h, cudaGetLastError(), "k_pack_real"))) return rc;
  return cuda_check(h, cudaMemcpyAsync(dst, st, n * nc * sizeof(double), cudaMemcpyDeviceToHost, h->stream),
                    "D2H values");
}

// Launch shape of a z-marching plane kernel: blocks over the flattened plane,
// and chunks of kc planes short enough to give the chip about 64 warps per SM
// (a chunk re-reads one plane, so at most 16 planes gain nothing more).  Where
// a plane has fewer than FB cells a block is its warps, and at most 16
// cells share their warp with the next chunks: 2×2×4096 in blocks of FB
// threads, with 4 of them at work, took 61 µs for h_from_e, now 6.5.
struct PlaneShape {
  dim3 grid;
  int threads, kc, zs;
};
static PlaneShape plane_shape(const fdfd_handle *h) {
  const long long plane = (long long)h->N[0] * h->N[1], warps = (plane + 31) / 32;
  PlaneShape s;
  s.threads = (int)std::min<long long>(FB, 32 * warps);
  s.zs = plane <= 16 ? (int)(32 / plane) : 1;
  s.kc = (int)std::max(1ll, std::min(16ll, warps * h->N[2] / (152 * 64 * s.zs)));
  // blockIdx.y is limited to 65535 chunks
  s.kc = std::max(s.kc, (h->N[2] + 65534) / 65535);
  const int chunks = (h->N[2] + s.kc - 1) / s.kc;
  s.grid = dim3((unsigned)((plane + FB - 1) / FB), (unsigned)((chunks + s.zs - 1) / s.zs), 1);
  return s;
}

int h_from_e_dev_impl(fdfd_handle *h, const double2 *e, const double2 *jm, double2 *hout) {
  const OpArgs<double> a = op_args<double>(h);
  const Extra<double> ex = make_extra<double>(h);
  // i/ω for complex ω
  const double wr = h->omega[0], wi = h->omega[1], d = wr * wr + wi * wi;
  if (!(d > 0.0)) return set_error(h, FDFD_ERR_ARG, "h_from_e needs ω ≠ 0");
  const double2 iow = make_double2(wi / d, wr / d);
  const PlaneShape ps = plane_shape(h);
  const bool bl = h->bloch[0] || h->bloch[1] || h->bloch[2];
  const auto kern = iow.x == 0.0 ? (bl ? k_h_from_e<true, true> : k_h_from_e<true, false>)
                                 : (bl ? k_h_from_e<false, true> : k_h_from_e<false, false>);
  kern<<<ps.grid, ps.threads, 0, h->stream>>>(a, ex, e, jm, hout, iow, ps.kc, ps.zs);
  h->launches++;
  return cuda_check(h, cudaGetLastError(), "k_h_from_e");
}

int e_from_h_dev_impl(fdfd_handle *h, const double2 *hin, const double2 *je, double2 *eout) {
  if (h->has_off)
    return set_error(h, FDFD_ERR_UNSUPPORTED, "e_from_h needs a diagonal ε (Pε \\ …), as in the reference");
  const OpArgs<double> a = op_args<double>(h);
  const Extra<double> ex = make_extra<double>(h);
  // −i/ω for complex ω
  const double wr = h->omega[0], wi = h->omega[1], d = wr * wr + wi * wi;
  if (!(d > 0.0)) return set_error(h, FDFD_ERR_ARG, "e_from_h needs ω ≠ 0");
  const double2 miow = make_double2(-wi / d, -wr / d);
  k_e_from_h<<<152 * 8, 256, 0, h->stream>>>(a, ex, hin, je, eout, miow);
  h->launches++;
  return cuda_check(h, cudaGetLastError(), "k_e_from_h");
}

int corner_mean_dev_impl(fdfd_handle *h, int hfield, const double2 *in, double2 *out) {
  const OpArgs<double> a = op_args<double>(h);
  const Extra<double> ex = make_extra<double>(h);
  // weights: E backward mean wp (own), wm; H forward mean kinds 6 (own) and 7
  MeanW wt;
  for (int w = 0; w < 3; ++w) {
    wt.own[w] = hfield ? h->coef64 + 6 * h->coef_stride + h->coef_off[w] : a.wp[w];
    wt.nb[w] = hfield ? h->coef64 + 7 * h->coef_stride + h->coef_off[w] : a.wm[w];
  }
  const PlaneShape ps = plane_shape(h);
  const bool bl = h->bloch[0] || h->bloch[1] || h->bloch[2];
  const auto kern = hfield ? (bl ? k_corner_mean<true, true> : k_corner_mean<true, false>)
                           : (bl ? k_corner_mean<false, true> : k_corner_mean<false, false>);
  kern<<<ps.grid, ps.threads, 0, h->stream>>>(a, ex, wt, in, out, ps.kc, ps.zs);
  h->launches++;
  return cuda_check(h, cudaGetLastError(), "k_corner_mean");
}

}  // namespace fdfd
