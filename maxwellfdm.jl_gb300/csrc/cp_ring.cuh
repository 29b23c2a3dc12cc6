// Filling a shared-memory ring of tile planes by cp.async from every thread
// of a block: for kernels that march along z over a 32-wide (x, y) tile and
// read a one-cell halo, where TMA does not serve — an x pitch that is no
// multiple of 16 bytes, periodic axes (TMA zero-fills beyond the grid).
#pragma once

#include "operator_common.cuh"
#include "tma_util.cuh"

namespace fdfd {

// A slot holds BY rows (tile rows −1 … BY−2) of XW cells (columns −XOFF …),
// three complex components per cell.  Cells outside the grid become 0, those
// beyond a periodic axis the wrapped ones — copied raw and multiplied by
// their Bloch phase once landed.  A complex64 row whose pitch is a multiple
// of 16 bytes goes in 16-byte copies from column i0−2 on, any other row
// element by element from column i0−1 (8 bytes each in complex64: 95×89×83
// took 20.7 µs with the wrap tests in every copy, 18.2 with the lane's
// offsets prepared once).
template <typename R, int NW, int BY, int XW, int XOFF>
struct CpRing {
  using C = typename CT<R>::C;
  static constexpr int NCOPY = 4;
  static constexpr int NEL = 3 * (TX + 2);       // elements of columns −1 … TX
  static constexpr int NVEC = 3 * (TX + 4) / 2;  // 16-byte pairs of columns −2 … TX+1
  const C *x;
  int i0, j0, w, lane, row3;
  bool vec, bx, by, bz;
  bool phx, phy, phz;  // Bloch phases other than 1
  int cof[NCOPY];      // per copy of the lane: its offset in the row, −1 outside the grid

  __device__ __forceinline__ void init(const OpArgs<R> &a, const Extra<R> &ex, const C *x_, int i0_, int j0_, int w_,
                                       int lane_) {
    x = x_;
    i0 = i0_;
    j0 = j0_;
    w = w_;
    lane = lane_;
    row3 = 3 * a.N[0];
    bx = a.bloch[0];
    by = a.bloch[1];
    bz = a.bloch[2];
    vec = sizeof(C) == 8 && (a.N[0] & 1) == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0;
#pragma unroll
    for (int n = 0; n < NCOPY; ++n) {
      const int t = lane + 32 * n;
      int off = vec ? 3 * (i0 - 2) + 2 * t : 3 * (i0 - 1) + t;
      if (off < 0) off = bx ? off + row3 : -1;
      else if (off >= row3) off = (bx && off < row3 + 3) ? off - row3 : -1;
      if (off < 0 || off >= row3 || t >= (vec ? NVEC : NEL)) off = -1;
      cof[n] = off;
    }
    phx = bx && (ex.ph[0].x != R(1) || ex.ph[0].y != R(0));
    phy = by && (ex.ph[1].x != R(1) || ex.ph[1].y != R(0));
    phz = bz && (ex.ph[2].x != R(1) || ex.ph[2].y != R(0));
  }
  __device__ __forceinline__ bool phased() const { return phx || phy || phz; }

  // Issue the warp's rows of plane q into the slot at `slot` (the rows left
  // over go to the last warps: the first ones carry halo jobs).
  __device__ __forceinline__ void copy(const OpArgs<R> &a, unsigned char *slot, int q) const {
    const bool zout = q < 0 || q >= a.N[2];
    const int gq = q < 0 ? q + a.N[2] : q >= a.N[2] ? q - a.N[2] : q;
    for (int r = NW - 1 - w; r < BY; r += NW) {
      int gj = j0 + r - 1;
      bool ok = !zout || bz;
      if (gj < 0) {
        ok = ok && by;
        gj += a.N[1];
      } else if (gj >= a.N[1]) {
        ok = ok && by && gj == a.N[1];
        gj -= a.N[1];
      }
      const C *src = x + (ok ? row3 * (gj + (long long)a.N[1] * gq) : 0);
      const uint32_t dst = smem_u32(slot) + r * (XW * 3 * (int)sizeof(C));
      if (vec) {
#pragma unroll
        for (int n = 0; n < 2; ++n) {
          const bool in = ok && cof[n] >= 0;
          if (lane + 32 * n < NVEC) cp_async<16>(dst + (lane + 32 * n) * 16, src + (in ? cof[n] : 0), in);
        }
      } else {
#pragma unroll
        for (int n = 0; n < NCOPY; ++n) {
          const bool in = ok && cof[n] >= 0;
          if (lane + 32 * n < NEL)
            cp_async<sizeof(C)>(dst + ((XOFF - 1) * 3 + lane + 32 * n) * (int)sizeof(C), src + (in ? cof[n] : 0), in);
        }
      }
    }
  }

  // Multiply the wrapped cells of landed plane q by their phases (the warp's
  // own rows, so only the warp has to have seen its copies land).
  __device__ __forceinline__ void phase(const OpArgs<R> &a, const Extra<R> &ex, unsigned char *slot, int q) const {
    __syncwarp();
    const bool zw = phz && (q < 0 || q >= a.N[2]);
    for (int r = NW - 1 - w; r < BY; r += NW) {
      const int gj = j0 + r - 1;
      const bool yw = phy && (gj < 0 || gj >= a.N[1]);
      C *row = reinterpret_cast<C *>(slot) + (r * XW + XOFF - 1) * 3;
      if (zw || yw) {
        C p = zw ? (q < 0 ? ex.phinv[2] : ex.ph[2]) : mk(R(1), R(0));
        if (yw) p = cmul(p, gj < 0 ? ex.phinv[1] : ex.ph[1]);
        for (int e = lane; e < NEL; e += 32) row[e] = cmul(row[e], p);
        __syncwarp();
      }
      if (phx && lane < 6) {  // column −1 of the first tile, column N_x of the last
        const int e = lane < 3 ? lane : 3 * (a.N[0] - i0 + 1) + lane - 3;
        if (lane < 3 ? i0 == 0 : e < NEL) row[e] = cmul(row[e], lane < 3 ? ex.phinv[0] : ex.ph[0]);
      }
    }
  }
};

}  // namespace fdfd
