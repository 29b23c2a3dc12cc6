// On-device material assignment and Kottke subpixel smoothing.
//
// Replaces calc_matparams! (src/model/full.jl:16-70): assign_param! finds
// the object index (oind) at every sample point, smooth_param! re-computes
// ε on voxels whose corners see more than one object.  The dual-voxel trick
// of the reference is kept: the voxel around an E_w sample has its corners
// on H_w sample points, so ε_ww smoothing reads the object indices sampled at
// H_w positions (full.jl:58-60, 64); the voxel around an E-voxel corner (where
// the off-diagonal ε lives) has its corners at cell centres (full.jl:61, 65).
//
// Rules (shared with the CPU oracle):
//   * objects are applied in add_obj! order with atomicMax on the index, so
//     the last-added object wins; index 0 is the background;
//   * ghost samples: Bloch axes copy the periodic image, a symmetry (PEC)
//     axis copies dual index 0 into the dual ghost and evaluates the primal
//     ghost on the boundary plane;
//   * a voxel with exactly two objects gets ε̃ = ⟨ε⁻¹⟩⁻¹ P + ⟨ε⟩ (I − P),
//     P = n nᵀ, with n the outward normal of the higher-priority object at
//     its point nearest the voxel centre and the fill fraction the exact
//     volume of the voxel behind that tangent plane; more than two objects:
//     mean of the corner ε (off-diagonal 0);
//   * a design region (per-cell ε) overrides: ε_ww = mean of the 4 cells
//     around the E_w edge, off-diagonals 0 at corners touching the region.
// This file is compiled with --fmad=false: every product and sum rounds
// exactly as in the oracle, so object indices and masks are bit-identical.
#include <algorithm>
#include <cmath>
#include <vector>

#include "fdfd_internal.cuh"

namespace fdfd {

int finish_eps(fdfd_handle *h, bool refresh, const unsigned *corners);
int ensure_oflags(fdfd_handle *h);
int ensure_eps_buffers(fdfd_handle *h, bool off);

struct DevObj {
  int kind;
  double eps;
  double p[6];
};

struct Axes {
  const double *pos[3];  // (N+1) sample positions per axis for this sample set
  int n[3];              // extents of the array being indexed
};

__device__ __forceinline__ bool inside(const DevObj &o, double x, double y, double z) {
  if (o.kind == FDFD_SHAPE_SPHERE) {
    const double dx = __dsub_rn(x, o.p[0]), dy = __dsub_rn(y, o.p[1]), dz = __dsub_rn(z, o.p[2]);
    const double d2 = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
    return d2 <= __dmul_rn(o.p[3], o.p[3]);
  }
  if (o.kind == FDFD_SHAPE_CYLZ) {
    const double dx = __dsub_rn(x, o.p[0]), dy = __dsub_rn(y, o.p[1]);
    return __dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)) <= __dmul_rn(o.p[2], o.p[2]);
  }
  return x >= o.p[0] && x <= o.p[3] && y >= o.p[1] && y <= o.p[4] && z >= o.p[2] && z <= o.p[5];
}

// The seven sample sets whose object indices are needed: E_w (0-2, the N³
// samples), H_w (3-5) and cell centres (6), both extended by a ghost sample
// per axis ((N+1)³).
constexpr int NSETS = 7;
struct SampleSets {
  int *o[NSETS];
  Axes ax[NSETS];
};

// Object indices of every set: blockIdx.y = object, blockIdx.z = set, threads
// stride over the object's index box.
__global__ void k_assign(SampleSets S, const DevObj *objs, const int *boxes) {
  const int q = blockIdx.y, set = blockIdx.z;
  const DevObj o = objs[q];
  const Axes &ax = S.ax[set];
  int *oind = S.o[set];
  const int *b = boxes + 6 * ((long long)set * gridDim.y + q);  // lo0, lo1, lo2, hi0, hi1, hi2 (inclusive lo, exclusive hi)
  const int e0 = b[3] - b[0], e1 = b[4] - b[1], e2 = b[5] - b[2];
  if (e0 <= 0 || e1 <= 0 || e2 <= 0) return;
  auto put = [&](int i, int j, int k) {
    if (inside(o, ax.pos[0][i], ax.pos[1][j], ax.pos[2][k]))
      atomicMax(&oind[i + (long long)ax.n[0] * (j + (long long)ax.n[1] * k)], q + 1);
  };
  const long long vol = (long long)e0 * e1 * e2;
  if (vol < (1ll << 30)) {  // 32-bit index arithmetic
    for (unsigned t = blockIdx.x * blockDim.x + threadIdx.x; t < (unsigned)vol; t += gridDim.x * blockDim.x) {
      const unsigned u = t / (unsigned)e0;
      put(b[0] + (int)(t % (unsigned)e0), b[1] + (int)(u % (unsigned)e1), b[2] + (int)(u / (unsigned)e1));
    }
  } else {
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < vol; t += (long long)gridDim.x * blockDim.x)
      put(b[0] + (int)(t % e0), b[1] + (int)((t / e0) % e1), b[2] + (int)(t / ((long long)e0 * e1)));
  }
}

// ------------------------------------------------------------ Kottke
__device__ double sz_volume(double m1, double m2, double m3, double a) {
  const double m12 = m1 + m2;
  if (a < m1) {
    const double t = a / m1;
    return ((t * a) * a) / ((6.0 * m2) * m3);
  }
  if (a < m2) return (a * (a - m1)) / ((2.0 * m2) * m3) + (m1 * m1) / ((6.0 * m2) * m3);
  if (a < fmin(m12, m3)) {
    const double q = a - m2;
    const double base = ((((3.0 * a) * a) - ((3.0 * a) * m1)) + (m1 * m1)) / ((6.0 * m2) * m3);
    return base - ((((q / m1) * q) * q) / ((6.0 * m2) * m3));
  }
  if (m3 < m12) {
    const double q2 = a - m2, q3 = a - m3;
    const double base = ((((3.0 * a) * a) - ((3.0 * a) * m1)) + (m1 * m1)) / ((6.0 * m2) * m3);
    return base - (((((q2 / m1) * q2) * q2) + (((q3 / m1) * q3) * q3)) / ((6.0 * m2) * m3));
  }
  return ((2.0 * a) - m12) / (2.0 * m3);
}

__device__ double volfrac_plane(const double lo[3], const double hi[3], const double n[3], const double r0[3]) {
  double m[3];
  double d = 0.0;
  for (int a = 0; a < 3; ++a) {
    const double side = hi[a] - lo[a];
    double ma = n[a] * side;
    d += n[a] * (r0[a] - lo[a]);
    if (ma < 0.0) {
      d -= ma;
      ma = -ma;
    }
    m[a] = ma;
  }
  const double s = (m[0] + m[1]) + m[2];
  if (s <= 0.0) return 0.5;
  double alpha = d / s;
  if (alpha <= 0.0) return 0.0;
  if (alpha >= 1.0) return 1.0;
  double v0 = m[0] / s, v1 = m[1] / s, v2 = m[2] / s;
  // ascending sort of three
  if (v0 > v1) { double t = v0; v0 = v1; v1 = t; }
  if (v1 > v2) { double t = v1; v1 = v2; v2 = t; }
  if (v0 > v1) { double t = v0; v0 = v1; v1 = t; }
  const double tiny = 1e-12;
  if (v0 < tiny * v2) v0 = 0.0;
  if (v1 < tiny * v2) v1 = 0.0;
  const bool flip = alpha > 0.5;
  if (flip) alpha = 1.0 - alpha;
  const double v = sz_volume(v0, v1, v2, alpha);
  return flip ? 1.0 - v : v;
}

__device__ void normal_point(const DevObj &o, const double xc[3], double n[3], double r0[3]) {
  if (o.kind == FDFD_SHAPE_SPHERE) {
    const double v0 = xc[0] - o.p[0], v1 = xc[1] - o.p[1], v2 = xc[2] - o.p[2];
    const double nr = sqrt((v0 * v0 + v1 * v1) + v2 * v2);
    if (nr == 0.0) { n[0] = 1.0; n[1] = 0.0; n[2] = 0.0; }
    else { n[0] = v0 / nr; n[1] = v1 / nr; n[2] = v2 / nr; }
    for (int a = 0; a < 3; ++a) r0[a] = o.p[a] + o.p[3] * n[a];
    return;
  }
  if (o.kind == FDFD_SHAPE_CYLZ) {
    // radial in the xy-plane (the disk's normal); z follows the point
    const double v0 = xc[0] - o.p[0], v1 = xc[1] - o.p[1], v2 = 0.0;
    const double nr = sqrt((v0 * v0 + v1 * v1) + v2 * v2);
    if (nr == 0.0) { n[0] = 1.0; n[1] = 0.0; n[2] = 0.0; }
    else { n[0] = v0 / nr; n[1] = v1 / nr; n[2] = 0.0; }
    r0[0] = o.p[0] + o.p[2] * n[0];
    r0[1] = o.p[1] + o.p[2] * n[1];
    r0[2] = xc[2];
    return;
  }
  double best = -INFINITY;
  for (int a = 0; a < 3; ++a) {
    for (int side = 0; side < 2; ++side) {
      const double dist = side == 0 ? (o.p[a] - xc[a]) : (xc[a] - o.p[3 + a]);
      if (dist > best) {
        best = dist;
        for (int b = 0; b < 3; ++b) { n[b] = 0.0; r0[b] = xc[b]; }
        n[a] = side == 0 ? -1.0 : 1.0;
        r0[a] = side == 0 ? o.p[a] : o.p[3 + a];
      }
    }
  }
}

__device__ __forceinline__ double obj_eps(const DevObj *objs, double eps_bg, int q) {
  return q == 0 ? eps_bg : objs[q - 1].eps;
}

// Kottke tensor of a voxel [lo, hi] whose 8 corner indices are c[]: ε̃ as
// mean m and difference d of ε̃ = m I + d n nᵀ, with the normal n (m the
// mean of the corner ε and d = 0 where more than two objects meet).
__device__ void smoothed_tensor(const int c[8], const DevObj *objs, double eps_bg, const double lo[3],
                                const double hi[3], double &m, double &d, double n[3]) {
  int qmin = c[0], qmax = c[0];
  for (int t = 1; t < 8; ++t) { qmin = min(qmin, c[t]); qmax = max(qmax, c[t]); }
  bool two = true;
  for (int t = 0; t < 8; ++t) two = two && (c[t] == qmin || c[t] == qmax);
  n[0] = n[1] = n[2] = 0.0;
  if (two) {
    const double efg = obj_eps(objs, eps_bg, qmax), ebg = obj_eps(objs, eps_bg, qmin);
    double xc[3], r0[3];
    for (int a = 0; a < 3; ++a) xc[a] = 0.5 * (lo[a] + hi[a]);
    normal_point(objs[qmax - 1], xc, n, r0);
    const double f = volfrac_plane(lo, hi, n, r0);
    m = f * efg + (1.0 - f) * ebg;
    const double eh = 1.0 / (f / efg + (1.0 - f) / ebg);
    d = eh - m;
  } else {
    double s = 0.0;
    for (int t = 0; t < 8; ++t) s += obj_eps(objs, eps_bg, c[t]);
    m = s / 8.0;
    d = 0.0;
  }
}

// What the smoothing kernels read and write.  Voxel set s < 3 is ε_ss at its
// E_s samples (voxel corners at H_s samples), set 3 the off-diagonal ε at
// the E-voxel corners (voxel corners at cell centres).
struct SmoothArgs {
  int N[3], bloch[3];
  long long nc;
  const int *oe[3];   // object indices at the E_w samples (N³)
  const int *ov[4];   // and at the voxel corners of each set ((N+1)³)
  const double *prim[3], *dual[3];
  const DevObj *objs;
  double eps_bg;
  double *eps, *eoff;
  float *eps32, *eoff32;
  uint8_t *smask;
  unsigned int *nnz;
  uint8_t *flag[3];   // off-diagonal flags of groups of TY, 1 and 2 rows
  int tiles_x;
};

// Source index of extended index t along axis a of voxel set s: a symmetry
// wall's dual ghost copies dual index 0, Bloch ghosts the periodic image.
__device__ __forceinline__ int ghost_src(const SmoothArgs &A, int s, int a, int t) {
  const bool dual = s == 3 || a != s;
  if (dual) return t == 0 ? (A.bloch[a] ? A.N[a] : 1) : t;
  return t == A.N[a] && A.bloch[a] ? 0 : t;
}
// the 8 corner indices in the oracle's order (ravel of o[i:i+2, j:j+2, k:k+2])
__device__ __forceinline__ void corners8(const SmoothArgs &A, int s, int i, int j, int k, int c[8]) {
  const int *o = A.ov[s];
  const long long n0 = A.N[0] + 1, n1 = A.N[1] + 1;
  const int x0 = ghost_src(A, s, 0, i), x1 = ghost_src(A, s, 0, i + 1);
  const int y0 = ghost_src(A, s, 1, j), y1 = ghost_src(A, s, 1, j + 1);
  const int z0 = ghost_src(A, s, 2, k), z1 = ghost_src(A, s, 2, k + 1);
  const int xs[2] = {x0, x1}, ys[2] = {y0, y1}, zs[2] = {z0, z1};
  int t = 0;
#pragma unroll
  for (int a = 0; a < 2; ++a)
#pragma unroll
    for (int b = 0; b < 2; ++b)
#pragma unroll
      for (int d = 0; d < 2; ++d) c[t++] = o[xs[a] + n0 * (ys[b] + n1 * zs[d])];
}

// Voxels of one object: ε of that object, no smoothing.  The others are only
// marked (smask 1) for k_smooth.  Threads run over the flattened x-y plane,
// blockIdx.y strides the planes.
__global__ void __launch_bounds__(256) k_classify(SmoothArgs A) {
  const int plane = A.N[0] * A.N[1];
  const int p = blockIdx.x * 256 + threadIdx.x;
  if (p >= plane) return;
  const int i = p % A.N[0], j = p / A.N[0];
  for (int k = blockIdx.y; k < A.N[2]; k += gridDim.y) {
    const long long cell = (long long)plane * k + p;
    uchar4 mask = make_uchar4(0, 0, 0, 0);
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      int c[8];
      corners8(A, s, i, j, k, c);
      bool same = true;
#pragma unroll
      for (int t = 1; t < 8; ++t) same = same && (c[t] == c[0]);
      if (!same) {
        (&mask.x)[s] = 1;
      } else if (s < 3) {
        const double e = obj_eps(A.objs, A.eps_bg, A.oe[s][cell]);
        A.eps[s * A.nc + cell] = e;
        A.eps32[s * A.nc + cell] = (float)e;
      } else {
#pragma unroll
        for (int q = 0; q < 3; ++q) {
          A.eoff[q * A.nc + cell] = 0.0;
          A.eoff32[q * A.nc + cell] = 0.0f;
        }
      }
    }
    reinterpret_cast<uchar4 *>(A.smask)[cell] = mask;
  }
}

// One marked voxel: its smoothed ε in both precisions and, where an
// off-diagonal is not 0, the flags of the outputs that read it (the corner's
// own cell and the one before it on each axis — across the wrap of a periodic
// one — in groups of g rows).
__device__ void smooth_voxel(const SmoothArgs &A, long long entry, unsigned &cnt) {
  const int s = (int)(entry & 3);
  const long long cell = entry >> 2;
  const int plane = A.N[0] * A.N[1];
  const int k = (int)(cell / plane), p = (int)(cell - (long long)plane * k);
  const int g[3] = {p % A.N[0], p / A.N[0], k};
  int c[8];
  corners8(A, s, g[0], g[1], g[2], c);
  double lo[3], hi[3], n[3], m, d;
  for (int a = 0; a < 3; ++a) {
    const double *pos = (s < 3 && a == s) ? A.prim[a] : A.dual[a];
    lo[a] = pos[g[a]];
    hi[a] = pos[g[a] + 1];
  }
  smoothed_tensor(c, A.objs, A.eps_bg, lo, hi, m, d, n);
  if (s < 3) {
    const double e = m + d * (n[s] * n[s]);
    A.eps[s * A.nc + cell] = e;
    A.eps32[s * A.nc + cell] = (float)e;
    return;
  }
  const double o[3] = {0.0 + d * (n[0] * n[1]), 0.0 + d * (n[1] * n[2]), 0.0 + d * (n[2] * n[0])};
  for (int q = 0; q < 3; ++q) {
    A.eoff[q * A.nc + cell] = o[q];
    A.eoff32[q * A.nc + cell] = (float)o[q];
  }
  if (o[0] == 0.0 && o[1] == 0.0 && o[2] == 0.0) return;
  cnt++;
  const int is[2] = {g[0], cell_before(g[0], A.N[0], A.bloch[0])};
  const int js[2] = {g[1], cell_before(g[1], A.N[1], A.bloch[1])};
  const int kb = cell_before(k, A.N[2], A.bloch[2]);
  for (int f = 0; f < 3; ++f) {
    const int rows = f == 0 ? TY : f;
    for (const int u : is)
      for (const int v : js) {
        const long long tc = u / TX + (long long)A.tiles_x * (v / rows);
        A.flag[f][tc * A.N[2] + k] = 1;
        A.flag[f][tc * A.N[2] + kb] = 1;
      }
  }
}

// The marked voxels, 32 at a time: about 300 FP64 instructions each (a dozen
// divides), which cost a warp the same for one lane as for 32, and they lie
// on surfaces — computed where they were found, nearly every warp that met
// an interface paid for one or two lanes (514 µs at 96³ with 40 spheres).
// Each warp scans the masks (its 32-cell groups interleaved over the grid, so
// all warps meet about the same number) and queues what it finds.
constexpr int SMOOTH_WARPS = 4;
__global__ void __launch_bounds__(SMOOTH_WARPS * 32) k_smooth(SmoothArgs A) {
  __shared__ long long queue[SMOOTH_WARPS][64];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  long long *q = queue[w];
  const long long nw = (long long)gridDim.x * SMOOTH_WARPS;
  unsigned cnt = 0;
  int held = 0;
  for (long long base = (blockIdx.x * (long long)SMOOTH_WARPS + w) * 32; base < A.nc; base += nw * 32) {
    const long long cell = base + lane;
    uchar4 m = make_uchar4(0, 0, 0, 0);
    if (cell < A.nc) m = reinterpret_cast<const uchar4 *>(A.smask)[cell];
    if (!__any_sync(0xffffffffu, (m.x | m.y | m.z | m.w) != 0)) continue;
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      const bool hit = (&m.x)[s] != 0;
      const unsigned b = __ballot_sync(0xffffffffu, hit);
      if (hit) q[held + __popc(b & ((1u << lane) - 1u))] = 4 * cell + s;
      held += __popc(b);
      if (held >= 32) {
        __syncwarp();
        const long long e = q[lane], rest = q[32 + lane];
        smooth_voxel(A, e, cnt);
        held -= 32;
        __syncwarp();
        if (lane < held) q[lane] = rest;
        __syncwarp();
      }
    }
  }
  __syncwarp();
  if (lane < held) smooth_voxel(A, q[lane], cnt);
  if (cnt) atomicAdd(A.nnz, cnt);
}

__device__ __forceinline__ int wrap_or_clamp(int t, int N, int bloch) {
  if (t < 0) return bloch ? t + N : 0;
  if (t >= N) return bloch ? t - N : N - 1;
  return t;
}

struct DesignDev {
  int lo[3], hi[3];
  const double *eps;  // x fastest over the region
  int bloch[3];
};

__device__ __forceinline__ bool in_region(const DesignDev &d, int i, int j, int k) {
  return i >= d.lo[0] && i < d.hi[0] && j >= d.lo[1] && j < d.hi[1] && k >= d.lo[2] && k < d.hi[2];
}

__device__ __forceinline__ double cell_value(const DesignDev &d, const int *oc, int N0, int N1, const DevObj *objs,
                                             double eps_bg, int i, int j, int k) {
  if (in_region(d, i, j, k)) {
    const int e0 = d.hi[0] - d.lo[0], e1 = d.hi[1] - d.lo[1];
    return d.eps[(i - d.lo[0]) + (long long)e0 * ((j - d.lo[1]) + (long long)e1 * (k - d.lo[2]))];
  }
  // cell centre = dual ext index + 1 on every axis
  return obj_eps(objs, eps_bg, oc[(i + 1) + (long long)(N0 + 1) * ((j + 1) + (long long)(N1 + 1) * (k + 1))]);
}

__global__ void k_design_diag(int w, int N0, int N1, int N2, DesignDev d, const int *oc, const DevObj *objs,
                              double eps_bg, double *eps, uint8_t *smask) {
  const long long nc = (long long)N0 * N1 * N2;
  const int N[3] = {N0, N1, N2};
  const int u0 = (w == 0) ? 1 : 0, u1 = (w == 2) ? 1 : 2;
  for (long long cell = blockIdx.x * (long long)blockDim.x + threadIdx.x; cell < nc;
       cell += (long long)gridDim.x * blockDim.x) {
    const int g[3] = {(int)(cell % N0), (int)((cell / N0) % N1), (int)(cell / ((long long)N0 * N1))};
    double acc = 0.0;
    bool touch = false;
    for (int s0 = -1; s0 <= 0; ++s0)
      for (int s1 = -1; s1 <= 0; ++s1) {
        int t[3] = {g[0], g[1], g[2]};
        t[u0] = wrap_or_clamp(g[u0] + s0, N[u0], d.bloch[u0]);
        t[u1] = wrap_or_clamp(g[u1] + s1, N[u1], d.bloch[u1]);
        acc += cell_value(d, oc, N0, N1, objs, eps_bg, t[0], t[1], t[2]);
        touch = touch || in_region(d, t[0], t[1], t[2]);
      }
    if (touch) {
      eps[w * nc + cell] = 0.25 * acc;
      smask[4 * cell + w] = 2;
    }
  }
}

__global__ void k_design_off(int N0, int N1, int N2, DesignDev d, double *eoff, uint8_t *smask) {
  const long long nc = (long long)N0 * N1 * N2;
  const int N[3] = {N0, N1, N2};
  for (long long cell = blockIdx.x * (long long)blockDim.x + threadIdx.x; cell < nc;
       cell += (long long)gridDim.x * blockDim.x) {
    const int g[3] = {(int)(cell % N0), (int)((cell / N0) % N1), (int)(cell / ((long long)N0 * N1))};
    bool touch = false;
    for (int s = 0; s < 8; ++s) {
      int t[3];
      for (int a = 0; a < 3; ++a) t[a] = wrap_or_clamp(g[a] - ((s >> (2 - a)) & 1), N[a], d.bloch[a]);
      touch = touch || in_region(d, t[0], t[1], t[2]);
    }
    if (touch) {
      eoff[cell] = eoff[nc + cell] = eoff[2 * nc + cell] = 0.0;
      smask[4 * cell + 3] = 2;
    }
  }
}

// ------------------------------------------------------------ host
namespace {
// Device scratch of one call, cut from one allocation.  Up to KEEP bytes stay
// with the handle for the next call (an allocation and a free cost as much
// as the smoothing itself at small sizes); larger ones are freed at the end.
struct Scratch {
  static constexpr size_t KEEP = 64u << 20;
  fdfd_handle *h;
  char *base = nullptr;
  size_t used = 0;
  explicit Scratch(fdfd_handle *h_) : h(h_) {}
  ~Scratch() {
    if (base && base != h->setup_scratch) cudaFree(base);
  }
  static size_t pad(size_t n) { return (n + 255) / 256 * 256; }
  int reserve(size_t bytes) {
    if (bytes <= h->setup_bytes) {
      base = static_cast<char *>(h->setup_scratch);
      return FDFD_OK;
    }
    void *p = nullptr;
    if (dev_malloc(&p, bytes) != cudaSuccess) {
      cudaGetLastError();
      return set_error(h, FDFD_ERR_NOMEM, "cudaMalloc in fdfd_smooth_objects failed");
    }
    base = static_cast<char *>(p);
    if (bytes <= KEEP) {
      cudaFree(h->setup_scratch);
      h->setup_scratch = p;
      h->setup_bytes = bytes;
    }
    return FDFD_OK;
  }
  template <typename T>
  T *get(size_t n) {
    T *p = reinterpret_cast<T *>(base + used);
    used += pad(n * sizeof(T));
    return p;
  }
};

// index range [first, last] of sorted positions within [a - tiny, b + tiny]
void index_range(const double *pos, int n, double a, double b, int *lo, int *hi) {
  const double pad = 1e-9 * (1.0 + std::fabs(a) + std::fabs(b));
  *lo = (int)(std::lower_bound(pos, pos + n, a - pad) - pos);
  *hi = (int)(std::upper_bound(pos, pos + n, b + pad) - pos);
}
}  // namespace

int smooth_objects_impl(fdfd_handle *h, const double *const lprim[3], const fdfd_object *objs, int nobj,
                        double eps_bg, const fdfd_design *design) {
  const int N0 = h->N[0], N1 = h->N[1], N2 = h->N[2];
  const long long nc = h->ncell;
  const long long next = (long long)(N0 + 1) * (N1 + 1) * (N2 + 1);
  int rc = FDFD_OK;
  // per-axis positions: primal with +end ghost (N+1), dual with −end ghost (N+1)
  std::vector<double> prim[3], dual[3];
  for (int w = 0; w < 3; ++w) {
    const int N = h->N[w];
    prim[w].assign(lprim[w], lprim[w] + N + 1);
    for (int i = 0; i < N; ++i)
      if (!(prim[w][i + 1] > prim[w][i])) return set_error(h, FDFD_ERR_ARG, "lprim must be strictly increasing");
    const double L = prim[w][N] - prim[w][0];
    std::vector<double> mid(N);
    for (int i = 0; i < N; ++i) mid[i] = 0.5 * (prim[w][i] + prim[w][i + 1]);
    const double g = h->bloch[w] ? mid[N - 1] - L : 2.0 * prim[w][0] - mid[0];
    dual[w].resize(N + 1);
    dual[w][0] = g;
    for (int i = 0; i < N; ++i) dual[w][i + 1] = mid[i];
  }
  for (int q = 0; q < nobj; ++q) {
    if (objs[q].kind != FDFD_SHAPE_SPHERE && objs[q].kind != FDFD_SHAPE_BOX && objs[q].kind != FDFD_SHAPE_CYLZ)
      return set_error(h, FDFD_ERR_ARG, "unknown shape kind");
    if (!(objs[q].eps > 0.0)) return set_error(h, FDFD_ERR_UNSUPPORTED, "object ε must be real and positive");
  }
  if (!(eps_bg > 0.0)) return set_error(h, FDFD_ERR_UNSUPPORTED, "background ε must be real and positive");
  if (design) {
    for (int a = 0; a < 3; ++a)
      if (design->lo[a] < 0 || design->hi[a] > h->N[a] || design->lo[a] >= design->hi[a] || !design->eps_cells)
        return set_error(h, FDFD_ERR_ARG, "bad design region");
  }
  // Host side of one upload: positions, objects, the objects' index boxes in
  // every sample set.  Set types per axis: 0 primal, 1 dual; extended sets
  // ((N+1)³ with ghosts) take all N+1 positions, the N³ E samples the first N
  // primal ones or the dual ones after the ghost.
  auto is_dual = [](int set, int a) { return set == 6 || (set < 3 ? a == set : a != set - 3); };
  const size_t nob = (size_t)std::max(1, nobj);
  size_t npos = 0;
  for (int w = 0; w < 3; ++w) npos += 2 * (size_t)(h->N[w] + 1);
  const size_t ne = design ? (size_t)(design->hi[0] - design->lo[0]) * (design->hi[1] - design->lo[1]) *
                                 (design->hi[2] - design->lo[2])
                           : 0;
  const size_t up_obj = Scratch::pad(npos * sizeof(double)), up_box = up_obj + Scratch::pad(nob * sizeof(DevObj));
  const size_t up_nnz = up_box + Scratch::pad(6 * NSETS * nob * sizeof(int)), up_bytes = up_nnz + 256;
  std::vector<char> up(up_bytes, 0);
  double *hpos = reinterpret_cast<double *>(up.data());
  const double *hprim[3], *hdual[3];
  size_t off_prim[3], off_dual[3];
  {
    size_t o = 0;
    for (int w = 0; w < 3; ++w) {
      off_prim[w] = o;
      hprim[w] = hpos + o;
      o = std::copy(prim[w].begin(), prim[w].end(), hpos + o) - hpos;
      off_dual[w] = o;
      hdual[w] = hpos + o;
      o = std::copy(dual[w].begin(), dual[w].end(), hpos + o) - hpos;
    }
  }
  DevObj *hob = reinterpret_cast<DevObj *>(up.data() + up_obj);
  int *hbox = reinterpret_cast<int *>(up.data() + up_box);
  long long vmax = 1;  // points of the largest index box
  for (int q = 0; q < nobj; ++q) {
    hob[q].kind = objs[q].kind;
    hob[q].eps = objs[q].eps;
    for (int t = 0; t < 6; ++t) hob[q].p[t] = objs[q].p[t];
    double lo[3], hi[3];
    if (objs[q].kind == FDFD_SHAPE_SPHERE)
      for (int w = 0; w < 3; ++w) { lo[w] = objs[q].p[w] - objs[q].p[3]; hi[w] = objs[q].p[w] + objs[q].p[3]; }
    else if (objs[q].kind == FDFD_SHAPE_CYLZ) {
      for (int w = 0; w < 2; ++w) { lo[w] = objs[q].p[w] - objs[q].p[2]; hi[w] = objs[q].p[w] + objs[q].p[2]; }
      lo[2] = -HUGE_VAL;
      hi[2] = HUGE_VAL;
    } else
      for (int w = 0; w < 3; ++w) { lo[w] = objs[q].p[w]; hi[w] = objs[q].p[3 + w]; }
    int r[3][2][2][2];  // [axis][dual][extended][lo, hi]
    for (int w = 0; w < 3; ++w)
      for (int e = 0; e < 2; ++e) {
        index_range(hprim[w], h->N[w] + e, lo[w], hi[w], &r[w][0][e][0], &r[w][0][e][1]);
        index_range(hdual[w] + (1 - e), h->N[w] + e, lo[w], hi[w], &r[w][1][e][0], &r[w][1][e][1]);
      }
    for (int set = 0; set < NSETS; ++set) {
      long long vol = 1;
      for (int w = 0; w < 3; ++w) {
        const int *e = r[w][is_dual(set, w) ? 1 : 0][set < 3 ? 0 : 1];
        for (int v = 0; v < 2; ++v) hbox[6 * ((size_t)set * nobj + q) + 3 * v + w] = e[v];
        vol *= std::max(0, e[1] - e[0]);
      }
      vmax = std::max(vmax, vol);
    }
  }

  Scratch buf(h);
  const size_t e_bytes = Scratch::pad(nc * sizeof(int)), x_bytes = Scratch::pad(next * sizeof(int));
  if ((rc = buf.reserve(up_bytes + 3 * e_bytes + 4 * x_bytes + Scratch::pad(ne * sizeof(double))))) return rc;
  if (!h->smask) {
    if (dev_malloc(&h->smask, 4 * (size_t)nc) != cudaSuccess) {
      cudaGetLastError();
      return set_error(h, FDFD_ERR_NOMEM, "cudaMalloc(smask) failed");
    }
  }
  if ((rc = ensure_eps_buffers(h, true))) return rc;
  if ((rc = ensure_oflags(h))) return rc;

  char *dup = buf.get<char>(up_bytes);
  int *oind = reinterpret_cast<int *>(buf.get<char>(3 * e_bytes + 4 * x_bytes));
  double *deps = buf.get<double>(ne);
  const double *dpos = reinterpret_cast<const double *>(dup);
  const DevObj *dobj = reinterpret_cast<const DevObj *>(dup + up_obj);
  cudaStream_t st = h->stream;
  if ((rc = cuda_check(h, cudaMemcpyAsync(dup, up.data(), up_bytes, cudaMemcpyHostToDevice, st), "upload objects")))
    return rc;
  if ((rc = cuda_check(h, cudaMemsetAsync(oind, 0, 3 * e_bytes + 4 * x_bytes, st), "memset indices"))) return rc;

  SampleSets S;
  SmoothArgs A;
  for (int set = 0; set < NSETS; ++set) {
    S.o[set] = reinterpret_cast<int *>(reinterpret_cast<char *>(oind) +
                                       (set < 3 ? set * e_bytes : 3 * e_bytes + (set - 3) * x_bytes));
    for (int w = 0; w < 3; ++w) {
      const bool du = is_dual(set, w);
      const double *base = dpos + (du ? off_dual[w] : off_prim[w]);
      S.ax[set].pos[w] = (set < 3 && du) ? base + 1 : base;
      S.ax[set].n[w] = set < 3 ? h->N[w] : h->N[w] + 1;
    }
  }
  for (int w = 0; w < 3; ++w) {
    A.N[w] = h->N[w];
    A.bloch[w] = h->bloch[w];
    A.oe[w] = S.o[w];
    A.prim[w] = dpos + off_prim[w];
    A.dual[w] = dpos + off_dual[w];
  }
  for (int s = 0; s < 4; ++s) A.ov[s] = S.o[3 + s];
  A.nc = nc;
  A.objs = dobj;
  A.eps_bg = eps_bg;
  A.eps = h->eps64;
  A.eoff = h->eoff64;
  A.eps32 = h->eps32;
  A.eoff32 = h->eoff32;
  A.smask = h->smask;
  A.nnz = reinterpret_cast<unsigned int *>(dup + up_nnz);
  A.flag[0] = h->oflag;
  A.flag[1] = h->oflag_rows[0];
  A.flag[2] = h->oflag_rows[1];
  A.tiles_x = (h->N[0] + TX - 1) / TX;
  const int gx = (int)std::min(64ll, vmax / 2048 + 1);  // about eight points per thread of the largest box
  if (nobj > 0) k_assign<<<dim3(gx, nobj, NSETS), 256, 0, st>>>(S, dobj, reinterpret_cast<const int *>(dup + up_box));
  const long long pblk = ((long long)N0 * N1 + 255) / 256;
  k_classify<<<dim3((unsigned)pblk, (unsigned)std::min(N2, 65535)), 256, 0, st>>>(A);
  k_smooth<<<152 * 2, SMOOTH_WARPS * 32, 0, st>>>(A);
  if ((rc = cuda_check(h, cudaGetLastError(), "smoothing kernels"))) return rc;
  h->has_design = design != nullptr;
  if (design) {
    for (int a = 0; a < 3; ++a) {
      h->design_lo[a] = design->lo[a];
      h->design_hi[a] = design->hi[a];
    }
    DesignDev dd;
    if ((rc = cuda_check(h, cudaMemcpyAsync(deps, design->eps_cells, ne * sizeof(double), cudaMemcpyHostToDevice, st),
                         "upload design")))
      return rc;
    for (int a = 0; a < 3; ++a) {
      dd.lo[a] = design->lo[a];
      dd.hi[a] = design->hi[a];
      dd.bloch[a] = h->bloch[a];
    }
    dd.eps = deps;
    for (int w = 0; w < 3; ++w)
      k_design_diag<<<152 * 8, 256, 0, st>>>(w, N0, N1, N2, dd, S.o[6], dobj, eps_bg, h->eps64, h->smask);
    k_design_off<<<152 * 8, 256, 0, st>>>(N0, N1, N2, dd, h->eoff64, h->smask);
    if ((rc = cuda_check(h, cudaGetLastError(), "design kernels"))) return rc;
  }
  // the corner lists of the new ε, so that their count comes with nnz (a
  // design region's flags are not yet up to date)
  bool lists = false;
  if (!design && (rc = queue_corner_lists(h, A.nnz + 1, &lists))) return rc;
  unsigned int cnt[2] = {0, 0};  // nnz, corners
  cudaMemcpyAsync(cnt, A.nnz, sizeof(cnt), cudaMemcpyDeviceToHost, st);
  if ((rc = cuda_check(h, cudaStreamSynchronize(st), "smoothing sync"))) return rc;
  // design zeroing can only remove off-diagonals; keep the flag conservative
  h->has_off = cnt[0] > 0;
  // the FP32 copies and the flags are written already, except where a design
  // region changed ε since
  return finish_eps(h, design != nullptr, lists ? &cnt[1] : nullptr);
}

}  // namespace fdfd
