// Grid-wide reductions and the scalar recurrences of the Krylov solvers.
//
// Every reducing kernel writes its partial sums per block; the last block
// to arrive (atomic counter) sums them in block order — so the result is
// deterministic — and runs the scalar update of the solver step
// (finalise).  No block ever waits on another: the counter is only read by
// the block that incremented it last.  complex128 kernels sum in FP64;
// complex64 kernels sum in double-float FP32 arithmetic (DF below) up to
// the single value per sum that is widened for finalise.
#pragma once

#include "fdfd_internal.cuh"

namespace fdfd {

enum FinMode : int {
  FIN_NONE = 0,    // store the sums in sc->dot0 / sc->dot1
  FIN_ALPHA = 1,   // BiCGSTAB: α = ρ / (r̂, v)
  FIN_OMEGA = 2,   // BiCGSTAB: ω = (t, s) / (t, t)
  FIN_XR = 3,      // BiCGSTAB: ρ' = (r̂, r), β = ρ'/ρ · α/ω, ‖r‖², stop tests
  FIN_RESID = 4,   // ‖b − A x‖² into dot0.x (reliable update / final check)
  FIN_COCG_A = 5,  // COCG: α = ρ / (pᵀ q)
  FIN_COCG_R = 6,  // COCG: ρ' = rᵀ r, β = ρ'/ρ, ‖r‖², stop tests
  FIN_BL_RHO = 7,    // BiCGStab(ℓ) inside a cycle: ρ₁ = (r̂, r_j), β = α ρ₁/ρ₀, ρ₀ = ρ₁
  FIN_BL_CYCLE = 8,  // BiCGStab(ℓ) cycle end: ρ₀ = −ω ρ₀, then as FIN_BL_RHO; ‖r₀‖², stop tests
  FIN_BL_REDO = 9,   // after a replaced residual: ρ₁ = (r̂, r₀) against the stored −ω ρ₀
};

// a / b, called by a converged warp: a warp's FP64 instruction takes 64
// cycles of its scheduler's pipe for one lane as for 32, so lane 1 divides
// the imaginary part in the same instructions as the other lanes the real one.
__device__ __forceinline__ double2 dcdiv(double2 a, double2 b) {
  const bool im = (threadIdx.x & 31) == 1;
  const double d = b.x * b.x + b.y * b.y;
  const double p = im ? a.y : a.x, q = im ? -a.x : a.y;
  const double v = (p * b.x + q * b.y) / d;
  return make_double2(__shfl_sync(0xffffffffu, v, 0), __shfl_sync(0xffffffffu, v, 1));
}
__device__ __forceinline__ double2 dcmul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ bool dfinite(double2 a) { return isfinite(a.x) && isfinite(a.y); }

__device__ __forceinline__ void stop_tests(KScalars *sc, double rr) {
  sc->rr = rr;
  sc->iter += 1;
  if (rr > sc->rr_max) sc->rr_max = rr;
  if (!isfinite(rr)) { sc->done = 1; sc->reason = 4; return; }
  if (rr <= sc->stop2) { sc->done = 1; sc->reason = 1; return; }
  if (rr <= sc->upd2 * sc->rr_max) { sc->done = 1; sc->reason = 2; return; }
}

// The scalar step of a reduction, run by the first warp of the last block
// (all lanes hold the same sums; lane 0 stores).
__device__ inline void finalise(int mode, KScalars *sc, double2 d0, double2 d1) {
  const bool w = (threadIdx.x & 31) == 0;
  const double2 rho = sc->rho, alpha = sc->alpha, omega = sc->omega, rho_pre = sc->rho_pre;
  __syncwarp();  // every lane has read the old scalars
  if (w) {
    sc->dot0 = d0;
    sc->dot1 = d1;
  }
  auto stop = [&](int reason) {
    if (w) {
      sc->done = 1;
      sc->reason = reason;
    }
  };
  // the stop tests of an iteration's end; a vanished scalar is a breakdown
  // unless they already stop the iteration
  auto broken = [&](bool tests) {
    if (!w) return;
    if (tests) stop_tests(sc, d1.x);
    if (!sc->done) {
      sc->done = 1;
      sc->reason = 3;
    }
  };
  auto zero = [](double2 v) { return v.x == 0.0 && v.y == 0.0; };
  switch (mode) {
    case FIN_ALPHA:
    case FIN_COCG_A: {
      if (!dfinite(d0)) { stop(4); break; }
      if (zero(d0)) { stop(3); break; }
      const double2 al = dcdiv(rho, d0);
      if (w) sc->alpha = al;
      break;
    }
    case FIN_OMEGA: {
      if (!dfinite(d0) || !isfinite(d1.x)) { stop(4); break; }
      if (w) sc->omega = d1.x > 0.0 ? make_double2(d0.x / d1.x, d0.y / d1.x) : make_double2(0.0, 0.0);
      break;
    }
    case FIN_XR: {
      if (zero(omega) || zero(d0)) { broken(true); break; }
      const double2 be = dcmul(dcdiv(d0, rho), dcdiv(alpha, omega));
      if (w) {
        sc->beta = be;
        sc->rho = d0;
        stop_tests(sc, d1.x);
      }
      break;
    }
    case FIN_BL_RHO:
    case FIN_BL_REDO:
    case FIN_BL_CYCLE: {
      double2 rho0 = mode == FIN_BL_RHO ? rho : rho_pre;
      if (mode == FIN_BL_CYCLE) {
        rho0 = make_double2(-(omega.x * rho.x - omega.y * rho.y), -(omega.x * rho.y + omega.y * rho.x));
        if (w) {
          sc->rho_pre = rho0;
          sc->bl_steps = 0;  // x holds this cycle's steps: a breakdown found from here on has none to add
        }
      }
      if (!dfinite(d0)) { stop(4); break; }
      if (zero(rho0)) { broken(mode == FIN_BL_CYCLE); break; }
      const double2 be = dcmul(alpha, dcdiv(d0, rho0));
      if (w) {
        sc->beta = be;
        sc->rho = d0;
        if (mode == FIN_BL_CYCLE) stop_tests(sc, d1.x);
      }
      break;
    }
    case FIN_COCG_R: {
      if (zero(rho)) { stop(3); break; }
      const double2 be = dcdiv(d0, rho);
      if (w) {
        sc->beta = be;
        sc->rho = d0;
        stop_tests(sc, d1.x);
      }
      break;
    }
    default:
      break;
  }
}

// The BiCGStab(ℓ) shadow vector r̂, generated from the DOF index instead of
// stored: r̂_i = (a + i·b)/32768 with a, b the two 16-bit halves (as signed
// integers) of a 32-bit integer hash of i — Chris Wellons' "lowbias32"
// mixing function (xor-shift / multiply rounds).  Any fixed r̂ is a valid
// shadow vector; a random one converged at least as fast as r̂ = r₀ on
// these systems, and generating it saves a vector read in every operator
// application with a dot product.  The values are exact in FP32, so both
// precisions use the same r̂.
__host__ __device__ __forceinline__ uint32_t shadow_hash(uint32_t x) {
  x ^= x >> 16;
  x *= 0x7feb352dU;
  x ^= x >> 15;
  x *= 0x846ca68bU;
  x ^= x >> 16;
  return x;
}
template <typename R>
__device__ __forceinline__ typename CT<R>::C shadow(long long dof) {
  const uint32_t hsh = shadow_hash((uint32_t)dof);
  if constexpr (sizeof(R) == 4) {
    // the same values without integer→float conversions: a half h, read as
    // signed, is (h ^ 0x8000) − 32768; the float with bits 0x4B000000 | v is
    // 2²³ + v exactly, and (2²³ + v)·2⁻¹⁵ − (2⁸ + 1) = (v − 32768)/32768
    // is exact in one fused multiply-add per lane
    const float2 b = make_float2(__uint_as_float(0x4B000000u | ((hsh & 0xffffu) ^ 0x8000u)),
                                 __uint_as_float(0x4B000000u | ((hsh >> 16) ^ 0x8000u)));
    return __ffma2_rn(b, make_float2(1.0f / 32768.0f, 1.0f / 32768.0f), make_float2(-257.0f, -257.0f));
  } else {
    // the double with high word 0x42400000 and low word v is 2³⁷ + v·2⁻¹⁵
    // exactly: one FP64 instruction per value (a conversion and a product
    // would be two)
    return mk(__hiloint2double(0x42400000, (int)((hsh & 0xffffu) ^ 0x8000u)) - 137438953473.0,
              __hiloint2double(0x42400000, (int)((hsh >> 16) ^ 0x8000u)) - 137438953473.0);
  }
}

template <typename R>
__device__ __forceinline__ typename CT<R>::C tocr(double2 v) {
  return mk(R(v.x), R(v.y));
}

// Complex scalars of the recurrence in the kernel's precision (at(i) gives
// the i-th as double2).  complex64 kernels convert each one once per block
// into shared memory: an FP64 → FP32 conversion runs on the narrow FP64
// pipe, and done by every thread it held back the first vector loads by
// microseconds.  Every thread of the block must call it.
template <typename R, int NS, typename F>
__device__ __forceinline__ void scalars(F at, typename CT<R>::C (&out)[NS]) {
  using C = typename CT<R>::C;
  if constexpr (sizeof(R) == 8) {
#pragma unroll
    for (int i = 0; i < NS; ++i) out[i] = at(i);
  } else {
    __shared__ C s[NS];
    if (threadIdx.x < NS) s[threadIdx.x] = tocr<R>(at(threadIdx.x));
    __syncthreads();
#pragma unroll
    for (int i = 0; i < NS; ++i) out[i] = s[i];
  }
}

// Error-free FP32 addition (Knuth's TwoSum): s + e == a + b exactly.
__device__ __forceinline__ void two_sum_f(float a, float b, float &s, float &e) {
  s = a + b;
  const float bb = s - a;
  e = (a - (s - bb)) + (b - bb);
}

// Double-float value hi + lo: about 48 significant bits carried in FP32
// arithmetic.  The GPU's FP64 pipe (conversions included) is a small
// fraction of its FP32 pipe, so the complex64 kernels keep every
// cross-thread and cross-block sum in this form.
struct DF {
  float hi, lo;
};
__device__ __forceinline__ DF df_add(DF a, DF b) {
  float s, e;
  two_sum_f(a.hi, b.hi, s, e);
  e += a.lo + b.lo;
  DF r;
  two_sum_f(s, e, r.hi, r.lo);
  return r;
}
__device__ __forceinline__ DF df_shfl_xor(DF v, int o) {
  return DF{__shfl_xor_sync(0xffffffffu, v.hi, o), __shfl_xor_sync(0xffffffffu, v.lo, o)};
}
__device__ __forceinline__ double df_widen(DF v) { return (double)v.hi + (double)v.lo; }

// Warp reduce-scatter of K double-float values per lane (K a power of two,
// ≤ 32): butterfly levels 16, 8, … each halve the values a lane keeps
// (lanes with the level's bit set keep the upper half), then plain
// butterfly levels once one value is left — K−1+(5−log2 K) additions per
// lane instead of 5K.  Lane l ends with the warp sum of value
// l >> (5 − log2 K) in v[0]; the order of additions is fixed.
template <int M, int O>
struct DfScatter {
  static __device__ __forceinline__ void run(DF *v, int lane) {
    if constexpr (M > 1) {
      const bool up = (lane & O) != 0;
#pragma unroll
      for (int i = 0; i < M / 2; ++i) {
        const DF keep = up ? v[M / 2 + i] : v[i];
        const DF send = up ? v[i] : v[M / 2 + i];
        v[i] = df_add(keep, df_shfl_xor(send, O));
      }
      DfScatter<M / 2, O / 2>::run(v, lane);
    } else {
      v[0] = df_add(v[0], df_shfl_xor(v[0], O));
      DfScatter<1, O / 2>::run(v, lane);
    }
  }
};
template <int M>
struct DfScatter<M, 0> {
  static __device__ __forceinline__ void run(DF *, int) {}
};
template <int K>
constexpr int df_shift() {
  return K >= 32 ? 0 : K >= 16 ? 1 : K >= 8 ? 2 : K >= 4 ? 3 : K >= 2 ? 4 : 5;
}

// Block and grid sums of KR double-float values per thread (v holds K ≥ KR
// slots, K a power of two, the slots from KR on zero).  Writes the block's
// KR partials (float2 each, KR/2 double2 slots of red.part per block) and
// returns true in the block that arrives last, which then holds the grid
// sums, widened to FP64, in tot (shared, KR entries).  Every thread of the
// block must call it.
template <int NT, int K, int KR>
__device__ bool df_block_sums_last(DF (&v)[K], RedBuf red, double *tot) {
  static_assert((K & (K - 1)) == 0 && K <= 32 && KR <= K && (KR % 2) == 0, "DF block sums");
  constexpr int NW = NT / 32;
  __shared__ DF wred[NW][K];
  __shared__ bool last;
  const int tid = threadIdx.x + blockDim.x * (threadIdx.y + blockDim.y * threadIdx.z);
  const int lane = tid & 31, wid = tid >> 5;
  DfScatter<K, 16>::run(v, lane);
  if ((lane & ((1 << df_shift<K>()) - 1)) == 0) wred[wid][lane >> df_shift<K>()] = v[0];
  __syncthreads();
  const unsigned nblk = gridDim.x * gridDim.y * gridDim.z;
  const unsigned bid = blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z);
  float2 *part = reinterpret_cast<float2 *>(red.part);
  if (tid < KR) {
    DF s = wred[0][tid];
#pragma unroll
    for (int w = 1; w < NW; ++w) s = df_add(s, wred[w][tid]);
    part[(long long)KR * bid + tid] = make_float2(s.hi, s.lo);
    __threadfence();
  }
  __syncthreads();
  if (tid == 0) last = atomicAdd(red.count, 1u) == nblk - 1;
  __syncthreads();
  if (!last) return false;
  __threadfence();
  // value q is summed by warp q mod NW: lanes over the blocks in a fixed
  // order, then a fixed butterfly
  for (int q = wid; q < KR; q += NW) {
    DF s{0.f, 0.f};
    for (unsigned b = lane; b < nblk; b += 32) {
      const float2 p = __ldcg(&part[(long long)KR * b + q]);
      s = df_add(s, DF{p.x, p.y});
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s = df_add(s, df_shfl_xor(s, o));
    if (lane == 0) tot[q] = df_widen(s);
  }
  __syncthreads();
  if (tid == 0) *red.count = 0u;
  return true;
}

// complex64 kernels: grid sums of the complex a0 and a1 (as four
// double-float reals), then finalise in the last block.
template <int NT>
__device__ inline void block_reduce_finalise_df(DF a0r, DF a0i, DF a1r, DF a1i, RedBuf red, int mode, KScalars *sc) {
  __shared__ double tot[4];
  DF v[4] = {a0r, a0i, a1r, a1i};
  if (!df_block_sums_last<NT, 4, 4>(v, red, tot)) return;
  if (threadIdx.x + blockDim.x * (threadIdx.y + blockDim.y * threadIdx.z) < 32 && sc)
    finalise(mode, sc, make_double2(tot[0], tot[1]), make_double2(tot[2], tot[3]));
}

// The FP64 counterparts for complex128 kernels.  The reduce-scatter matters
// more here: a butterfly on each of the Gram matrix's 28 sums is 140 FP64
// instructions of 64 cycles per warp, the scatter 31.
template <int M, int O>
struct DScatter {
  static __device__ __forceinline__ void run(double *v, int lane) {
    if constexpr (M > 1) {
      const bool up = (lane & O) != 0;
#pragma unroll
      for (int i = 0; i < M / 2; ++i) {
        const double keep = up ? v[M / 2 + i] : v[i];
        const double send = up ? v[i] : v[M / 2 + i];
        v[i] = keep + __shfl_xor_sync(0xffffffffu, send, O);
      }
      DScatter<M / 2, O / 2>::run(v, lane);
    } else {
      v[0] += __shfl_xor_sync(0xffffffffu, v[0], O);
      DScatter<1, O / 2>::run(v, lane);
    }
  }
};
template <int M>
struct DScatter<M, 0> {
  static __device__ __forceinline__ void run(double *, int) {}
};

// Block and grid sums of KR FP64 values per thread, as df_block_sums_last
// (KR doubles of red.part per block); tot holds the grid sums in the last
// block, which sums the blocks' partials with all its warps.
template <int NT, int K, int KR>
__device__ bool d_block_sums_last(double (&v)[K], RedBuf red, double *tot) {
  static_assert((K & (K - 1)) == 0 && K <= 32 && KR <= K && (KR % 2) == 0, "FP64 block sums");
  constexpr int NW = NT / 32;
  constexpr int G = KR <= NW ? NW / KR : 1;  // warps that share one value's partials
  __shared__ double wred[NW][K];
  __shared__ bool last;
  const int tid = threadIdx.x + blockDim.x * (threadIdx.y + blockDim.y * threadIdx.z);
  const int lane = tid & 31, wid = tid >> 5;
  DScatter<K, 16>::run(v, lane);
  if ((lane & ((1 << df_shift<K>()) - 1)) == 0) wred[wid][lane >> df_shift<K>()] = v[0];
  __syncthreads();
  const unsigned nblk = gridDim.x * gridDim.y * gridDim.z;
  const unsigned bid = blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z);
  double *part = reinterpret_cast<double *>(red.part);
  if (tid < KR) {
    double s = wred[0][tid];
#pragma unroll
    for (int w = 1; w < NW; ++w) s += wred[w][tid];
    part[(long long)KR * bid + tid] = s;
    __threadfence();
  }
  __syncthreads();
  if (tid == 0) last = atomicAdd(red.count, 1u) == nblk - 1;
  __syncthreads();
  if (!last) return false;
  __threadfence();
  for (int q = wid; q < KR * G; q += NW) {
    const int val = q % KR, g = q / KR;
    double s = 0.0;
    for (unsigned b = lane + 32 * g; b < nblk; b += 32 * G) s += __ldcg(&part[(long long)KR * b + val]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) wred[g][val] = s;
  }
  __syncthreads();
  if (tid < KR) {
    double s = wred[0][tid];
#pragma unroll
    for (int g = 1; g < G; ++g) s += wred[g][tid];
    tot[tid] = s;
  }
  __syncthreads();
  if (tid == 0) *red.count = 0u;
  return true;
}

// complex128 kernels: grid sums of the complex a0 and a1, then finalise in
// the last block.  Must be called by every thread of the block.
template <int NT>
__device__ inline void block_reduce_finalise(double2 a0, double2 a1, RedBuf red, int mode, KScalars *sc) {
  __shared__ double tot[4];
  double v[4] = {a0.x, a0.y, a1.x, a1.y};
  if (!d_block_sums_last<NT, 4, 4>(v, red, tot)) return;
  if (threadIdx.x + blockDim.x * (threadIdx.y + blockDim.y * threadIdx.z) < 32 && sc)
    finalise(mode, sc, make_double2(tot[0], tot[1]), make_double2(tot[2], tot[3]));
}

// Per-thread accumulator: FP64 for double kernels; for float kernels a
// compensated (Neumaier) FP32 sum, handed to the block reduction as a
// double-float — products and per-thread sums in FP32, every cross-thread
// and cross-block addition in double-float (float kernels) or FP64.
template <typename R> struct Acc;
template <> struct Acc<double> {
  double s = 0.0;
  __device__ __forceinline__ void add(double v) { s += v; }
  __device__ __forceinline__ double get() const { return s; }
};
template <> struct Acc<float> {
  float s = 0.f, c = 0.f;
  __device__ __forceinline__ void add(float v) {
    float t = s + v;
    c += (fabsf(s) >= fabsf(v)) ? ((s - t) + v) : ((v - t) + s);
    s = t;
  }
  __device__ __forceinline__ DF df() const {
    DF r;
    two_sum_f(s, c, r.hi, r.lo);
    return r;
  }
};

// Short per-thread sum (an operator kernel's epilogue adds at most one term
// per cell of a thread's z-chunk): plain FP32 for float kernels.
template <typename R> struct ShortAcc;
template <> struct ShortAcc<double> {
  double s = 0.0;
  __device__ __forceinline__ void add(double v) { s += v; }
  __device__ __forceinline__ double get() const { return s; }
};
template <> struct ShortAcc<float> {
  float s = 0.f;
  __device__ __forceinline__ void add(float v) { s += v; }
  __device__ __forceinline__ DF df() const { return DF{s, 0.f}; }
};

// The same where a thread owns RW rows: a plane's terms are summed first, so
// that the chain has one term per plane as with one row per thread (added row
// by row, its FP32 error was 1.3 to 1.9 times as large: random data, 4 to 32
// planes).
template <typename R, int RW>
struct RowAcc {
  ShortAcc<R> acc;
  R p = R(0);
  __device__ __forceinline__ void add(int r, R v) {
    if constexpr (RW == 1) acc.add(v);
    else p = r == 0 ? v : p + v;
  }
  __device__ __forceinline__ void end_plane() {
    if constexpr (RW > 1) {
      acc.add(p);
      p = R(0);
    }
  }
};

// Grid sums a0 = a0r + i·a0i and a1 (real) of a reducing kernel, then the
// solver's scalar step `mode` in the last block (the accumulators'
// precision picks the FP64 or the double-float path).
template <int NT, typename A, typename B>
__device__ inline void sum_finalise(const A &a0r, const A &a0i, const B &a1, RedBuf red, int mode, KScalars *sc) {
  if constexpr (sizeof(a0r.s) == 4)
    block_reduce_finalise_df<NT>(a0r.df(), a0i.df(), a1.df(), DF{0.f, 0.f}, red, mode, sc);
  else
    block_reduce_finalise<NT>(make_double2(a0r.get(), a0i.get()), make_double2(a1.get(), 0.0), red, mode, sc);
}
template <int NT, typename A>
__device__ inline void sum_finalise(const A &a0r, const A &a0i, RedBuf red, int mode, KScalars *sc) {
  if constexpr (sizeof(a0r.s) == 4)
    block_reduce_finalise_df<NT>(a0r.df(), a0i.df(), DF{0.f, 0.f}, DF{0.f, 0.f}, red, mode, sc);
  else
    block_reduce_finalise<NT>(make_double2(a0r.get(), a0i.get()), make_double2(0.0, 0.0), red, mode, sc);
}

// Programmatic dependent launch: a kernel lets the next one in the stream
// start its prologue early (launch_dependents) and waits for the previous
// kernel's results to be complete and visible (wait) before reading them.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Launch with programmatic stream serialisation (when h->pdl): the kernel
// may begin while its predecessor in the stream is finishing; the kernel's
// own pdl_wait() orders its reads.  Recorded as programmatic edges when the
// stream is being captured into a CUDA graph.
template <typename... KArgs, typename... Args>
inline cudaError_t launch_k(const fdfd_handle *h, void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem,
                            Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = h->stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = h->pdl ? at : nullptr;
  cfg.numAttrs = h->pdl ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kern, args...);
}

}  // namespace fdfd
