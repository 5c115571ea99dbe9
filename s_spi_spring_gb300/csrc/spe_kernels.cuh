// Fused row / column pass kernels of the phase-retrieval iteration.
//
// Layout in HBM: the population is P individuals of N x N complex64
// (interleaved re/im, x fastest, i = x + y*N), individual p at offset p*N*N.
// A 2D transform is a row pass (transforms along x, a few rows per CTA) and
// a column pass (transforms along y, 16 columns per CTA).  One iteration of
// HIO / RAAR / ER is
//   column pass: T -> FFT+ (y) -> masked modulus projection -> FFT- (y) -> T
//   row pass:    T -> FFT- (x) -> /N^2 -> support update with rho, S -> rho
//                  -> FFT+ (x) -> T
// so the iterate rho and the half-transformed scratch T are each read and
// written once per iteration, with every FFT stage, the projection and the
// update fused into the two passes.
#pragma once
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <type_traits>

#include "spe_fft.cuh"
#include "spe_internal.h"

namespace spe {

enum { AX_ROWS = 0, AX_COLS = 1 };

// per-CTA partial results: NRED doubles per CTA (sums in fixed order later)
constexpr int NRED = 4;

// ---------------------------------------------------------------------------
// point operations shared by the ops
// ---------------------------------------------------------------------------

// Phase gate of apply_support_* (reference gpu_context.cu:526-530):
// out <=> atan2(y, x) > hi or atan2(y, x) < -lo, where the reference compares
// the float atan2 against the double (1-real)*M_PI; the host passes the
// largest floats not above those doubles, so the float comparison takes the
// same decision.  atan2 costs ~30 instructions; the cross product of the
// point with the boundary ray, D = cos(T)|y| - sin(T) x, decides
// |arg| > T whenever |D| > 4e-6 (|x|+|y|) -- an angle margin far above the
// rounding of atan2f and of the thresholds -- and only points inside that
// narrow band take the atan2f comparison.
using GateK = Gate;  // hi, lo: float thresholds; chi/shi, clo/slo: their cos and sin

__device__ __forceinline__ bool phase_out(float2 v, const GateK& g) {
  const float ay = fabsf(v.y);
  // zeros (most of a density outside its object): arg = +-0 for x = +0, +-pi
  // for x = -0, without the arc tangent's slow path
  if (v.x == 0.f && ay == 0.f) {
    const float ph = copysignf(signbit(v.x) ? 3.14159265358979f : 0.f, v.y);
    return (ph > g.hi) || (ph < -g.lo);
  }
  const bool up = !(v.y < 0.f);  // y = +0 belongs to the upper half plane (atan2(+0, x) >= 0)
  const float c = up ? g.chi : g.clo;
  const float s = up ? g.shi : g.slo;
  const float D = fmaf(c, ay, -s * v.x);
  const float band = 4e-6f * (fabsf(v.x) + ay);
  if (D > band) return true;
  if (D < -band) return false;
  const float ph = atan2f(v.y, v.x);
  return (ph > g.hi) || (ph < -g.lo);
}

// Masked modulus projection P_M (reference sub_intensities,
// gpu_context.cu:79-111).  a >= 0: known amplitude; a < -1.5: upper bound
// -a-2; otherwise unknown.  The known-amplitude rescale a/|F| uses the
// hardware reciprocal square root (2 ulp; the reference is built with
// --use_fast_math and divides approximately as well).
__device__ __forceinline__ float2 project(float2 F, float a) {
  const float m2 = fmaf(F.x, F.x, F.y * F.y);  // explicit: the paired kernels round the same way
  if (a >= 0.f) {
    if (m2 > 0.f) {
      const float s = a * rsqrtf(m2);
      return make_float2(F.x * s, F.y * s);
    }
    float sn, cs;
    sincosf(atan2f(F.y, F.x), &sn, &cs);
    return make_float2(a * cs, a * sn);
  }
  if (a < -1.5f) {
    const float b = -a - 2.f;
    const float m = sqrtf(m2);
    if (m > b) {
      const float s = __fdiv_rn(b, m);
      return make_float2(F.x * s, F.y * s);
    }
  }
  return F;
}

// (sqrtf takes its slow path for an argument of 0, which most pixels outside
// an object are)
__device__ __forceinline__ float cabsf2(float2 v) {
  const float m2 = v.y * v.y + v.x * v.x;
  const float m = sqrtf(m2 == 0.f ? 1.f : m2);
  return m2 == 0.f ? 0.f : m;
}

// ---------------------------------------------------------------------------
// block reduction of NRED values per CTA into partials[slot*NRED + k]
// (k < NSUM: sums, k >= NSUM: maxima)
//
// A warp's floats are added exactly, as integers: three 22-bit digits of each,
// counted from the largest value's exponent (66 bits: nothing that a double
// would keep is left out), and one warp-wide integer reduction a digit.  The warps'
// sums are then doubles.  A double add takes the SM 16 cycles a warp: with five
// per value and warp in a shuffle tree those were a third of the loss's column
// pass (104 us at 512^2 x 64, 70 of them the pass itself) and 40% of the error
// metrics'; here one warp per value converts the warps' sums side by side.
// (Pairs of floats, 48 bits: errors up to 2.5e-14 of a sum whose terms span six
// decades, where doubles' are 4e-16 and these nothing; loss and gradient 1024^2
// x 32 313 us against 323 here, ten refinement steps 512^2 x 64 1320 against
// 1339, evaluation 512^2 x 64 473 against 476.)
// ---------------------------------------------------------------------------
// a += b as a pair of floats, high part and rounding error (Knuth's two-sum)
__device__ __forceinline__ void add_pair(float& hi, float& lo, float b) {
  const float s = __fadd_rn(hi, b), t = __fsub_rn(s, hi);
  lo = __fadd_rn(lo, __fadd_rn(__fsub_rn(hi, __fsub_rn(s, t)), __fsub_rn(b, t)));
  hi = s;
}
// digits of the sum in x, y, z, the exponent field of the largest value in w;
// w = 255: not finite, x the float sum
__device__ __forceinline__ int4 warp_sum(float v) {
  const unsigned most = __reduce_max_sync(0xffffffffu, __float_as_uint(fabsf(v)));
  if (most >= 0x7f800000u) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    return make_int4(__float_as_int(v), 0, 0, 255);
  }
  // |v| < 2^(w - 126): |x| < 2^22 (w >= 24: the scale is a float).  x + M holds
  // the nearest whole number to x in its last bits; the rest is exact.
  const int w = max((int)(most >> 23), 24);
  constexpr float M = 12582912.f;  // 1.5 * 2^23, bits 0x4b400000
  auto digit = [&](float& x) {
    const float t = __fadd_rn(x, M);
    x = __fmul_rn(__fsub_rn(x, __fsub_rn(t, M)), 4194304.f);
    return __reduce_add_sync(0xffffffffu, __float_as_int(t) - 0x4b400000);
  };
  float x = __fmul_rn(v, __int_as_float((275 - w) << 23));
  int4 s;
  s.x = digit(x);
  s.y = digit(x);
  s.z = digit(x);
  s.w = w;
  return s;
}
__device__ __forceinline__ double warp_sum_value(int4 s) {
  if (s.w == 255) return (double)__int_as_float(s.x);
  // whole numbers below 2^51, exact, through the last bits of 1.5 * 2^52
  auto whole = [](long long i) { return __longlong_as_double(i + 0x4338000000000000ll) - 6755399441055744.0; };
  const double v = fma(whole(s.z), 1.0 / 4194304, whole((long long)s.x * 4194304 + s.y));
  return v * __hiloint2double((s.w - 170 + 1023) << 20, 0);  // v in units of 2^(w - 170)
}
// nt: threads of the CTA (whole warps, at most MOST); low: null, or (LOW) what
// the threads' sums v lack
template <int MOST, int NSUM, int NMAX, bool LOW = false>
__device__ __forceinline__ void block_reduce_store(double* __restrict__ partials, size_t slot, const float (&v)[NRED],
                                                   int nt = MOST, const float* low = nullptr) {
  static_assert(NSUM + NMAX <= NRED, "too many reduction values");
  __shared__ int4 sums[NSUM > 0 ? NSUM * (LOW ? 2 : 1) : 1][MOST / 32];
  __shared__ float top[NMAX > 0 ? NMAX : 1][MOST / 32];
  const int t = threadIdx.x, lane = t & 31, wid = t >> 5, nw = nt / 32;
#pragma unroll
  for (int k = 0; k < NSUM; ++k) {
    const int4 s = warp_sum(v[k]);
    if (lane == 0) sums[k][wid] = s;
    if (LOW) {
      const int4 l = warp_sum(low[k]);
      if (lane == 0) sums[NSUM + k][wid] = l;
    }
  }
#pragma unroll
  for (int k = 0; k < NMAX; ++k) {
    float m = v[NSUM + k];
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) m = fmaxf(m, __shfl_down_sync(0xffffffffu, m, off));
    if (lane == 0) top[k][wid] = m;
  }
  __syncthreads();
  for (int k = wid; k < NSUM; k += nw) {
    double a = lane < nw ? warp_sum_value(sums[k][lane]) : 0.0;
    if (LOW && lane < nw) a += warp_sum_value(sums[NSUM + k][lane]);
#pragma unroll
    for (int off = MOST > 512 ? 16 : MOST > 256 ? 8 : MOST > 128 ? 4 : 2; off > 0; off >>= 1)
      a += __shfl_down_sync(0xffffffffu, a, off);
    if (lane == 0) partials[slot * NRED + k] = a;
  }
  if (t < NMAX) {
    float m = top[t][0];
    for (int w = 1; w < nw; ++w) m = fmaxf(m, top[t][w]);
    partials[slot * NRED + NSUM + t] = m;
  }
}
// block argmax of (value, raster index): larger value wins, ties go to the
// lower index; writes partials[blockIdx.x*NRED + {0,1}] = {value, index}
template <int NT, bool ANY = false>
__device__ __forceinline__ void block_argmax_store(double* __restrict__ partials, float mx, int idx) {
  constexpr int NW = NT / 32;
  __shared__ float rv[NW > 0 ? NW : 1];
  __shared__ int ri[NW > 0 ? NW : 1];
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
    const float ov = __shfl_down_sync(0xffffffffu, mx, off);
    const int oi = __shfl_down_sync(0xffffffffu, idx, off);
    if (ov > mx || (ov == mx && oi < idx)) {
      mx = ov;
      idx = oi;
    }
  }
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) {
    rv[wid] = mx;
    ri[wid] = idx;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    float m = rv[0];
    int i = ri[0];
    for (int w = 1; w < (ANY ? (int)blockDim.x / 32 : NW); ++w) {
      if (rv[w] > m || (rv[w] == m && ri[w] < i)) {
        m = rv[w];
        i = ri[w];
      }
    }
    partials[(size_t)blockIdx.x * NRED + 0] = m;
    partials[(size_t)blockIdx.x * NRED + 1] = (double)i;
  }
}

// Programmatic dependent launch: a kernel launched with the programmatic
// stream serialisation attribute may start while the previous kernel of the
// stream drains.  It lets its own dependents start early, loads what no
// kernel writes (the twiddle tables), then waits until the previous grid has
// completed and its writes are visible before touching the population.
// Without the attribute both instructions are no-ops.
__device__ __forceinline__ void pdl_enter() {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// ---------------------------------------------------------------------------
// the pass kernel
//
// Row pass (AXIS == AX_ROWS): a CTA owns W consecutive rows of one
// individual; thread t handles row c = t / TPT, positions x = elem_pos(e, j)
// with j = t % TPT, so each warp reads and writes 256-byte row segments.
// Column pass: a CTA owns W consecutive columns; thread t handles column
// c = t % W, positions y = elem_pos(e, j) with j = t / W, so a warp covers
// W-element row segments of consecutive rows.
// ---------------------------------------------------------------------------
template <int N, int AXIS>
struct PassCfg {
  static constexpr int W = (AXIS == AX_ROWS) ? TileW<N>::rows : TileW<N>::cols;
  static constexpr int TPT = Plan<N>::TPT;
  static constexpr int NT = W * TPT;
  static constexpr int E = Elems<N>::value;
  static constexpr int TWN = (TwiddleTable<N>::size() + 1) & ~1;
  using Lay = typename std::conditional<AXIS == AX_ROWS, LayPad<N, W>, LaySwz<N, W>>::type;
  static constexpr size_t SMEM = (size_t)(TWN + Lay::SIZE) * sizeof(float2);
  // resident CTAs per SM the register allocation must allow: the register
  // budget per thread grows with the elements a thread holds
  static constexpr int REGS = (E <= 8) ? 64 : (E <= 16 ? 96 : 128);
  static constexpr int MINB_RAW = 65536 / (NT * REGS);
  static constexpr int MINB = MINB_RAW < 1 ? 1 : (MINB_RAW > 4 ? 4 : MINB_RAW);
};

// A pixel as an op sees it: gi, its offset in the row-major arrays (density,
// support, magnitudes); ti, its offset in the scratch arrays that only
// passes touch (equal to gi, or in the blocked order of spe_blocked.cuh); a,
// the per-pixel operand of an op with AMP (amplitude, or band weight),
// which the pass loads.
struct Px {
  size_t gi, ti;
  float a;
  int p, y, x;
};

// An op over a thread's E elements held in registers: load, transform,
// pointwise step, transform, store.  px(e): the pixel of element e; fft(v,
// sign, nth): the tile's first or second transform (std::integral_constants).
template <int N, int E, class Lay, class Op, class PxF, class Fft>
__device__ __forceinline__ void pass_elements(const Op& op, const PxF& px, typename Op::Acc& acc, const Fft& fft) {
  using First = std::integral_constant<int, 0>;
  using Second = std::integral_constant<int, 1>;
  float2 v[E];
  if constexpr (Op::PAIR) {
    float2 u[E];
    if constexpr (Op::FETCH) {
      typename Op::Raw r[E];
#pragma unroll
      for (int e = 0; e < E; ++e) r[e] = op.fetch(px(e));
#pragma unroll
      for (int e = 0; e < E; ++e) op.form_pair(r[e], v[e], u[e], acc);
    } else {
#pragma unroll
      for (int e = 0; e < E; ++e) op.load_pair(px(e), v[e], u[e], acc);
    }
    fft(v, std::integral_constant<int, Op::FFT1>(), First());
#pragma unroll
    for (int e = 0; e < E; ++e) op.store_pair(v[e], px(e), 0);
    fft(u, std::integral_constant<int, Op::FFT1>(), Second());
#pragma unroll
    for (int e = 0; e < E; ++e) op.store_pair(u[e], px(e), 1);
  } else {
    if constexpr (Op::FETCH) {
      typename Op::Raw r[E];
#pragma unroll
      for (int e = 0; e < E; ++e) r[e] = op.fetch(px(e));
#pragma unroll
      for (int e = 0; e < E; ++e) v[e] = op.form(r[e], px(e), acc);
    } else {
#pragma unroll
      for (int e = 0; e < E; ++e) v[e] = op.load(px(e), acc);
    }
    if constexpr (Op::FFT1 != 0) fft(v, std::integral_constant<int, Op::FFT1>(), First());
    if constexpr (Op::FFT2 != 0) {
#pragma unroll
      for (int e = 0; e < E; ++e) v[e] = op.mid(v[e], px(e), op.fetch_mid(px(e)), acc);
      fft(v, std::integral_constant<int, Op::FFT2>(), Second());
    }
    if constexpr (Op::FETCH_STORE) {
      typename Op::Raw r[E];
#pragma unroll
      for (int e = 0; e < E; ++e) r[e] = op.fetch_store(px(e));
#pragma unroll
      for (int e = 0; e < E; ++e) op.store(v[e], px(e), r[e]);
    } else {
#pragma unroll
      for (int e = 0; e < E; ++e) op.store(v[e], px(e), acc);
    }
  }
}

template <int N, int AXIS, class Op>
__global__ void __launch_bounds__(PassCfg<N, AXIS>::NT, PassCfg<N, AXIS>::MINB)
    pass_kernel(const Op op, const float2* __restrict__ twg) {
  using C = PassCfg<N, AXIS>;
  constexpr int W = C::W, TPT = C::TPT, NT = C::NT, E = C::E;
  extern __shared__ float2 smem[];
  float2* tw = smem;
  float2* buf = smem + C::TWN;
  constexpr int TWS = TwiddleTable<N>::size();
  pdl_enter();
  for (int i = threadIdx.x; i < TWS; i += NT) tw[i] = twg[i];

  const int t = threadIdx.x;
  const int c = (AXIS == AX_ROWS) ? t / TPT : t % W;
  const int j = (AXIS == AX_ROWS) ? t % TPT : t / W;
  constexpr int TPI = N / W;  // tiles per individual
  const int p = op.first + blockIdx.x / TPI;
  const int fixed = (blockIdx.x % TPI) * W + c;  // row (row pass) or column (column pass)
  const size_t base = (size_t)p * N * N;
  typename Op::Acc acc;
  pdl_wait();
  auto px = [&](int e) {
    const int l = elem_pos<N>(e, j);
    Px q;
    q.p = p;
    q.y = (AXIS == AX_ROWS) ? fixed : l;
    q.x = (AXIS == AX_ROWS) ? l : fixed;
    q.gi = q.ti = base + (size_t)q.y * N + q.x;
    q.a = Op::AMP ? __ldg(op.amp(p, N) + (size_t)q.y * N + q.x) : 0.f;
    return q;
  };
  pass_elements<N, E, typename C::Lay, Op>(op, px, acc, [&](float2* v, auto sign, auto) {
    fft_reg<N, typename C::Lay, decltype(sign)::value>(v, buf, tw, c, j);
  });
  if constexpr (Op::NSUM + Op::NMAX > 0) {
    float r[NRED];
    acc.values(r);
    block_reduce_store<NT, Op::NSUM, Op::NMAX>(op.partials, blockIdx.x, r);
  }
  if constexpr (Op::PEAK) block_argmax_store<NT>(op.partials, acc.mx, acc.idx);
}

struct NoAcc {
  __device__ void values(float (&v)[NRED]) const {
#pragma unroll
    for (int k = 0; k < NRED; ++k) v[k] = 0.f;
  }
};

// ---------------------------------------------------------------------------
// ops
// ---------------------------------------------------------------------------
struct OpBase {
  static constexpr int NSUM = 0, NMAX = 0, PEAK = 0;
  static constexpr bool AMP = false;   // reads amp(): A, one n x n array per pattern
  static constexpr bool PAIR = false;  // two arrays through the pass (load_pair, store_pair)
  // load in two steps, fetch and form: for a load that computes with branches
  // (roots, the phase gate), across which a thread's memory reads are not
  // reordered -- all are issued before the first value is formed
  static constexpr bool FETCH = false;
  static constexpr bool FETCH_STORE = false;  // likewise fetch_store, then store
  // run-time sides: a thread's sums as pairs of floats (ThreadSums)
  static constexpr bool PAIRS = true;
  // likewise the operands of the pointwise step: fetch_mid, then mid
  struct Mid {};
  template <class Q>
  __device__ Mid fetch_mid(const Q&) const {
    return {};
  }
  int first = 0;
  double* partials = nullptr;
  const float* A = nullptr;
  // individuals per pattern when the engine holds several patterns (slot p
  // uses pattern p / ipp); 0: one pattern shared by all
  int ipp = 0;
  __device__ __forceinline__ const float* amp(int p, int n) const {
    return ipp > 0 ? A + (size_t)(p / ipp) * n * n : A;
  }
};
// most ops keep the value between two transforms
struct OpKeep : OpBase {
  template <class Acc>
  __device__ float2 mid(float2 v, const Px&, const Mid&, Acc&) const {
    return v;
  }
};

// Source transforms of the first row pass: rho itself, or its modulus with
// the complex sum of rho in the partials.
enum { SRC_RHO = 0, SRC_ABS_SUM = 1 };

// row pass: load rho (or its modulus) -> FFT+ (x) -> T
template <int SRC>
struct OpRowsForward : OpKeep {
  static constexpr int FFT1 = +1, FFT2 = 0;
  static constexpr int NSUM = SRC == SRC_ABS_SUM ? 2 : 0, NMAX = 0;
  const float2* rho;
  float2* T;
  struct Acc {
    float s = 0.f, t = 0.f;
    __device__ void values(float (&v)[NRED]) const {
      v[0] = s;
      v[1] = t;
      v[2] = v[3] = 0.f;
    }
  };
  static constexpr bool FETCH = SRC == SRC_ABS_SUM;
  using Raw = float2;
  __device__ float2 fetch(const Px& q) const { return rho[q.gi]; }
  __device__ float2 form(float2 v, const Px&, Acc& acc) const {
    if (SRC == SRC_ABS_SUM) {
      acc.s += v.x;
      acc.t += v.y;
      v = make_float2(cabsf2(v), 0.f);
    }
    return v;
  }
  __device__ float2 load(const Px& q, Acc& acc) const { return form(fetch(q), q, acc); }
  __device__ void store(float2 v, const Px& q, Acc&) const { T[q.ti] = v; }
};

// row pass of the evaluation: rho gated by the support (apply_support_er on a
// copy) -> FFT+ (x) -> T, its summed modulus in the partials (get_module_sum,
// gpu_context.cu:219-246), and |rho| -> FFT+ (x) -> T2, from one read of rho
struct OpRowsEvaluate : OpBase {
  static constexpr int FFT1 = +1, FFT2 = 0, NSUM = 1;
  static constexpr bool PAIR = true;
  const float2* rho;
  const int* S;
  float2 *T, *T2;
  GateK g;
  struct Acc {
    float s = 0.f;
    __device__ void values(float (&v)[NRED]) const {
      v[0] = s;
      v[1] = v[2] = v[3] = 0.f;
    }
  };
  static constexpr bool FETCH = true;
  struct Raw {
    float2 v;
    int s;
  };
  __device__ Raw fetch(const Px& q) const { return {rho[q.gi], S[q.gi]}; }
  __device__ void form_pair(const Raw& r, float2& v, float2& u, Acc& acc) const {
    u = make_float2(cabsf2(r.v), 0.f);
    const float t = r.s == 0 || phase_out(r.v, g) ? 0.f : (float)r.s;
    v = make_float2(r.v.x * t, r.v.y * t);
    acc.s += r.s == 0 || r.s == 1 ? u.x * t : cabsf2(v);
  }
  __device__ void load_pair(const Px& q, float2& v, float2& u, Acc& acc) const { form_pair(fetch(q), v, u, acc); }
  __device__ void store_pair(float2 v, const Px& q, int second) const { (second ? T2 : T)[q.ti] = v; }
};

// column pass: T -> FFT+ (y) -> P_M -> FFT- (y) -> T
struct OpColsProject : OpBase {
  static constexpr int FFT1 = +1, FFT2 = -1;
  static constexpr bool AMP = true;
  float2* T;
  using Acc = NoAcc;
  __device__ float2 load(const Px& q, Acc&) const { return T[q.ti]; }
  __device__ float2 mid(float2 v, const Px& q, const Mid&, Acc&) const { return project(v, q.a); }
  __device__ void store(float2 v, const Px& q, Acc&) const { T[q.ti] = v; }
};

// Support updates (reference apply_support_{hio,raar,er},
// gpu_context.cu:519-593).  rp: the projected iterate rho', prev: the
// previous iterate (the reference's buffer, always equal to rho).
enum { UPD_HIO = 0, UPD_RAAR = 1, UPD_ER = 2 };

template <int UPD>
__device__ __forceinline__ float2 update(float2 rp, float2 prev, int s, float beta, const GateK& g) {
  if (UPD == UPD_ER) {
    const float t = phase_out(rp, g) ? 0.f : (float)s;
    return make_float2(rp.x * t, rp.y * t);
  } else if (UPD == UPD_HIO) {
    const float t = phase_out(rp, g) ? 0.f : (float)s;
    const float u = 1.f - t;
    const float2 q = __ffma2_rn(make_float2(-beta, -beta), rp, prev);  // prev - beta rp
    return make_float2(fmaf(q.x, u, rp.x * t), fmaf(q.y, u, rp.y * t));
  } else {
    const float2 refl = make_float2(2.f * rp.x - prev.x, 2.f * rp.y - prev.y);
    if (s == 0 || phase_out(refl, g)) {
      const float k = 1.f - 2.f * beta;
      return __ffma2_rn(make_float2(beta, beta), prev, __fmul2_rn(make_float2(k, k), rp));
    }
    return rp;
  }
}

// row pass of an iteration: T -> FFT- (x) -> /N^2 -> update -> rho -> FFT+ (x) -> T
template <int UPD>
struct OpRowsIterate : OpBase {
  static constexpr int FFT1 = -1, FFT2 = +1;
  float2* T;
  float2* rho;
  const int* S;
  float scale, beta;
  GateK g;
  using Acc = NoAcc;
  __device__ float2 load(const Px& q, Acc&) const { return T[q.ti]; }
  struct Mid {
    float2 prev;
    int s;
  };
  __device__ Mid fetch_mid(const Px& q) const {
    return {(UPD == UPD_ER) ? make_float2(0.f, 0.f) : rho[q.gi], S[q.gi]};
  }
  __device__ float2 mid(float2 v, const Px& q, const Mid& m, Acc&) const {
    const float2 rp = make_float2(v.x * scale, v.y * scale);
    const float2 r = update<UPD>(rp, m.prev, m.s, beta, g);
    rho[q.gi] = r;
    return r;
  }
  __device__ void store(float2 v, const Px& q, Acc&) const { T[q.ti] = v; }
};

// last row pass of a call: T -> FFT- (x) -> /N^2 -> rho (the trailing
// modulus projection of GPU_context::HIO/RAAR/ER, gpu_context.cu:803-812)
struct OpRowsFinal : OpKeep {
  static constexpr int FFT1 = -1, FFT2 = 0;
  float2* T;
  float2* out;
  float scale;
  using Acc = NoAcc;
  __device__ float2 load(const Px& q, Acc&) const { return T[q.ti]; }
  __device__ void store(float2 v, const Px& q, Acc&) const {
    out[q.gi] = make_float2(v.x * scale, v.y * scale);
  }
};

// ---- shrink-wrap (reference GPU_context::SW/SWA, gpu_context.cu:906-1027)

// row pass: T -> FFT- (x) -> |./N^2| (get_module) -> FFT+ (x) -> T
struct OpRowsModulusForward : OpBase {
  static constexpr int FFT1 = -1, FFT2 = +1;
  float2* T;
  float scale;
  using Acc = NoAcc;
  __device__ float2 load(const Px& q, Acc&) const { return T[q.ti]; }
  __device__ float2 mid(float2 v, const Px&, const Mid&, Acc&) const {
    return make_float2(cabsf2(make_float2(v.x * scale, v.y * scale)), 0.f);
  }
  __device__ void store(float2 v, const Px& q, Acc&) const { T[q.ti] = v; }
};

// column pass: T -> FFT+ (y) -> * exp(-r^2/sigma_ft^2) (smooth_intensities,
// r measured from the corner origin) -> FFT- (y) -> T
struct OpColsBlur : OpBase {
  static constexpr int FFT1 = +1, FFT2 = -1;
  float2* T;
  int n;
  float sig2;  // sigma_ft^2
  using Acc = NoAcc;
  __device__ float2 load(const Px& q, Acc&) const { return T[q.ti]; }
  __device__ float2 mid(float2 v, const Px& q, const Mid&, Acc&) const {
    const int xx = (q.x >= n / 2) ? q.x - n : q.x;
    const int yy = (q.y >= n / 2) ? q.y - n : q.y;
    const float r2 = (float)(xx * xx + yy * yy);
    const float k = expf(-__fdiv_rn(r2, sig2));
    return make_float2(v.x * k, v.y * k);
  }
  __device__ void store(float2 v, const Px& q, Acc&) const { T[q.ti] = v; }
};

// row pass: T -> FFT- (x) -> M = |.| (float), per-CTA max (get_max_module)
struct OpRowsMagnitude : OpKeep {
  static constexpr int FFT1 = -1, FFT2 = 0, NSUM = 0, NMAX = 1;
  const float2* T;
  float* M;
  struct Acc {
    float mx = 0.f;
    __device__ void values(float (&v)[NRED]) const {
      v[0] = mx;
      v[1] = v[2] = v[3] = 0.f;
    }
  };
  __device__ float2 load(const Px& q, Acc&) const { return T[q.ti]; }
  __device__ void store(float2 v, const Px& q, Acc& acc) const {
    const float m = cabsf2(v);
    M[q.gi] = m;
    acc.mx = fmaxf(acc.mx, m);
  }
};

// ---- error metrics (reference GPU_context::get_error, gpu_context.cu:1030-1134)

// column pass on the transform of the gated density: FFT+ (y) gives F;
// accumulate sum_{A>=0} (A-|F|)^2, sum_{A>=0} A^2 and max |F|
// (get_error_gpu, get_max_module); then P_M -> FFT- (y) -> T
struct OpColsError : OpBase {
  static constexpr int FFT1 = +1, FFT2 = -1, NSUM = 2, NMAX = 1;
  static constexpr bool AMP = true;
  float2* T;
  struct Acc {
    float e = 0.f, a2 = 0.f, mx = 0.f;
    __device__ void values(float (&v)[NRED]) const {
      v[0] = e;
      v[1] = a2;
      v[2] = mx;
      v[3] = 0.f;
    }
  };
  __device__ float2 load(const Px& q, Acc&) const { return T[q.ti]; }
  __device__ float2 mid(float2 v, const Px& q, const Mid&, Acc& acc) const {
    const float m = cabsf2(v);
    acc.mx = fmaxf(acc.mx, m);
    if (q.a >= 0.f) {
      acc.a2 += q.a * q.a;
      acc.e += (q.a - m) * (q.a - m);
    }
    return project(v, q.a);
  }
  __device__ void store(float2 v, const Px& q, Acc&) const { T[q.ti] = v; }
};

// row pass: T -> FFT- (x) -> /N^2 -> real-space error terms of
// get_real_error_gpu (gpu_context.cu:386-434), including its x*xs term
struct OpRowsRealError : OpKeep {
  static constexpr int FFT1 = -1, FFT2 = 0, NSUM = 2, NMAX = 0;
  const float2* T;
  const int* S;
  float scale;
  struct Acc {
    float err = 0.f, nrm = 0.f;
    __device__ void values(float (&v)[NRED]) const {
      v[0] = err;
      v[1] = nrm;
      v[2] = v[3] = 0.f;
    }
  };
  __device__ float2 load(const Px& q, Acc&) const { return T[q.ti]; }
  __device__ void store(float2 v, const Px& q, Acc& acc) const {
    const float2 r = make_float2(v.x * scale, v.y * scale);
    const int s = S[q.gi];
    acc.nrm += r.y * r.y + r.x * r.x;
    // (the gated support counts where it is 0, gate or not)
    if (s == 0) {
      const float xs = r.x * 0.f, ys = r.y * 0.f;
      acc.err += (r.y - ys) * (r.y - ys) + (r.x * xs) * (r.x * xs);
    }
  }
};

// ---- cross-correlations (get_symmetry / get_shift, gpu_context.cu:1157-1463)

// Band-pass weight of multiply() (gpu_context.cu:1157-1200), squared.
__device__ __forceinline__ float bandpass2(int x, int y, int n, float minr, float maxr) {
  const float fx = (float)((x >= n / 2) ? x - n : x);
  const float fy = (float)((y >= n / 2) ? y - n : y);
  const float radius = sqrtf(fx * fx + fy * fy);
  const float sigtot = (float)((double)n * (double)minr / 2. + 1e-12);
  const float sig = (float)((double)sigtot / 10.);
  const float eff = radius - (sigtot - sig);
  float coeff = eff > 0.f ? 1.f - expf(-__fdiv_rn(eff * eff, sig * sig)) : 0.f;
  const float sigtotm = (float)((double)n * (double)maxr / 2. + 1e-12);
  const float sigm = (float)((double)sigtotm / 10.);
  const float effm = radius - (sigtotm - sigm);
  const float coeffm = effm > 0.f ? expf(-__fdiv_rn(effm * effm, sigm * sigm)) : 1.f;
  coeff *= coeffm;
  return coeff * coeff;
}

// The operand of the correlation ops: the weight above, or -1 where A < 0
// (those pixels are left out).  One table per pattern and call: evaluated per
// pixel of every individual, the two exponentials and four divisions made the
// cross-power pass 2.4 times as long as its transform (154 against 65 us at
// 512^2 x 64).
__device__ __forceinline__ float band_weight(float a, int x, int y, int n, float minr, float maxr) {
  return a < 0.f ? -1.f : bandpass2(x, y, n, minr, maxr);
}
__device__ __forceinline__ float2 weighted(float2 c, float w) {
  return w < 0.f ? make_float2(0.f, 0.f) : make_float2(c.x * w, c.y * w);
}

// normalize_ft_shift with exponent 1 (gpu_context.cu:37-50): identity, NaN
// where |D| == 0 (the float root of a sum of squares is 0 only where the sum is).
__device__ __forceinline__ float2 ft_shift_norm(float2 d) {
  if (d.y * d.y + d.x * d.x == 0.f) {
    const float q = __int_as_float(0x7fffffff);
    return make_float2(q, q);
  }
  return d;
}

// band[pattern][y][x] = band_weight of A, row-major
static __global__ void k_band_table(const float* __restrict__ A, float* __restrict__ band, int n, size_t total,
                                    float minr, float maxr) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
    const int pix = (int)(i % ((size_t)n * n));
    band[i] = band_weight(A[i], pix % n, pix / n, n, minr, maxr);
  }
}
static cudaError_t launch_band_table(const float* A, float* band, int n, int npatterns, float minr, float maxr,
                                     cudaStream_t st) {
  k_band_table<<<152 * 8, 256, 0, st>>>(A, band, n, (size_t)npatterns * n * n, minr, maxr);
  return cudaGetLastError();
}

// conj(d) r (SIGN = -1) or d r (SIGN = +1)
template <int SIGN>
__device__ __forceinline__ float2 cross_power(float2 d, float2 r) {
  const float sd = (float)SIGN * d.y;
  return make_float2(d.x * r.x - sd * r.y, d.x * r.y + sd * r.x);
}

// column pass of the symmetry metric: T = FFT(|rho|) along x -> FFT+ (y) = D
// -> D D w -> FFT- (y) -> T, and the sum of |D|^2 w in the partials.  The
// peak of |FFT-(conj(D) D w)|^2 needs no transform: its input is real and not
// negative, so the largest value is the one at the origin, the squared sum.
struct OpColsSymmetry : OpBase {
  static constexpr int FFT1 = +1, FFT2 = -1, NSUM = 1;
  static constexpr bool AMP = true;
  float2* T;
  struct Acc {
    float s = 0.f;
    __device__ void values(float (&v)[NRED]) const {
      v[0] = s;
      v[1] = v[2] = v[3] = 0.f;
    }
  };
  __device__ float2 load(const Px& q, Acc&) const { return T[q.ti]; }
  __device__ float2 mid(float2 v, const Px& q, const Mid&, Acc& acc) const {
    const float2 d = ft_shift_norm(v);
    acc.s += weighted(make_float2(d.y * d.y + d.x * d.x, 0.f), q.a).x;
    return weighted(cross_power<+1>(d, d), q.a);
  }
  __device__ void store(float2 v, const Px& q, Acc&) const { T[q.ti] = v; }
};

// row pass: T -> FFT- (x) -> |.|^2; per-CTA max and the raster index of its
// first occurrence (encoded as a double-precision pair: value, index)
struct OpRowsPeak : OpKeep {
  static constexpr int FFT1 = -1, FFT2 = 0, PEAK = 1;
  const float2* T;
  int n;
  struct Acc {
    float mx = 0.f;
    int idx = 0x7fffffff;
    __device__ void values(float (&v)[NRED]) const {
      v[0] = v[1] = v[2] = v[3] = 0.f;
    }
  };
  __device__ float2 load(const Px& q, Acc&) const { return T[q.ti]; }
  __device__ void store(float2 v, const Px& q, Acc& a) const {
    const float val = v.x * v.x + v.y * v.y;
    const int i = q.y * n + q.x;
    // strict '>' in raster order keeps the first maximum; NaN never wins
    if (val > a.mx || (val == a.mx && val > 0.f && i < a.idx)) {
      a.mx = val;
      a.idx = i;
    }
  }
};

// column pass on the row-transformed starting density: FFT+ (y) gives F;
// sum over known pixels of |F|^2 and of A^2 (Initialize_rec's scaling,
// src/solver.cpp:938-947); nothing is stored
struct OpColsKnownPower : OpKeep {
  static constexpr int FFT1 = +1, FFT2 = 0, NSUM = 2, NMAX = 0;
  static constexpr bool AMP = true;
  const float2* T;
  struct Acc {
    float f2 = 0.f, a2 = 0.f;
    __device__ void values(float (&v)[NRED]) const {
      v[0] = f2;
      v[1] = a2;
      v[2] = v[3] = 0.f;
    }
  };
  __device__ float2 load(const Px& q, Acc&) const { return T[q.ti]; }
  __device__ void store(float2 v, const Px& q, Acc& acc) const {
    if (q.a >= 0.f) {
      acc.f2 += v.x * v.x + v.y * v.y;
      acc.a2 += q.a * q.a;
    }
  }
};

// ---- far-field loss and its adjoint (gradient refinement; no reference
// counterpart).  F = FFT+(S rho) (the transform of the iteration).  Over the
// known pixels (A >= 0):
//   amplitude: L = sum (|F| - A)^2,            dL/dconj(F) = (|F| - A) F/|F|
//   Poisson:   L = sum |F|^2 - A^2 log(|F|^2 + eps), dL/dconj(F) = (1 - A^2/(|F|^2+eps)) F
// The gradient in the convention of complex autograd (2 dL/dconj(z), the
// steepest-ascent direction) is G = 2 S FFT-(dL/dconj(F)) (FFT- is the
// adjoint of FFT+; no normalisation).
enum { LOSS_AMPLITUDE = 0, LOSS_POISSON = 1 };

// adds the loss term to `sum`; *g: 2 dL/dconj(F) (roundings spelled out, so that
// every kernel's sums have the same bits)
template <int LOSS>
__device__ __forceinline__ void loss_term(float2 F, float a, float eps, float& sum, float2* g) {
  const float m2 = fmaf(F.x, F.x, __fmul_rn(F.y, F.y));
  if (LOSS == LOSS_AMPLITUDE) {
    const float m = sqrtf(m2);
    const float d = m - a;
    const float f = m > 0.f ? 2.f * d / m : 0.f;
    if (g) *g = make_float2(f * F.x, f * F.y);
    sum = fmaf(d, d, sum);
  } else {
    // the hardware logarithm and reciprocal (a few ulp) instead of the
    // IEEE-rounded logf and division: the loss and the gradient stay within
    // the errors stated against the FP64 oracle, at a third of the
    // instructions of this term
    const float i = __fmul_rn(a, a);
    const float den = __fadd_rn(m2, eps);
    const float f = 2.f * (1.f - __fdividef(i, den));
    if (g) *g = make_float2(f * F.x, f * F.y);
    sum = __fadd_rn(sum, fmaf(-i, __logf(den), m2));
  }
}

// row pass: S rho -> FFT+ (x) -> T
struct OpRowsSupportForward : OpKeep {
  static constexpr int FFT1 = +1, FFT2 = 0;
  const float2* rho;
  const int* S;
  float2* T;
  using Acc = NoAcc;
  __device__ float2 load(const Px& q, Acc&) const {
    return S[q.gi] > 0 ? rho[q.gi] : make_float2(0.f, 0.f);
  }
  __device__ void store(float2 v, const Px& q, Acc&) const { T[q.ti] = v; }
};

// column pass: T -> FFT+ (y) = F -> loss terms; with GRAD, -> 2 dL/dconj(F)
// -> FFT- (y) -> T
template <int LOSS, bool GRAD>
struct OpColsLoss : OpBase {
  static constexpr bool PAIRS = false;  // (on the plain plan a thread's share does not change)
  static constexpr int FFT1 = +1, FFT2 = GRAD ? -1 : 0, NSUM = 1, NMAX = 0;
  static constexpr bool AMP = true;
  float2* T;
  float eps;
  struct Acc {
    float l = 0.f;
    __device__ void values(float (&v)[NRED]) const {
      v[0] = l;
      v[1] = v[2] = v[3] = 0.f;
    }
  };
  __device__ float2 load(const Px& q, Acc&) const { return T[q.ti]; }
  __device__ float2 mid(float2 v, const Px& q, const Mid&, Acc& acc) const {
    float2 g = make_float2(0.f, 0.f);
    if (q.a >= 0.f) loss_term<LOSS>(v, q.a, eps, acc.l, &g);
    return g;
  }
  __device__ void store(float2 v, const Px& q, Acc& acc) const {
    if (GRAD) {
      T[q.ti] = v;
    } else if (q.a >= 0.f) {
      loss_term<LOSS>(v, q.a, eps, acc.l, nullptr);
    }
  }
};

// row pass: T -> FFT- (x) -> G = scale[p] * S * (.)
struct OpRowsGradOut : OpKeep {
  static constexpr int FFT1 = -1, FFT2 = 0;
  const float2* T;
  const int* S;
  float2* G;
  const float* scale;  // per item (upstream gradient), or null for 1
  using Acc = NoAcc;
  __device__ float2 load(const Px& q, Acc&) const { return T[q.ti]; }
  __device__ void store(float2 v, const Px& q, Acc&) const {
    const float f = S[q.gi] > 0 ? (scale ? scale[q.p - first] : 1.f) : 0.f;
    G[q.gi] = make_float2(v.x * f, v.y * f);
  }
};

// row pass: T -> FFT- (x) = the gradient G (inside the support) -> one Adam
// step on the item's density, per real component, with the moments m, v:
//   m += (1 - b1) (G - m);  v = b2 v + (1 - b2) G^2
//   rho -= step_size * m / (sqrt(v) / sqrt_bc2 + eps)
// (step_size = lr / (1 - b1^t), sqrt_bc2 = sqrt(1 - b2^t): torch.optim.Adam
// without weight decay, complex parameters as pairs of reals)
struct AdamParams {
  float b1, b2, step_size, inv_sqrt_bc2, eps;
  // one real component: moments mm, vv and parameter p after gradient g
  // (roundings spelled out: every kernel's step has the same bits)
  __device__ __forceinline__ float upd(float g, float& mm, float& vv, float p) const {
    mm = fmaf(1.f - b1, __fsub_rn(g, mm), mm);
    vv = fmaf(vv, b2, __fmul_rn(__fmul_rn(1.f - b2, g), g));
    const float den = fmaf(sqrtf(vv), inv_sqrt_bc2, eps);
    return fmaf(-step_size, mm / den, p);
  }
  // a complex pixel: gradient g (zeroed outside the support s)
  __device__ __forceinline__ void step(float2 g, int s, float2& mm, float2& vv, float2& p) const {
    if (s <= 0) g = make_float2(0.f, 0.f);
    p.x = upd(g.x, mm.x, vv.x, p.x);
    p.y = upd(g.y, mm.y, vv.y, p.y);
  }
};

struct OpRowsGradAdam : OpKeep {
  static constexpr int FFT1 = -1, FFT2 = 0;
  const float2* T;
  const int* S;
  float2* rho;
  float2* m;
  float2* v;
  AdamParams ap;
  using Acc = NoAcc;
  __device__ float2 load(const Px& q, Acc&) const { return T[q.ti]; }
  __device__ void store(float2 g, const Px& q, Acc&) const {
    float2 mm = m[q.gi], vv = v[q.gi], p = rho[q.gi];
    ap.step(g, S[q.gi], mm, vv, p);
    m[q.gi] = mm;
    v[q.gi] = vv;
    rho[q.gi] = p;
  }
};

// ---- generic 2D transforms on arrays of items (item p at offset p*N*N)

// column pass: src -> FFT(S) (y) -> dst
template <int S>
struct OpColsTransform : OpKeep {
  static constexpr int FFT1 = S, FFT2 = 0;
  const float2* src;
  float2* dst;
  using Acc = NoAcc;
  __device__ float2 load(const Px& q, Acc&) const { return src[q.ti]; }
  __device__ void store(float2 v, const Px& q, Acc&) const { dst[q.ti] = v; }
};

// column pass: src -> FFT+ (y) -> |.| -> M (float)
struct OpColsMagnitude : OpKeep {
  static constexpr int FFT1 = +1, FFT2 = 0;
  const float2* src;
  float* M;
  using Acc = NoAcc;
  __device__ float2 load(const Px& q, Acc&) const { return src[q.ti]; }
  __device__ void store(float2 v, const Px& q, Acc&) const { M[q.gi] = cabsf2(v); }
};

// column pass over pairs: item p forms the band-passed cross-power spectra of
// D[xi[p]] with Dref[ri[p]] -- conj(D) Dref and D Dref (multiply() of
// gpu_context.cu:1157-1200), zero where A < 0 -- then FFT- (y) -> dst[p] and
// dst2[p].  Items are numbered from 0 (first == 0).  Both products are formed
// from one read of the spectra.
struct OpColsCrossPower : OpBase {
  static constexpr int FFT1 = -1, FFT2 = 0;
  static constexpr bool AMP = true, PAIR = true;
  const float2* D;
  const float2* Dref;
  const int* xi;
  const int* ri;
  float2* dst;
  float2* dst2;
  size_t npix;
  int norm_d, norm_ref;  // apply normalize_ft_shift
  using Acc = NoAcc;
  __device__ void load_pair(const Px& q, float2& c1, float2& c2, Acc&) const {
    const size_t pix = q.ti - (size_t)q.p * npix;
    float2 d = D[(size_t)__ldg(xi + q.p) * npix + pix];
    float2 r = Dref[(size_t)__ldg(ri + q.p) * npix + pix];
    if (norm_d) d = ft_shift_norm(d);
    if (norm_ref) r = ft_shift_norm(r);
    c1 = weighted(cross_power<-1>(d, r), q.a);
    c2 = weighted(cross_power<+1>(d, r), q.a);
  }
  __device__ void store_pair(float2 v, const Px& q, int second) const { (second ? dst2 : dst)[q.ti] = v; }
};

// ---- crossover (reference cross_density / cross_density_real /
// cross_support, gpu_context.cu:1699-1883; the gathered parents of
// prepare_parents / reshift_parent, 1536-1694)

// (read-only loads: one read of the item serves a thread's pixels, whatever is
// stored in between)
__device__ __forceinline__ ShiftItem load_item(const ShiftItem* p) {
  static_assert(sizeof(ShiftItem) == 48, "three 16-byte reads");
  union {
    int4 v[3];
    ShiftItem it;
  } u;
#pragma unroll
  for (int i = 0; i < 3; ++i) u.v[i] = __ldg(reinterpret_cast<const int4*>(p) + i);
  return u.it;
}

// source pixel (row-major offset) of destination pixel (x, y)
__device__ __forceinline__ int shift_source(const ShiftItem& it, int x, int y, int n) {
  if (!it.polar) return y * n + x;
  int ix = (it.flip ? n - 1 - x : x) - it.sx, iy = (it.flip ? n - 1 - y : y) - it.sy;
  if (ix < 0) ix += n;
  if (ix >= n) ix -= n;
  if (iy < 0) iy += n;
  if (iy >= n) iy -= n;
  return iy * n + ix;
}
// modulus kept, phase (mirrored by the flip) + the item's: a rotation
__device__ __forceinline__ float2 shift_value(const ShiftItem& it, float2 v) {
  if (!it.polar) return v;
  const float y = it.flip ? -v.y : v.y;
  return make_float2(fmaf(v.x, it.pc, -y * it.ps), fmaf(v.x, it.ps, y * it.pc));
}

// whether pixel (ix, iy) of child c comes from the crossed parents
__device__ __forceinline__ bool cross_pixel(int ix, int iy, int n, const CrossChild& c, int crosssym,
                                            const int* __restrict__ cmaps, int cmap_total) {
  int x = ix, y = iy;
  if (x >= n / 2) x -= n;
  if (y >= n / 2) y -= n;
  float radius = sqrtf((float)(x * x + y * y));
  if ((double)radius >= n / 2.) radius = (float)(n / 2 - 1);
  float angle = atan2f((float)y, (float)x);
  if (crosssym && angle < 0.f) angle = (float)((double)angle + 3.14159265358979323846);
  angle += c.rot;
  float sn, cs;
  sincosf(angle, &sn, &cs);
  x = (int)(cs * radius) + n / 2;
  y = (int)(sn * radius) + n / 2;
  const int cx = (x + c.ox) / c.ssx;
  const int cy = (y + c.oy) / c.ssy;
  const int cell = cx + cy * c.csx;
  const bool inside = cx >= 0 && cy >= 0 && cx < c.csx && cy < c.csy && c.cmap + cell < cmap_total;
  return inside && cmaps[c.cmap + cell] == 1;
}

// parent 1 at an unmeasured pixel of Fourier space, pulled towards the average
// (avgmod: the averaged modulus, amod: the modulus of the averaged density)
__device__ __forceinline__ float2 cross_average(float2 d1, float avgmod, float amod, float use_average) {
  const float mod1 = sqrtf(d1.x * d1.x + d1.y * d1.y);
  if (use_average > 0.f) {
    const float avg = (float)((double)(avgmod + amod) * 0.5);
    const float newmod = (float)((double)(avg * use_average) + (1. - (double)use_average) * (double)mod1);
    if (mod1 > 0.f) {
      const float r = newmod / mod1;
      d1 = make_float2(d1.x * r, d1.y * r);
    }
  } else if (use_average < 0.f && mod1 > 0.f) {
    const float loc = fabsf(use_average);
    const float maxmod = avgmod, minmod = amod;
    float newmod = mod1;
    if (newmod < minmod)
      newmod = (float)((double)(minmod * loc) + (double)newmod * (1. - (double)loc));
    else if (newmod > maxmod)
      newmod = (float)((double)(maxmod * loc) + (double)newmod * (1. - (double)loc));
    const float r = newmod / mod1;
    d1 = make_float2(d1.x * r, d1.y * r);
  }
  return d1;
}

// a child's new support S_new = [S1 + S2' S3' S' > 0.5] and its operands
struct ChildSupport {
  int s1, a, b, c, self;
};
__device__ __forceinline__ ChildSupport child_support(const CrossArgs& a, const CrossChild* c, size_t npix, size_t i) {
  const int* ws = a.Ws + (size_t)__ldg(&c->w) * 3 * npix + i;
  return {a.S[(size_t)__ldg(&c->p1) * npix + i], ws[0], ws[npix], ws[2 * npix],
          a.update_support ? 0 : a.S[(size_t)__ldg(&c->self) * npix + i]};
}
// child -> its population slot: apply_support_er with the new support
// (gpu_context.cu:2114); the support from the crossover or the parent's own
__device__ __forceinline__ void child_store(const CrossArgs& a, const CrossChild* c, size_t npix, size_t i, float2 v,
                                            const ChildSupport& r, const GateK& g) {
  const int s = r.s1 + r.b * r.c * r.a > 0 ? 1 : 0;
  const float t = s == 0 || phase_out(v, g) ? 0.f : 1.f;
  const size_t d = (size_t)__ldg(&c->dst) * npix + i;
  a.rho_out[d] = make_float2(v.x * t, v.y * t);
  a.S_out[d] = a.update_support ? s : r.self;
}

// last row pass of a Fourier-space child: C[w] -> FFT- (x) -> /N^2 -> slot
struct OpRowsChild : OpKeep {
  static constexpr int FFT1 = -1, FFT2 = 0;
  static constexpr bool FETCH_STORE = true;
  CrossArgs a;
  size_t npix;
  float scale;
  GateK g;
  using Acc = NoAcc;
  using Raw = ChildSupport;
  __device__ float2 load(const Px& q, Acc&) const { return a.C[q.ti]; }
  __device__ Raw fetch_store(const Px& q) const {
    return child_support(a, a.children + q.p, npix, q.gi - (size_t)q.p * npix);
  }
  __device__ void store(float2 v, const Px& q, const Raw& r) const {
    child_store(a, a.children + q.p, npix, q.gi - (size_t)q.p * npix, make_float2(v.x * scale, v.y * scale), r, g);
  }
};

}  // namespace spe
