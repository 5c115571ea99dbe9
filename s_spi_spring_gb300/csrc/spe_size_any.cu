// Pattern sides without a compiled plan: the same operations as the
// size-specialised units (spe_sizes.cuh), with the side a run-time value.
//
// The reference plans any side with cuFFT (cufftPlan2d(n, n),
// src/gpu/gpu_context.h:29), and its front end produces arbitrary sides:
// the pattern is cropped to max(shape) by default and may be rescaled to any
// size (spring/pattern_manager.py:61-84) -- the reference's own example
// patterns of 1054 x 1024 become 1054 x 1054.  Sides with a compiled plan
// (16 ... 2048, spe_sizes.cuh) keep their register-resident kernels; every
// other side runs here.
//
// One pass kernel serves every operation: a CTA holds W whole lines (rows or
// columns) of one individual in shared memory, applies the operation's load,
// transforms, pointwise step and store (the same op functors as the
// compiled passes), and reduces its partial sums.  The 1D transform is a
// self-sorting Stockham FFT over the factors of the side (2 .. 10, as few as
// make up the side, then the larger primes), with the twiddles of a table
// exp(2 pi i m / n) computed in double and held in shared memory.  Radices 2
// to 10 run as butterflies in registers (a thread reads the R inputs of one butterfly,
// applies its twiddles and the radix-R DFT, writes R outputs), and so do the
// primes 11 .. 31, with the symmetric form of the prime DFT; a larger prime
// radix, up to the side itself, runs the same symmetric form with run-time
// R over shared memory (about R real multiply-adds per point).  Sides are
// limited only by their lines fitting in shared memory (n <= 9386).
#include <algorithm>
#include <map>
#include <memory>
#include <mutex>

#include "spe_radices.h"
#include "spe_sizes.cuh"

namespace spe {
namespace {

constexpr int kAnyThreads = 512;     // most threads of a pass CTA
constexpr int kAnyThreadsBig = 256;  // the same for plans with a prime radix of 11 or more (128 registers each)

constexpr size_t kAnySmem = 220 * 1024;  // shared-memory budget of one CTA (two line buffers)

struct AnyPlan {
  int n;                  // side
  int W;                  // lines per CTA
  int LS;                 // shared-memory stride of a line (odd: conflict-free 8-byte columns)
  int nrad;               // radix passes
  int rad[kMaxRadices];   // radices in pass order
  int threads;            // of a CTA
  int big;                // a prime radix of 11 or more (any_pass_prime, any_pass_sym: the BIG kernels)
  // divisors of the index arithmetic as fast-division constants (fdiv):
  // the side, and per pass the butterflies per line n / R and the stride NS of
  // the pass's outputs
  unsigned inv_n;
  int ns[kMaxRadices];
  unsigned inv_m[kMaxRadices], inv_ns[kMaxRadices];
};

// x / d as one multiply-high, inv = ceil(2^32 / d) (0 encodes d = 1).  Exact
// for x < 2^17 and d < 2^15: with x = q d + s and inv d = 2^32 + r, r < d,
// x inv / 2^32 = q + (s + x r / 2^32) / d, and s + x r / 2^32 < d.  Every
// index divided here is below W n < 2^17 (make_plan narrows W to that).
__host__ __device__ constexpr unsigned fdiv_inv(int d) { return d <= 1 ? 0u : 0xFFFFFFFFu / (unsigned)d + 1u; }
__device__ __forceinline__ int fdiv(int x, unsigned inv) { return inv ? (int)__umulhi((unsigned)x, inv) : x; }

// The symmetric form of an odd prime DFT (spelled out before any_pass_prime), in
// place on R registers: (R-1)^2 real multiply-adds instead of the direct
// sums' 4 (R-1)^2.
template <int R, int S, int Q, int RR>
__device__ __forceinline__ void sym_terms(const float2* a, const float2* b, float2& A, float2& B) {
  if constexpr (RR <= (R - 1) / 2) {
    constexpr float c = float(ct_cos_frac(RR * Q, R));
    constexpr float s = float(S * ct_sin_frac(RR * Q, R));
    A.x = fmaf(a[RR - 1].x, c, A.x);
    A.y = fmaf(a[RR - 1].y, c, A.y);
    B.x = fmaf(b[RR - 1].x, s, B.x);
    B.y = fmaf(b[RR - 1].y, s, B.y);
    sym_terms<R, S, Q, RR + 1>(a, b, A, B);
  }
}
template <int R, int S, int Q>
__device__ __forceinline__ void sym_outputs(const float2* a, const float2* b, float2 x0, float2* v) {
  if constexpr (Q <= (R - 1) / 2) {
    float2 A = x0, B = make_float2(0.f, 0.f);
    sym_terms<R, S, Q, 1>(a, b, A, B);
    v[Q] = make_float2(A.x - B.y, A.y + B.x);
    v[R - Q] = make_float2(A.x + B.y, A.y - B.x);
    sym_outputs<R, S, Q + 1>(a, b, x0, v);
  }
}
template <int R, int S>
__device__ __forceinline__ void dft_odd_sym(float2* v) {
  constexpr int H = (R - 1) / 2;
  float2 a[H], b[H];
  const float2 x0 = v[0];
  float2 sum = x0;
#pragma unroll
  for (int r = 1; r <= H; ++r) {
    a[r - 1] = cadd(v[r], v[R - r]);
    b[r - 1] = csub(v[r], v[R - r]);
    sum = cadd(sum, a[r - 1]);
  }
  v[0] = sum;
  sym_outputs<R, S, 1>(a, b, x0, v);
}

// 6 and 10: with SPLIT by the prime-factor algorithm (Good, Thomas): n = Q n1 + 2
// n2 and k = Q k1 + (Q + 1) k2 mod R = 2 Q make the transform one of 2 by one of
// Q with no twiddles between them, so that a plan of few large radices rounds no
// more than one of 2, 3, 4, 5 and 8: over 18 sides from 54 to 1200 the rms error
// of a transform is 0.98 of that plan's on average (0.90 at 100, 0.93 at 1000,
// 1.06 at 54 and 270, which have a 9 as well); with twiddles inside 6 and 10 it was
// 1.03 (1.07 at 1000, 1.12 at 54).  Without SPLIT, beside a prime radix of 11 or
// more, whose pass is most of the error: twiddles, the same to the bit as one
// pass of 2 and one of Q.
template <int R, int S, bool SPLIT>
__device__ __forceinline__ void small_dft(float2* v) {
  if constexpr (R == 5 || R == 7) {
    dft_odd_sym<R, S>(v);
  } else if constexpr (SPLIT ? R == 6 || R == 10 : R == 10) {  // (dft has no factor 5)
    constexpr int Q = R / 2;
    float2 y[R];
#pragma unroll
    for (int n2 = 0; n2 < Q; ++n2) {
      const int i = SPLIT ? 2 * n2 : n2, j = SPLIT ? (Q + 2 * n2) % R : Q + n2;
      y[2 * n2] = cadd(v[i], v[j]);
      y[2 * n2 + 1] = csub(v[i], v[j]);
    }
    if constexpr (!SPLIT) twiddle_block<R, 2, Q, S, 1>(y);
#pragma unroll
    for (int k1 = 0; k1 < 2; ++k1) {
      float2 t[Q];
#pragma unroll
      for (int n2 = 0; n2 < Q; ++n2) t[n2] = y[n2 * 2 + k1];
      if constexpr (Q == 3) dft<3, S>(t);
      else dft_odd_sym<Q, S>(t);
#pragma unroll
      for (int k2 = 0; k2 < Q; ++k2) v[SPLIT ? (Q * k1 + (Q + 1) * k2) % R : k1 + 2 * k2] = t[k2];
    }
  } else {
    dft<R, S>(v);
  }
}

// The dynamic shared memory of pass_any: two line buffers and the side's
// twiddle table.  The pass functions below are not inlined (one copy of each
// serves every operation's kernel) and take offsets into it, not pointers, so
// that their accesses are shared-memory accesses, and the plan's values they
// need by value.
extern __shared__ float2 sm_any[];

struct PassArgs {  // one pass of the plan
  int cur, oth, tw;  // offsets of the line buffers and the table in sm_any
  int nl, n, LS, NS;
  unsigned inv_m, inv_ns;
};

// One Stockham pass of radix R as butterflies: each thread reads the R
// inputs x[b + r n/R] of a butterfly, multiplies them by w_{NS R}^{k r}
// (k = b mod NS), runs the radix-R DFT in registers and writes its R
// outputs at (b/NS) NS R + k + q NS.
template <int R, int S, bool BIG>
__device__ __noinline__ void any_pass_r(const PassArgs a) {
  const float2* cur = sm_any + a.cur;
  float2* oth = sm_any + a.oth;
  const float2* tw = sm_any + a.tw;
  const int n = a.n, LS = a.LS, m = n / R, NS = a.NS, tstep = n / (NS * R);
  const int total = a.nl * m;
  for (int i = threadIdx.x; i < total; i += blockDim.x) {
    const int c = fdiv(i, a.inv_m), b = i - c * m;
    const int bq = fdiv(b, a.inv_ns), k = b - bq * NS;
    const float2* src = cur + c * LS + b;
    float2 v[R];
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = src[r * m];
    if (NS > 1) {
      const int e = k * tstep;  // < n / R
      int idx = 0;
#pragma unroll
      for (int r = 1; r < R; ++r) {
        idx += e;
        float2 w = tw[idx];
        if (S < 0) w.y = -w.y;
        v[r] = cmul(v[r], w);
      }
    }
    small_dft<R, S, !BIG>(v);
    float2* dst = oth + c * LS + bq * NS * R + k;
#pragma unroll
    for (int q = 0; q < R; ++q) dst[q * NS] = v[q];
  }
}

// Radix-R DFT of an odd prime R in its symmetric form (the terms r and R-r
// paired): with a_r = x_r + x_{R-r}, b_r = x_r - x_{R-r}, r = 1 .. (R-1)/2,
//   X_0 = x_0 + sum_r a_r,
//   X_q = A_q + i B_q,  X_{R-q} = A_q - i B_q,  q = 1 .. (R-1)/2,
//   A_q = x_0 + sum_r a_r cos(2 pi r q / R),  B_q = sum_r b_r S sin(2 pi r q / R),
// with the cosines and sines compile-time constants: (R-1)^2 real
// multiply-adds for the R outputs, against 4 (R-1)^2 for the direct sums.
// Output q goes to dst[q * NS] as soon as it is formed, so only the a_r,
// b_r and one output pair are live.
template <int R, int S, int Q>
__device__ __forceinline__ void odd_sym_outputs(const float2* a, const float2* b, float2 x0, float2* dst, int NS) {
  if constexpr (Q <= (R - 1) / 2) {
    float2 A = x0, B = make_float2(0.f, 0.f);
    sym_terms<R, S, Q, 1>(a, b, A, B);
    dst[Q * NS] = make_float2(A.x - B.y, A.y + B.x);
    dst[(R - Q) * NS] = make_float2(A.x + B.y, A.y - B.x);
    odd_sym_outputs<R, S, Q + 1>(a, b, x0, dst, NS);
  }
}

// One Stockham pass of an odd prime radix R (11 .. 31) as butterflies: the
// inputs and twiddles of any_pass_r, the symmetric DFT above.  Not inlined:
// one copy per (R, S) serves every operation's pass kernel.
template <int R, int S>
__device__ __noinline__ void any_pass_prime(const PassArgs a) {
  constexpr int H = (R - 1) / 2;
  const float2* cur = sm_any + a.cur;
  float2* oth = sm_any + a.oth;
  const float2* tw = sm_any + a.tw;
  const int nl = a.nl, n = a.n, LS = a.LS, m = n / R, NS = a.NS, tstep = n / (NS * R);
  const unsigned inv_m = a.inv_m, inv_ns = a.inv_ns;
  for (int i = threadIdx.x; i < nl * m; i += blockDim.x) {
    const int c = fdiv(i, inv_m), b = i - c * m;
    const int bq = fdiv(b, inv_ns), k = b - bq * NS;
    const float2* src = cur + c * LS + b;
    float2 v[R];
#pragma unroll
    for (int r = 0; r < R; ++r) v[r] = src[r * m];
    if (NS > 1) {
      const int e = k * tstep;  // < n / R
      int idx = 0;
#pragma unroll
      for (int r = 1; r < R; ++r) {
        idx += e;
        float2 w = tw[idx];
        if (S < 0) w.y = -w.y;
        v[r] = cmul(v[r], w);
      }
    }
    float2 sa[H], sb[H];
    float2 x0 = v[0], sum = v[0];
#pragma unroll
    for (int r = 1; r <= H; ++r) {
      sa[r - 1] = cadd(v[r], v[R - r]);
      sb[r - 1] = csub(v[r], v[R - r]);
      sum = cadd(sum, sa[r - 1]);
    }
    float2* dst = oth + c * LS + bq * NS * R + k;
    dst[0] = sum;
    odd_sym_outputs<R, S, 1>(sa, sb, x0, dst, NS);
  }
}

// Outputs of a symmetric pass (step 2 of any_pass_sym): kSymQ values of q for
// BB butterflies per thread, so that each a_r, b_r read serves kSymQ pairs and
// each table read BB butterflies; the multiply-adds of a pair's x and y are one
// packed instruction.  Consecutive threads take consecutive butterflies of one
// group of q: their table reads coincide and their inputs are contiguous.
// q = 0 takes the table's exp(0) = 1 exactly: X_0 = y_0 + sum a_r.
constexpr int kSymQ = 4;
template <int S, int BB>
__device__ __forceinline__ void any_sym_outputs(const PassArgs& a, int R) {
  constexpr int QB = kSymQ;
  const float2* cur = sm_any + a.cur;
  float2* oth = sm_any + a.oth;
  const float2* tw = sm_any + a.tw;
  const int n = a.n, LS = a.LS, NS = a.NS, H = (R - 1) / 2, m = n / R;
  const int G = (H + QB) / QB, nb = a.nl * m, ng = (nb + BB - 1) / BB;
  const unsigned inv_ng = fdiv_inv(ng);
  for (int i = threadIdx.x; i < ng * G; i += blockDim.x) {
    const int g = fdiv(i, inv_ng), up = i - g * ng;
    const float2* src[BB];
    float2* dst[BB];
    float2 A[BB][QB], B[BB][QB];
    bool live[BB];
#pragma unroll
    for (int v = 0; v < BB; ++v) {
      const int u0 = up + v * ng;
      live[v] = u0 < nb;
      const int u = live[v] ? u0 : up;  // a tail slot repeats the first butterfly, unstored
      const int c = fdiv(u, a.inv_m), b = u - c * m;
      const int bq = fdiv(b, a.inv_ns), k = b - bq * NS;
      src[v] = cur + c * LS + b;
      dst[v] = oth + c * LS + bq * NS * R + k;
#pragma unroll
      for (int t = 0; t < QB; ++t) {
        A[v][t] = src[v][0];
        B[v][t] = make_float2(0.f, 0.f);
      }
    }
    int idx[QB], step[QB];
#pragma unroll
    for (int t = 0; t < QB; ++t) {
      const int q = g * QB + t;
      idx[t] = 0;
      step[t] = q <= H ? q * m : 0;  // table index of exp(2 pi i r q / R) advances by q m mod n
    }
    for (int r = 1; r <= H; ++r) {
      float2 x[BB], y[BB];
#pragma unroll
      for (int v = 0; v < BB; ++v) {
        x[v] = src[v][r * m];
        y[v] = src[v][(R - r) * m];
      }
#pragma unroll
      for (int t = 0; t < QB; ++t) {
        idx[t] += step[t];
        if (idx[t] >= n) idx[t] -= n;
        const float2 w = tw[idx[t]];
        const float ws = S < 0 ? -w.y : w.y;
        const float2 cc = make_float2(w.x, w.x), ss = make_float2(ws, ws);
#pragma unroll
        for (int v = 0; v < BB; ++v) {
          A[v][t] = __ffma2_rn(x[v], cc, A[v][t]);
          B[v][t] = __ffma2_rn(y[v], ss, B[v][t]);
        }
      }
    }
#pragma unroll
    for (int v = 0; v < BB; ++v) {
      if (!live[v]) continue;
#pragma unroll
      for (int t = 0; t < QB; ++t) {
        const int q = g * QB + t;
        if (q == 0) {
          dst[v][0] = A[v][t];
        } else if (q <= H) {
          dst[v][q * NS] = make_float2(A[v][t].x - B[v][t].y, A[v][t].y + B[v][t].x);
          dst[v][(R - q) * NS] = make_float2(A[v][t].x + B[v][t].y, A[v][t].y - B[v][t].x);
        }
      }
    }
  }
}

// Butterflies per thread of any_sym_outputs (first: 1, 2 or 4) for nb butterflies
// and G groups of q, by the warps each of an SM's four schedulers gets and a
// warp's instructions per term (kSymQ table reads and their index steps, and
// per butterfly two reads and 2 kSymQ multiply-adds), and their product (second).
struct SymRounds {
  int first, second;
};
__host__ __device__ __forceinline__ SymRounds sym_rounds(int nb, int G) {
  const int c1 = (nb * G + 127) / 128 * 34, c2 = ((nb + 1) / 2 * G + 127) / 128 * 44,
            c4 = ((nb + 3) / 4 * G + 127) / 128 * 64;
  return c4 <= c2 && c4 <= c1 ? SymRounds{4, c4} : c2 <= c1 ? SymRounds{2, c2} : SymRounds{1, c1};
}

// One pass of an odd prime radix above 31, in the symmetric form of the
// prime DFT with run-time R (H = (R-1)/2), in two steps over shared memory:
//   1. per butterfly and pair (r, R-r), r = 1 .. H: y_r = x_r w^{k r},
//      y_{R-r} = x_{R-r} w^{k (R-r)} (the inter-pass twiddles), then
//      a_r = y_r + y_{R-r} into slot r and b_r = y_r - y_{R-r} into slot R-r,
//      in place (each element is read and written by one thread);
//   2. per butterfly and q = 0 .. H: X_0 = y_0 + sum a_r, and for q >= 1
//      X_q, X_{R-q} = A_q +- i B_q with A_q = y_0 + sum_r a_r cos(2 pi r q / R),
//      B_q = sum_r b_r S sin(2 pi r q / R), the cosines and sines read from
//      the side's table (exp(2 pi i t m / n) = exp(2 pi i t / R), m = n / R).
// About 2 real multiply-adds per input and output pair instead of 4 per
// input and output.
template <int S>
__device__ __noinline__ void any_pass_sym(const PassArgs a, int R) {
  float2* cur = sm_any + a.cur;
  const float2* tw = sm_any + a.tw;
  const int nl = a.nl, n = a.n, LS = a.LS, NS = a.NS, H = (R - 1) / 2;
  const int m = n / R, tstep = n / (NS * R);
  const unsigned inv_m = a.inv_m, inv_ns = a.inv_ns;
  const unsigned inv_h = fdiv_inv(H);
  // 1. twiddles and pairs, in place
  for (int i = threadIdx.x; i < nl * m * H; i += blockDim.x) {
    const int u = fdiv(i, inv_h), r = 1 + (i - u * H);  // u: butterfly of the tile
    const int c = fdiv(u, inv_m), b = u - c * m;
    const int k = b - fdiv(b, inv_ns) * NS;
    float2* src = cur + c * LS + b;
    float2 x = src[r * m], y = src[(R - r) * m];
    if (NS > 1) {
      const int e = k * tstep;  // w^{k r} = table[e r]; e < n / R, so e r < n
      float2 w1 = tw[e * r], w2 = tw[e * (R - r)];
      if (S < 0) {
        w1.y = -w1.y;
        w2.y = -w2.y;
      }
      x = cmul(x, w1);
      y = cmul(y, w2);
    }
    src[r * m] = cadd(x, y);
    src[(R - r) * m] = csub(x, y);
  }
  __syncthreads();
  // 2. output pairs
  const int bb = sym_rounds(nl * m, (H + kSymQ) / kSymQ).first;
  if (bb == 4) any_sym_outputs<S, 4>(a, R);
  else if (bb == 2) any_sym_outputs<S, 2>(a, R);
  else any_sym_outputs<S, 1>(a, R);
}

// The transform of the tile's nl lines: one pass per radix of the plan,
// ping-ponging between the two line buffers; on return `cur` holds it.
// BIG: the plan has a prime radix of 11 or more, whose pass functions need
// more registers than the rest; kernels without them are compiled
// separately so that the other sides keep their occupancy.
template <int S, bool BIG>
__device__ __forceinline__ void fft_any(float2*& cur, float2*& oth, const AnyPlan& pl, const float2* tw, int nl) {
  for (int ps = 0; ps < pl.nrad; ++ps) {
    const int R = pl.rad[ps];
    const PassArgs a{(int)(cur - sm_any), (int)(oth - sm_any), (int)(tw - sm_any), nl, pl.n, pl.LS, pl.ns[ps],
                     pl.inv_m[ps], pl.inv_ns[ps]};
    switch (R) {
      case 2: any_pass_r<2, S, BIG>(a); break;
      case 3: any_pass_r<3, S, BIG>(a); break;
      case 4: any_pass_r<4, S, BIG>(a); break;
      case 5: any_pass_r<5, S, BIG>(a); break;
      case 6: any_pass_r<6, S, BIG>(a); break;
      case 7: any_pass_r<7, S, BIG>(a); break;
      case 8: any_pass_r<8, S, BIG>(a); break;
      case 9: any_pass_r<9, S, BIG>(a); break;
      case 10: any_pass_r<10, S, BIG>(a); break;
      default:
        if constexpr (BIG) {
          switch (R) {
            case 11: any_pass_prime<11, S>(a); break;
            case 13: any_pass_prime<13, S>(a); break;
            case 17: any_pass_prime<17, S>(a); break;
            case 19: any_pass_prime<19, S>(a); break;
            case 23: any_pass_prime<23, S>(a); break;
            case 29: any_pass_prime<29, S>(a); break;
            case 31: any_pass_prime<31, S>(a); break;
            default: any_pass_sym<S>(a, R); break;
          }
        }
        // (kernels without BIG never see a radix of 11 or more: make_plan
        // sends every such plan to the BIG kernels)
        break;
    }
    __syncthreads();
    float2* t = cur;
    cur = oth;
    oth = t;
  }
}

// A thread's sums and maxima.  It may have tens of terms here (a tile of up to 32
// lines over as few as 64 threads, where the compiled passes have 4 to 16), so
// each is added to a pair of floats: the sum does not lose by the tile's shape.
template <class Op>
struct ThreadSums {
  static constexpr bool PAIRS = Op::PAIRS && Op::NSUM > 0;
  typename Op::Acc acc;
  float v[NRED] = {}, low[NRED] = {};
  // f(the accumulator of one element)
  template <class F>
  __device__ __forceinline__ auto element(const F& f) {
    if constexpr (PAIRS) {
      struct Fold {
        ThreadSums& s;
        typename Op::Acc one;
        __device__ __forceinline__ ~Fold() {
          float r[NRED];
          one.values(r);
#pragma unroll
          for (int k = 0; k < Op::NSUM; ++k) add_pair(s.v[k], s.low[k], r[k]);
#pragma unroll
          for (int k = Op::NSUM; k < Op::NSUM + Op::NMAX; ++k) s.v[k] = fmaxf(s.v[k], r[k]);
        }
      } fold{*this, {}};
      return f(fold.one);
    } else {
      return f(acc);
    }
  }
  __device__ __forceinline__ void finish() {
    if constexpr (PAIRS) {
#pragma unroll
      for (int k = 0; k < Op::NSUM; ++k)
        if (!isfinite(v[k])) low[k] = 0.f;  // (the error of an overflowed sum is not a number)
    } else {
      acc.values(v);
    }
  }
};

template <int AXIS, class Op, bool BIG>
// BIG kernels: two 256-thread CTAs per SM, 128 registers a thread (a few
// spilled bytes; one CTA per SM without the cap ran 30% slower at side 1054)
__global__ void __launch_bounds__(BIG ? kAnyThreadsBig : kAnyThreads, 2)
    pass_any(const Op op, const AnyPlan pl, const float2* __restrict__ tw) {
  const int NT = blockDim.x;
  const int n = pl.n, W = pl.W, LS = pl.LS;
  float2* cur = sm_any;
  float2* oth = sm_any + (size_t)W * LS;
  float2* tws = sm_any + (size_t)2 * W * LS;  // the twiddle table, n entries
  pdl_enter();
  for (int i = threadIdx.x; i < n; i += blockDim.x) tws[i] = __ldg(tw + i);
  const int tpi = (n + W - 1) / W;
  const int p = op.first + blockIdx.x / tpi;
  const int l0 = (blockIdx.x % tpi) * W;
  const int nl = min(W, n - l0);
  const size_t base = (size_t)p * n * n;
  const int tot = nl * n;
  const unsigned inv_nl = fdiv_inv(nl);
  ThreadSums<Op> sums;
  using Acc = typename Op::Acc;
  // element i of the tile: row passes walk along x (whole rows), column
  // passes across the tile's columns first (row segments of nl elements)
  const float* amp = Op::AMP ? op.amp(p, n) : nullptr;
  auto px = [&](int i, int& at) {
    int c, l;
    if (AXIS == AX_ROWS) {
      c = fdiv(i, pl.inv_n);
      l = i - c * n;
    } else {
      l = fdiv(i, inv_nl);
      c = i - l * nl;
    }
    at = c * LS + l;
    Px q;
    q.p = p;
    q.y = AXIS == AX_ROWS ? l0 + c : l;
    q.x = AXIS == AX_ROWS ? l : l0 + c;
    const int off = q.y * n + q.x;
    q.gi = q.ti = base + off;
    q.a = Op::AMP ? __ldg(amp + off) : 0.f;
    return q;
  };
  // a thread's elements in batches of U: the batch's memory reads are issued
  // before the first of them is used (one at a time, the waits for them were
  // 35-45% of the iteration's passes; eight at a time is 12% slower at 600 and
  // 1000, where a thread has ten elements)
  constexpr int U = 4;
  auto batches = [&](auto&& body) {
    for (int i0 = threadIdx.x; i0 < tot; i0 += NT * U) body(i0);
  };
  pdl_wait();
  if constexpr (Op::PAIR) {
    for (int second = 0; second < 2; ++second) {
      for (int i = threadIdx.x; i < tot; i += blockDim.x) {
        int at;
        const Px q = px(i, at);
        float2 v1, v2;
        Acc once;
        if (second) op.load_pair(q, v1, v2, once);
        else sums.element([&](Acc& a) { op.load_pair(q, v1, v2, a); });
        cur[at] = second ? v2 : v1;
      }
      __syncthreads();
      fft_any<Op::FFT1, BIG>(cur, oth, pl, tws, nl);
      for (int i = threadIdx.x; i < tot; i += blockDim.x) {
        int at;
        const Px q = px(i, at);
        op.store_pair(cur[at], q, second);
      }
      __syncthreads();
    }
  } else {
    batches([&](int i0) {
      int at[U];
      if constexpr (Op::FETCH) {
        typename Op::Raw r[U];
#pragma unroll
        for (int u = 0; u < U; ++u) if (i0 + u * NT < tot) r[u] = op.fetch(px(i0 + u * NT, at[u]));
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (i0 + u * NT < tot) {
            int x;
            cur[at[u]] = sums.element([&](Acc& a) { return op.form(r[u], px(i0 + u * NT, x), a); });
          }
      } else {
        float2 v[U];
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (i0 + u * NT < tot)
            v[u] = sums.element([&](Acc& a) { return op.load(px(i0 + u * NT, at[u]), a); });
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (i0 + u * NT < tot) cur[at[u]] = v[u];
      }
    });
    __syncthreads();
    if constexpr (Op::FFT1 != 0) fft_any<Op::FFT1, BIG>(cur, oth, pl, tws, nl);
    if constexpr (Op::FFT2 != 0) {
      batches([&](int i0) {
        Px q[U];
        int at[U];
        typename Op::Mid m[U];
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (i0 + u * NT < tot) {
            q[u] = px(i0 + u * NT, at[u]);
            m[u] = op.fetch_mid(q[u]);
          }
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (i0 + u * NT < tot)
            cur[at[u]] = sums.element([&](Acc& a) { return op.mid(cur[at[u]], q[u], m[u], a); });
      });
      __syncthreads();
      fft_any<Op::FFT2, BIG>(cur, oth, pl, tws, nl);
    }
#pragma unroll 4
    for (int i = threadIdx.x; i < tot; i += blockDim.x) {
      int at;
      const Px q = px(i, at);
      sums.element([&](Acc& a) { op.store(cur[at], q, a); });
    }
  }
  if constexpr (Op::NSUM + Op::NMAX > 0) {
    sums.finish();
    block_reduce_store<BIG ? kAnyThreadsBig : kAnyThreads, Op::NSUM, Op::NMAX, ThreadSums<Op>::PAIRS>(
        op.partials, blockIdx.x, sums.v, NT, sums.low);
  }
  if constexpr (Op::PEAK) block_argmax_store<BIG ? kAnyThreadsBig : kAnyThreads, true>(op.partials, sums.acc.mx, sums.acc.idx);
}

// ---------------------------------------------------------------------------
// plans
// ---------------------------------------------------------------------------
size_t smem_of(const AnyPlan& pl) { return (2 * (size_t)pl.W * pl.LS + pl.n) * sizeof(float2); }

int largest_radix(const AnyPlan& pl) { return *std::max_element(pl.rad, pl.rad + pl.nrad); }

// Threads of a pass CTA: those that keep the most threads of an SM (as many
// CTAs as its shared memory and registers hold) busy in the pass with the
// fewest butterflies (the largest radix), the larger of equals, as they have
// more reads in flight.  A run-time prime pass spreads over its outputs too
// and takes them all.  512 threads at every side left five of six idle at 100
// (935 -> 487 us for 8 iterations of 200 individuals).
int best_threads(const AnyPlan& pl) {
  const int top = pl.big ? kAnyThreadsBig : kAnyThreads, regs = pl.big ? 512 : 1024, rmax = largest_radix(pl);
  int best = top;
  if (rmax > 31) return top;
  const int fly = pl.W * (pl.n / rmax), ctas = (int)(kAnySmem / smem_of(pl));
  double most = 0.0;
  for (int t = 64; t <= top; t += 32) {
    const int rounds = (fly + t - 1) / t;
    const double busy = (double)std::min(ctas, regs / t) * fly / rounds;
    if (busy >= most) {
      most = busy;
      best = t;
    }
  }
  return best;
}

// plain: radices 8, 4 and the primes, 8 lines and the most threads.  A
// shrink-wrap takes these radices because its support is a threshold of what
// they transform: other radices round differently, and that may flip a pixel.
// The loss and the refinement take all three: they add a thread's terms in
// floats, without ThreadSums' pairs, so that another share of the pixels would
// move a loss in its ninth digit.
bool make_plan(int n, AnyPlan& pl, bool plain) {
  if (n < 2) return false;
  pl.n = n;
  pl.nrad = 0;
  // the part of the side without prime factors above 7: by the radices 2 .. 10
  // that suit it, or (`plain`) by 8, 4 and its primes; then the larger primes
  int smooth = 1, m = n;
  for (int f : {2, 3, 5, 7})
    for (; m % f == 0; m /= f) smooth *= f;
  if (plain) {
    for (int f : {8, 4, 2, 3, 5, 7})
      for (; smooth % f == 0; smooth /= f) pl.rad[pl.nrad++] = f;
  } else {
    pl.nrad = choose_radices(n, smooth, pl.rad);
  }
  for (int f = 11; m > 1 && pl.nrad < kMaxRadices;) {
    if (m % f == 0) {
      pl.rad[pl.nrad++] = f;
      m /= f;
    } else if (f * f > m) {
      f = m;
    } else {
      f += 2;
    }
  }
  if (m != 1) return false;
  pl.big = 0;
  pl.inv_n = fdiv_inv(n);
  for (int i = 0, ns = 1; i < pl.nrad; ns *= pl.rad[i], ++i) {
    pl.big |= pl.rad[i] >= 11 ? 1 : 0;
    pl.ns[i] = ns;
    pl.inv_m[i] = fdiv_inv(n / pl.rad[i]);
    pl.inv_ns[i] = fdiv_inv(ns);
  }
  pl.LS = n | 1;
  const size_t table = (size_t)n * sizeof(float2);
  const size_t per_line = 2 * (size_t)pl.LS * sizeof(float2);
  if (table + per_line > kAnySmem) return false;
  // two CTAs per SM where half the budget still holds two lines
  const size_t budget = (table + 2 * per_line <= kAnySmem / 2) ? kAnySmem / 2 : kAnySmem;
  const size_t w = (budget - table) / per_line;
  // lines per CTA: 8, and 32 with a run-time prime, whose pass has work for its
  // threads only with many lines (8 iterations of 64 individuals of 97^2 with
  // 8 / 16 / 32 lines 713 / 640 / 473 us, 100 of 263^2 8157 / 6821 / 5454; at
  // smooth sides fewer or more lines than 8 are slower)
  pl.W = (int)std::min<size_t>(w, plain || largest_radix(pl) <= 31 ? 8 : 32);
  pl.threads = plain ? (pl.big ? kAnyThreadsBig : kAnyThreads) : best_threads(pl);
  // the bounds of fdiv: indices below W n < 2^17, divisors below 2^15
  if (n >= (1 << 15)) return false;
  while (pl.W > 1 && (size_t)pl.W * n >= (1u << 17)) --pl.W;
  return (size_t)pl.W * n < (1u << 17);
}

struct AnyEntry {
  AnyPlan plan, plain, blur;  // blur: the plain radices on the plan's tiles
  SizeOps ops;
};

std::mutex g_any_mutex;
std::map<int, std::unique_ptr<AnyEntry>> g_any;

const AnyPlan& plan_of(int n) {
  std::lock_guard<std::mutex> lock(g_any_mutex);
  return g_any.at(n)->plan;
}
const AnyPlan& blur_of(int n) {
  std::lock_guard<std::mutex> lock(g_any_mutex);
  return g_any.at(n)->blur;
}
const AnyPlan& plain_of(int n) {
  std::lock_guard<std::mutex> lock(g_any_mutex);
  return g_any.at(n)->plain;
}

// Lines per CTA of one launch.  With a run-time prime: the width with the least
// rounds of its pass over the waves of CTAs (two per SM), as that pass is most
// of the time (100 of 263^2 with 25 / 16 / 8 lines 5454 / 6821 / 8157 us).  Else the plan's, halved
// while it would leave SMs without a CTA.
int launch_width(const AnyPlan& pl, int count) {
  const int R = largest_radix(pl), sms = sm_count();
  int W = pl.W;
  if (R <= 31) {
    while (W > 2 && (size_t)count * ((pl.n + W - 1) / W) < (size_t)sms) W /= 2;
    return W;
  }
  size_t least = ~size_t(0);
  for (int half = pl.W; half >= std::min(pl.W, 4); half /= 2) {
    const size_t ctas = (size_t)count * ((pl.n + half - 1) / half), waves = (ctas + 2 * sms - 1) / (2 * sms);
    const int nb = half * (pl.n / R), G = ((R - 1) / 2 + kSymQ) / kSymQ;
    const size_t cost = waves * sym_rounds(nb, G).second;
    if (cost <= least) {  // (the narrower of equals: shorter reads and writes)
      least = cost;
      W = half;
    }
  }
  return W;
}

template <int AXIS, class Op, bool BIG>
cudaError_t launch_any_k(const Op& op, AnyPlan pl, int count, cudaStream_t st, const float2* tw) {
  auto kern = pass_any<AXIS, Op, BIG>;
  static std::atomic<unsigned long long> configured{0ull};
  // the attribute is set to the largest budget once: it is an upper bound
  cudaError_t e = configure(kern, kAnySmem, configured);
  if (e != cudaSuccess || count <= 0) return e;
  // narrower tiles where the plan's leave SMs without a CTA (not where the op
  // reduces: its partials are one per tile of the plan)
  if (Op::NSUM + Op::NMAX == 0 && !Op::PEAK) pl.W = launch_width(pl, count);
  const int tpi = (pl.n + pl.W - 1) / pl.W;
  const int grid = (int)((unsigned)count * tpi), threads = pl.threads;
  const size_t smem = smem_of(pl);
  // the early launch pays where a pass is a few waves of CTAs (a prologue
  // beside the previous pass's drain: 111 -> 82 us for an evaluation of one
  // small pattern); over many waves it measured 0.6% slower (1054^2 x 16)
  if (grid <= 4 * sm_count()) return launch_pdl(kern, grid, threads, smem, st, op, pl, tw);
  kern<<<grid, threads, smem, st>>>(op, pl, tw);
  return cudaGetLastError();
}
template <int AXIS, class Op>
cudaError_t launch_any(const Op& op, const AnyPlan& pl, int count, cudaStream_t st, const float2* tw) {
  return pl.big ? launch_any_k<AXIS, Op, true>(op, pl, count, st, tw)
                : launch_any_k<AXIS, Op, false>(op, pl, count, st, tw);
}

// ---------------------------------------------------------------------------
// the operation table (the sequences of SizeImpl, spe_sizes.cuh, on pass_any)
// ---------------------------------------------------------------------------
struct SizeAny {
  static float scale(int n) { return (float)(1.0 / ((double)n * (double)n)); }

  template <int SRC>
  static OpRowsForward<SRC> rows_forward(const Ctx& c, const float2* src, float2* dst, double* partials) {
    OpRowsForward<SRC> op;
    op.first = c.first;
    op.partials = partials;
    op.rho = src;
    op.T = dst;
    return op;
  }

  static OpColsProject cols_project(const Ctx& c) {
    OpColsProject op;
    op.first = c.first;
    op.T = c.T;
    op.A = c.A;
    op.ipp = c.ipp;
    return op;
  }

  template <int UPD>
  static cudaError_t iterate_t(const Ctx& c, int iters, float beta, Gate g) {
    const AnyPlan& pl = plan_of(c.n);
    SPE_TRY((launch_any<AX_ROWS>(rows_forward<SRC_RHO>(c, c.rho, c.T, nullptr), pl, c.count, c.st, c.tw)));
    const OpColsProject proj = cols_project(c);
    OpRowsIterate<UPD> it;
    it.first = c.first;
    it.T = c.T;
    it.rho = c.rho;
    it.S = c.S;
    it.scale = scale(c.n);
    it.beta = beta;
    it.g = g;
    for (int i = 0; i < iters; ++i) {
      SPE_TRY((launch_any<AX_COLS>(proj, pl, c.count, c.st, c.tw)));
      if (i == 0 && c.mark) SPE_TRY(cudaEventRecord(c.mark, c.st));
      SPE_TRY((launch_any<AX_ROWS>(it, pl, c.count, c.st, c.tw)));
    }
    SPE_TRY((launch_any<AX_COLS>(proj, pl, c.count, c.st, c.tw)));
    if (iters == 0 && c.mark) SPE_TRY(cudaEventRecord(c.mark, c.st));
    OpRowsFinal fin;
    fin.first = c.first;
    fin.T = c.T;
    fin.out = c.rho;
    fin.scale = scale(c.n);
    return launch_any<AX_ROWS>(fin, pl, c.count, c.st, c.tw);
  }

  // tile widths are fixed by the plan: wc / wr are ignored
  static cudaError_t iterate(const Ctx& c, int upd, int iters, float beta, Gate g, int, int) {
    switch (upd) {
      case 0: return iterate_t<UPD_HIO>(c, iters, beta, g);
      case 1: return iterate_t<UPD_RAAR>(c, iters, beta, g);
      default: return iterate_t<UPD_ER>(c, iters, beta, g);
    }
  }

  static int one_width(int* out) {
    out[0] = 0;
    return 1;
  }

  static cudaError_t blur_magnitude(const Ctx& c, float sigma_ft) {
    const AnyPlan& pl = blur_of(c.n);
    SPE_TRY((launch_any<AX_ROWS>(rows_forward<SRC_RHO>(c, c.rho, c.T, nullptr), pl, c.count, c.st, c.tw)));
    SPE_TRY((launch_any<AX_COLS>(cols_project(c), pl, c.count, c.st, c.tw)));
    OpRowsModulusForward mf;
    mf.first = c.first;
    mf.T = c.T;
    mf.scale = scale(c.n);
    SPE_TRY((launch_any<AX_ROWS>(mf, pl, c.count, c.st, c.tw)));
    OpColsBlur bl;
    bl.first = c.first;
    bl.T = c.T;
    bl.n = c.n;
    bl.sig2 = sigma_ft * sigma_ft;
    SPE_TRY((launch_any<AX_COLS>(bl, pl, c.count, c.st, c.tw)));
    OpRowsMagnitude mg;
    mg.first = c.first;
    mg.partials = c.partials;
    mg.T = c.T;
    mg.M = c.M;
    return launch_any<AX_ROWS>(mg, pl, c.count, c.st, c.tw);
  }

  static cudaError_t error_terms(const Ctx& c, Gate g, double* p1, double* p2, double* p3) {
    const AnyPlan& pl = plan_of(c.n);
    OpRowsEvaluate ev;
    ev.first = c.first;
    ev.partials = p1;
    ev.rho = c.rho;
    ev.S = c.S;
    ev.T = c.T;
    ev.T2 = c.T2;
    ev.g = g;
    SPE_TRY((launch_any<AX_ROWS>(ev, pl, c.count, c.st, c.tw)));
    OpColsError ce;
    ce.first = c.first;
    ce.partials = p2;
    ce.T = c.T;
    ce.A = c.A;
    ce.ipp = c.ipp;
    SPE_TRY((launch_any<AX_COLS>(ce, pl, c.count, c.st, c.tw)));
    OpRowsRealError re;
    re.first = c.first;
    re.partials = p3;
    re.T = c.T;
    re.S = c.S;
    re.scale = scale(c.n);
    return launch_any<AX_ROWS>(re, pl, c.count, c.st, c.tw);
  }

  static cudaError_t symmetry(const Ctx& c, double* psum, double* ppeak) {
    const AnyPlan& pl = plan_of(c.n);
    OpColsSymmetry sy;
    sy.first = c.first;
    sy.partials = psum;
    sy.T = c.T2;
    sy.A = c.band;
    sy.ipp = c.ipp;
    SPE_TRY((launch_any<AX_COLS>(sy, pl, c.count, c.st, c.tw)));
    return rows_peak(c, pl, c.T2, ppeak);
  }

  static cudaError_t rows_peak(const Ctx& c, const AnyPlan& pl, const float2* T, double* partials) {
    OpRowsPeak pk;
    pk.first = c.first;
    pk.partials = partials;
    pk.T = T;
    pk.n = c.n;
    return launch_any<AX_ROWS>(pk, pl, c.count, c.st, c.tw);
  }

  // ---- generic transforms over `c.count` items starting at `data` (c.first ignored)
  static cudaError_t fft2(const Ctx& c, float2* data, int sign) {
    const AnyPlan& pl = plan_of(c.n);
    if (sign > 0) {
      Ctx z = c;
      z.first = 0;
      SPE_TRY((launch_any<AX_ROWS>(rows_forward<SRC_RHO>(z, data, data, nullptr), pl, c.count, c.st, c.tw)));
      OpColsTransform<+1> ct;
      ct.first = 0;
      ct.src = data;
      ct.dst = data;
      return launch_any<AX_COLS>(ct, pl, c.count, c.st, c.tw);
    }
    OpColsTransform<-1> ct;
    ct.first = 0;
    ct.src = data;
    ct.dst = data;
    SPE_TRY((launch_any<AX_COLS>(ct, pl, c.count, c.st, c.tw)));
    OpRowsFinal fin;
    fin.first = 0;
    fin.T = data;
    fin.out = data;
    fin.scale = scale(c.n);
    return launch_any<AX_ROWS>(fin, pl, c.count, c.st, c.tw);
  }

  static cudaError_t ft_magnitude(const Ctx& c, const float2* src, float2* tmp, float* M) {
    const AnyPlan& pl = plan_of(c.n);
    Ctx z = c;
    z.first = 0;
    SPE_TRY((launch_any<AX_ROWS>(rows_forward<SRC_RHO>(z, src, tmp, nullptr), pl, c.count, c.st, c.tw)));
    OpColsMagnitude cm;
    cm.first = 0;
    cm.src = tmp;
    cm.M = M;
    return launch_any<AX_COLS>(cm, pl, c.count, c.st, c.tw);
  }

  static cudaError_t abs_spectrum_items(const Ctx& c, const float2* src, float2* dst, double* psum) {
    const AnyPlan& pl = plan_of(c.n);
    Ctx z = c;
    z.first = 0;
    SPE_TRY((launch_any<AX_ROWS>(rows_forward<SRC_ABS_SUM>(z, src, dst, psum), pl, c.count, c.st, c.tw)));
    OpColsTransform<+1> ct;
    ct.src = dst;
    ct.dst = dst;
    return launch_any<AX_COLS>(ct, pl, c.count, c.st, c.tw);
  }

  static cudaError_t corr_peaks(const Ctx& c, const float2* D, const float2* Dref, const int* xi, const int* ri,
                                int norm_d, int norm_ref, float2* scratch1, float2* scratch2, double* part1,
                                double* part2) {
    const AnyPlan& pl = plan_of(c.n);
    OpColsCrossPower cp;
    cp.A = c.band;
    cp.D = D;
    cp.Dref = Dref;
    cp.xi = xi;
    cp.ri = ri;
    cp.dst = scratch1;
    cp.dst2 = scratch2;
    cp.npix = (size_t)c.n * c.n;
    cp.norm_d = norm_d;
    cp.norm_ref = norm_ref;
    SPE_TRY((launch_any<AX_COLS>(cp, pl, c.count, c.st, c.tw)));
    Ctx z = c;
    z.first = 0;
    SPE_TRY(rows_peak(z, pl, scratch1, part1));
    return rows_peak(z, pl, scratch2, part2);
  }

  static cudaError_t known_power(const Ctx& c, double* partials) {
    const AnyPlan& pl = plan_of(c.n);
    SPE_TRY((launch_any<AX_ROWS>(rows_forward<SRC_RHO>(c, c.rho, c.T, nullptr), pl, c.count, c.st, c.tw)));
    OpColsKnownPower kp;
    kp.first = c.first;
    kp.partials = partials;
    kp.T = c.T;
    kp.A = c.A;
    kp.ipp = c.ipp;
    return launch_any<AX_COLS>(kp, pl, c.count, c.st, c.tw);
  }

  // far-field loss: one partial per column tile (loss_tiles = tiles_cols)
  static cudaError_t grad_rows(const Ctx& c, const AnyPlan& pl, float2* grad, const float* scale) {
    OpRowsGradOut go;
    go.first = c.first;
    go.T = c.T;
    go.S = c.S;
    go.G = grad;
    go.scale = scale;
    return launch_any<AX_ROWS>(go, pl, c.count, c.st, c.tw);
  }
  template <int LOSS>
  static cudaError_t loss_grad_t(const Ctx& c, float eps, double* partials, float2* grad, const float* scale,
                                 int stage) {
    const AnyPlan& pl = plain_of(c.n);
    if (stage == GRAD_ROWS || stage == GRAD_BACKWARD) return grad_rows(c, pl, grad, scale);
    OpRowsSupportForward rf;
    rf.first = c.first;
    rf.rho = c.rho;
    rf.S = c.S;
    rf.T = c.T;
    SPE_TRY((launch_any<AX_ROWS>(rf, pl, c.count, c.st, c.tw)));
    if (!grad && stage == GRAD_ALL) {
      OpColsLoss<LOSS, false> cl;
      cl.first = c.first;
      cl.partials = partials;
      cl.T = c.T;
      cl.A = c.A;
      cl.ipp = c.ipp;
      cl.eps = eps;
      return launch_any<AX_COLS>(cl, pl, c.count, c.st, c.tw);
    }
    OpColsLoss<LOSS, true> cl;
    cl.first = c.first;
    cl.partials = partials;
    cl.T = c.T;
    cl.A = c.A;
    cl.ipp = c.ipp;
    cl.eps = eps;
    SPE_TRY((launch_any<AX_COLS>(cl, pl, c.count, c.st, c.tw)));
    return stage == GRAD_ALL ? grad_rows(c, pl, grad, scale) : cudaSuccess;
  }

  static cudaError_t loss_grad(const Ctx& c, int loss, float eps, double* partials, float2* grad,
                               const float* scale, int stage) {
    return loss == LOSS_POISSON ? loss_grad_t<LOSS_POISSON>(c, eps, partials, grad, scale, stage)
                                : loss_grad_t<LOSS_AMPLITUDE>(c, eps, partials, grad, scale, stage);
  }

  template <int LOSS>
  static cudaError_t adam_step_t(const Ctx& c, float eps, double* partials, float2* m, float2* v,
                                 const AdamStep& a) {
    const AnyPlan& pl = plain_of(c.n);
    OpRowsSupportForward rf;
    rf.first = c.first;
    rf.rho = c.rho;
    rf.S = c.S;
    rf.T = c.T;
    SPE_TRY((launch_any<AX_ROWS>(rf, pl, c.count, c.st, c.tw)));
    OpColsLoss<LOSS, true> cl;
    cl.first = c.first;
    cl.partials = partials;
    cl.T = c.T;
    cl.A = c.A;
    cl.ipp = c.ipp;
    cl.eps = eps;
    SPE_TRY((launch_any<AX_COLS>(cl, pl, c.count, c.st, c.tw)));
    OpRowsGradAdam ad;
    ad.first = c.first;
    ad.T = c.T;
    ad.S = c.S;
    ad.rho = c.rho;
    ad.m = m;
    ad.v = v;
    ad.ap = {a.b1, a.b2, a.step_size, a.inv_sqrt_bc2, a.eps};
    return launch_any<AX_ROWS>(ad, pl, c.count, c.st, c.tw);
  }

  static cudaError_t adam_step(const Ctx& c, int loss, float eps, double* partials, float2* m, float2* v,
                               const AdamStep& a) {
    return loss == LOSS_POISSON ? adam_step_t<LOSS_POISSON>(c, eps, partials, m, v, a)
                                : adam_step_t<LOSS_AMPLITUDE>(c, eps, partials, m, v, a);
  }
};

// exp(+2 pi i m / n), m < n, double angles rounded once to float
void fill_any(float2* out, int n) {
  for (int m = 0; m < n; ++m) {
    const double a = 2.0 * kPi * (double)m / (double)n;
    out[m] = make_float2((float)cos(a), (float)sin(a));
  }
}

}  // namespace

const SizeOps* size_ops_any(int n) {
  std::lock_guard<std::mutex> lock(g_any_mutex);
  auto it = g_any.find(n);
  if (it != g_any.end()) return &it->second->ops;
  std::unique_ptr<AnyEntry> en(new AnyEntry());
  if (!make_plan(n, en->plan, false) || !make_plan(n, en->plain, true)) return nullptr;
  en->blur = en->plain;
  en->blur.W = en->plan.W;
  en->blur.threads = best_threads(en->blur);
  const int tiles = (n + en->plan.W - 1) / en->plan.W, loss_tiles = (n + en->plain.W - 1) / en->plain.W;
  en->ops = SizeOps{n,
                    tiles,
                    tiles,
                    n,
                    &fill_any,
                    &SizeAny::iterate,
                    &SizeAny::blur_magnitude,
                    &SizeAny::error_terms,
                    &SizeAny::symmetry,
                    &SizeAny::fft2,
                    &SizeAny::ft_magnitude,
                    &SizeAny::abs_spectrum_items,
                    &SizeAny::corr_peaks,
                    nullptr,
                    &launch_band_table,
                    &SizeAny::one_width,
                    &SizeAny::one_width,
                    0,
                    0,
                    &SizeAny::known_power,
                    &SizeAny::loss_grad,
                    loss_tiles,
                    &SizeAny::adam_step,
                    0,
                    0,
                    0,
                    nullptr,
                    0};
  const SizeOps* out = &en->ops;
  g_any.emplace(n, std::move(en));
  return out;
}

}  // namespace spe
