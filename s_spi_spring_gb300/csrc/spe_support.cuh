// Far-field loss, its gradient and the Adam update through the support's rows.
//
// The density enters the loss only inside its support, and the gradient
// leaves it only there, so of the scratch between the row and the column
// passes nothing but the rows that hold support is ever not zero (forward)
// or not multiplied by zero (adjoint).  A support is compact -- the object is
// a few percent of the pixels and a quarter of the rows or less (the
// oversampling that phase retrieval needs) -- so these passes skip the other
// row tiles: the forward row pass flags the tiles with support and transforms
// those, the column pass reads and writes their rows only (the others are
// zeros in registers), and the last row pass transforms those.  A support that
// fills the field runs every tile.
//
// A caller may also ask for the column-transformed gradient itself, whole and
// row-major (LossRowMajor): the forward row pass still skips, the column pass
// writes every row and the last row pass reads every row.
//
// Measured on GB300 (row-major passes over every row before -> now): a loss and
// its gradient at 1024^2 x 32 511 -> 319 us, ten refinement steps at 512^2 x 64
// 3909 -> 1325 us.  The column pass transforms every column twice and is bound
// like the iteration's (spe_blocked.cuh); the row passes by the reads of the
// int32 support.  A support over more and more rows, loss and gradient at 512^2 x
// 64: 23% 150 us, 60% 192, all 258 against 214 before; the row passes then move
// 295 MB at 3.7 TB/s, the staged persistent ones before them at 5.5.
#pragma once
#include "spe_blocked.cuh"

namespace spe {

// Scratch layout: row tiles (WR rows, the unit that is skipped) one after the
// other, inside a tile the WR x BC pixels of a column-pass CTA together.  A
// tile occupies the bytes of its rows in row-major order, so that the gradient
// may replace the scratch in place.
template <int N>
struct LossT {
  static constexpr bool WHOLE = false;  // only the flagged row tiles are written
  static constexpr int WR = Blocked<N>::WR, BC = Blocked<N>::BC;
  static constexpr int XS = WR;  // offset of a step in x that is a multiple of BC, per column
  __host__ __device__ static constexpr int at(int y, int x) {
    return (y / WR) * (WR * N) + (x / BC) * (WR * BC) + (y % WR) * BC + x % BC;
  }
};

template <int N>
struct LossRowMajor {
  static constexpr bool WHOLE = true;
  static constexpr int XS = 1;
  __host__ __device__ static constexpr int at(int y, int x) { return y * N + x; }
};

template <int N>
struct LossRows : BlkCfg<N, Blocked<N>::WR, 1> {
  using C = BlkCfg<N, Blocked<N>::WR, 1>;
  static constexpr int MINB = C::E <= 8 ? 1024 / C::NT : 2;
};
template <int N>
struct LossCols : BlkCfg<N, Blocked<N>::BC, 2> {
  using C = BlkCfg<N, Blocked<N>::BC, 2>;
  static constexpr int MINB = C::E <= 8 ? 1024 / C::NT : 2;
};

// A thread's place in a row pass: row c of the tile, position j.
template <int N, class L>
struct RowSlot {
  int c, j, tile, p;
  size_t gi, ti;  // of element 0
  __device__ __forceinline__ RowSlot(int first) {
    constexpr int W = Blocked<N>::WR, TPI = N / W;
    c = threadIdx.x % W;
    j = threadIdx.x / W;
    tile = blockIdx.x;
    p = first + tile / TPI;
    gi = ((size_t)first * N + (size_t)tile * W + c) * N + j;
    ti = ((size_t)first * N + (size_t)tile * W) * N + L::at(c, j);
  }
};

// Whether the CTA's row tile holds support: 16-byte reads (two of them per
// thread; the tiles without, most of them, read nothing else)
template <int N>
__device__ __forceinline__ bool tile_has_support(const int* __restrict__ S, int first, int tile) {
  using C = LossRows<N>;
  const int4* s4 = reinterpret_cast<const int4*>(S + ((size_t)first * N + (size_t)tile * Blocked<N>::WR) * N);
  int4 m[C::E / 4];
  int any = 0;
#pragma unroll
  for (int i = 0; i < C::E / 4; ++i) m[i] = __ldg(s4 + threadIdx.x + i * C::NT);
#pragma unroll
  for (int i = 0; i < C::E / 4; ++i) any |= m[i].x > 0 || m[i].y > 0 || m[i].z > 0 || m[i].w > 0;
  return __syncthreads_or(any) != 0;
}

// S rho -> FFT+ (x) -> T for the row tiles with support, flagged in `flags`;
// clears `bad`
template <int N, class L>
__global__ void __launch_bounds__(LossRows<N>::NT, LossRows<N>::MINB)
    k_loss_rows_in(const float2* __restrict__ rho, const int* __restrict__ S, float2* __restrict__ T,
                   unsigned char* __restrict__ flags, unsigned* __restrict__ bad, int first,
                   const float2* __restrict__ twg) {
  using C = LossRows<N>;
  constexpr int E = C::E;
  extern __shared__ __align__(128) unsigned char sm[];
  float2* tw = reinterpret_cast<float2*>(sm);
  float2* xb = reinterpret_cast<float2*>(sm + C::TWB);
  pdl_enter();
  pdl_wait();
  const RowSlot<N, L> q(first);
  const bool any = tile_has_support<N>(S, first, q.tile);
  if (threadIdx.x == 0) {
    flags[(size_t)first * (N / Blocked<N>::WR) + q.tile] = any ? 1 : 0;
    if (bad && q.tile % (N / Blocked<N>::WR) == 0) bad[q.p] = 0u;
  }
  if (!any) return;
  int m[E];
#pragma unroll
  for (int e = 0; e < E; ++e) m[e] = __ldg(S + q.gi + C::step(e));
  float2 v[E];
#pragma unroll
  for (int e = 0; e < E; ++e) v[e] = m[e] > 0 ? __ldcg(rho + q.gi + C::step(e)) : make_float2(0.f, 0.f);
  load_twiddles<N>(tw, twg, C::NT);
  __syncthreads();
  fft_x<N, typename C::Lay, +1, 1, 0>(v, xb, tw, q.c, q.j);
#pragma unroll
  for (int e = 0; e < E; ++e) T[q.ti + (size_t)C::step(e) * L::XS] = v[e];
}

// T -> FFT+ (y) = F -> loss terms over the known pixels (one sum per tile); with
// GRAD -> 2 dL/dconj(F) -> FFT- (y) -> T.  Persistent: the flags of tile k + 2
// and the rows of tile k + 1 are read while tile k is transformed.  MARK: bad[p]
// is set where an item's result is not finite in any row, written or not: the
// row transform carries it to every pixel, and 0 times it is not a number.
template <int N, int LOSS, bool GRAD, class L, bool MARK>
__global__ void __launch_bounds__(LossCols<N>::NT, LossCols<N>::MINB)
    k_loss_cols(float2* __restrict__ T, const float* __restrict__ At, int ipp, const unsigned char* __restrict__ flags,
                unsigned* __restrict__ bad, int first, int count, float eps, double* __restrict__ partials,
                const float2* __restrict__ twg) {
  using C = LossCols<N>;
  using Lay = typename C::Lay;
  constexpr int E = C::E, NT = C::NT, W = Blocked<N>::BC, WR = Blocked<N>::WR, TPI = N / W;
  constexpr bool PF = E <= 8;
  // two exchange buffers in turn (an even number of exchanges a tile), one
  // where only the forward transform runs
  constexpr int NX = GRAD ? 2 : 1;
  static_assert(C::TPT % WR == 0 && C::NB % WR == 0 && E <= 32, "a thread's rows are tiles apart");
  extern __shared__ __align__(128) unsigned char sm[];
  float2* tw = reinterpret_cast<float2*>(sm);
  float2* xb = reinterpret_cast<float2*>(sm + C::TWB);
  pdl_enter();
  load_twiddles<N>(tw, twg, NT);
  const int t = threadIdx.x, c = t % W, j = t / W;
  const int ntiles = count * TPI;
  pdl_wait();
  __syncthreads();
  // the thread's rows of a tile's individual that hold support, as bits
  auto rows_of = [&](int tile) {
    const unsigned char* f = flags + (size_t)(first + tile / TPI) * (N / WR) + j / WR;
    unsigned r = 0;
#pragma unroll
    for (int e = 0; e < E; ++e) r |= __ldcg(f + C::step(e) / WR) ? 1u << e : 0u;
    return r;
  };
  auto tile_ptr = [&](int tile) {
    return T + (size_t)(first + tile / TPI) * N * N + L::at(j, (tile % TPI) * W + c);
  };
  auto fetch = [&](float2* v, int tile, unsigned rows) {
    const float2* g = tile_ptr(tile);
#pragma unroll
    for (int e = 0; e < E; ++e)
      v[e] = (rows >> e) & 1u ? __ldcg(g + (size_t)C::step(e) * N) : make_float2(0.f, 0.f);
  };
  int tile = blockIdx.x;
  unsigned rows = 0, nrows = 0;
  float2 v[E], nv[PF ? E : 1];
  if (tile < ntiles) {
    rows = rows_of(tile);
    if (PF) fetch(nv, tile, rows);
    const int nxt = tile + gridDim.x;
    if (nxt < ntiles) nrows = rows_of(nxt);
  }
  for (; tile < ntiles; tile += gridDim.x) {
    const int p = first + tile / TPI, nxt = tile + gridDim.x, nn = nxt + gridDim.x;
    if (PF) {
#pragma unroll
      for (int e = 0; e < E; ++e) v[e] = nv[PF ? e : 0];
    } else {
      fetch(v, tile, rows);
    }
    const float4* A4 = reinterpret_cast<const float4*>(At + (ipp > 0 ? (size_t)(p / ipp) * N * N : 0)) +
                       (size_t)((tile % TPI) * NT + t) * (E / 4);
    float4 a4[E / 4];
#pragma unroll
    for (int i = 0; i < E / 4; ++i) a4[i] = __ldg(A4 + i);
    fft_x<N, Lay, +1, NX, 0>(v, xb, tw, c, j);
    float acc = 0.f;
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const float a = e % 4 == 0 ? a4[e / 4].x : e % 4 == 1 ? a4[e / 4].y : e % 4 == 2 ? a4[e / 4].z : a4[e / 4].w;
      float2 d = make_float2(0.f, 0.f);
      if (a >= 0.f) loss_term<LOSS>(v[e], a, eps, acc, GRAD ? &d : nullptr);
      v[e] = d;
    }
    if (PF && nxt < ntiles) fetch(nv, nxt, nrows);
    if (GRAD) {
      fft_x<N, Lay, -1, NX, C::EX>(v, xb, tw, c, j);
      float2* g = tile_ptr(tile);
#pragma unroll
      for (int e = 0; e < E; ++e)
        if (L::WHOLE || ((rows >> e) & 1u)) g[(size_t)C::step(e) * N] = v[e];
      if constexpr (MARK) {
        float chk = 0.f;
#pragma unroll
        for (int e = 0; e < E; ++e) chk += 0.f * v[e].x + 0.f * v[e].y;
        if (chk != 0.f) bad[p] = 1u;
      }
    }
    const float r[NRED] = {acc, 0.f, 0.f, 0.f};
    block_reduce_store<NT, 1, 0>(partials, tile, r);
    rows = nrows;
    if (nn < ntiles) nrows = rows_of(nn);
  }
}

// T -> FFT- (x) -> G = scale[p] * S * (.) (G may be T); the row tiles without
// support (unless T is whole) are zeros, or not a number where bad[p]
template <int N, class L>
__global__ void __launch_bounds__(LossRows<N>::NT, LossRows<N>::MINB)
    k_loss_rows_out(const float2* T, const int* __restrict__ S, float2* G, const float* __restrict__ scale,
                    const unsigned char* __restrict__ flags, const unsigned* __restrict__ bad, int first,
                    const float2* __restrict__ twg) {
  using C = LossRows<N>;
  constexpr int E = C::E;
  extern __shared__ __align__(128) unsigned char sm[];
  float2* tw = reinterpret_cast<float2*>(sm);
  float2* xb = reinterpret_cast<float2*>(sm + C::TWB);
  pdl_enter();
  pdl_wait();
  const RowSlot<N, L> q(first);
  if (!L::WHOLE && !__ldcg(flags + (size_t)first * (N / Blocked<N>::WR) + q.tile)) {
    const float f = __ldcg(bad + q.p) ? __int_as_float(0x7fffffff) : 0.f;
    float2* z = G + ((size_t)first * N + (size_t)q.tile * Blocked<N>::WR) * N;
    if ((reinterpret_cast<uintptr_t>(z) & 15u) == 0) {
#pragma unroll
      for (int i = 0; i < E / 2; ++i) reinterpret_cast<float4*>(z)[threadIdx.x + i * C::NT] = make_float4(f, f, f, f);
    } else {
#pragma unroll
      for (int i = 0; i < E; ++i) z[threadIdx.x + i * C::NT] = make_float2(f, f);
    }
    return;
  }
  float2 v[E];
  int m[E];
#pragma unroll
  for (int e = 0; e < E; ++e) v[e] = __ldcg(T + q.ti + (size_t)C::step(e) * L::XS);
#pragma unroll
  for (int e = 0; e < E; ++e) m[e] = __ldg(S + q.gi + C::step(e));
  load_twiddles<N>(tw, twg, C::NT);
  __syncthreads();
  fft_x<N, typename C::Lay, -1, 1, 0>(v, xb, tw, q.c, q.j);  // (its barriers: the tile has been read)
  const float sc = scale ? scale[q.p - first] : 1.f;
  if (L::WHOLE) {
    int any = 0;
#pragma unroll
    for (int e = 0; e < E; ++e) any |= m[e] > 0;
    if (!__syncthreads_or(any)) {  // 0 or not a number, as above: no negative zeros
#pragma unroll
      for (int e = 0; e < E; ++e) G[q.gi + C::step(e)] = make_float2(fmaf(v[e].x, 0.f, 0.f), fmaf(v[e].y, 0.f, 0.f));
      return;
    }
  }
#pragma unroll
  for (int e = 0; e < E; ++e) {
    const float f = m[e] > 0 ? sc : 0.f;
    G[q.gi + C::step(e)] = make_float2(v[e].x * f, v[e].y * f);
  }
}

// T -> FFT- (x) = the gradient (inside the support) -> Adam step of the
// density.  OUTSIDE: the pixels outside the support too (their gradient is 0,
// their moments may not be); otherwise those hold zero moments, and the step
// leaves them as they are.  fresh: the moments are 0 and not read.  next: the
// updated density's FFT+ (x) goes to T, the next step's forward row pass.
template <int N, bool OUTSIDE>
__global__ void __launch_bounds__(LossRows<N>::NT, LossRows<N>::E <= 8 ? 768 / LossRows<N>::NT : 1)
    k_adam_rows(float2* __restrict__ T, const unsigned char* __restrict__ flags, const int* __restrict__ S,
                float2* __restrict__ rho, float2* __restrict__ m, float2* __restrict__ v, AdamParams ap, int fresh,
                int next, int first, const float2* __restrict__ twg) {
  using C = LossRows<N>;
  using Lay = typename C::Lay;
  constexpr int E = C::E;
  extern __shared__ __align__(128) unsigned char sm[];
  float2* tw = reinterpret_cast<float2*>(sm);
  float2* xb = reinterpret_cast<float2*>(sm + C::TWB);
  pdl_enter();
  pdl_wait();
  const RowSlot<N, LossT<N>> q(first);
  const bool any = __ldcg(flags + (size_t)first * (N / Blocked<N>::WR) + q.tile) != 0;
  if (!any && !OUTSIDE) return;
  int s[E];
#pragma unroll
  for (int e = 0; e < E; ++e) s[e] = __ldg(S + q.gi + C::step(e));
  float2 g[E];
  if (any) {
#pragma unroll
    for (int e = 0; e < E; ++e) g[e] = __ldcg(T + q.ti + (size_t)C::step(e) * LossT<N>::XS);
    load_twiddles<N>(tw, twg, C::NT);
    __syncthreads();
    fft_x<N, Lay, -1, 1, 0>(g, xb, tw, q.c, q.j);
  } else {
#pragma unroll
    for (int e = 0; e < E; ++e) g[e] = make_float2(0.f, 0.f);
  }
  // the operands of four pixels in flight at a time
#pragma unroll
  for (int e0 = 0; e0 < E; e0 += 4) {
    float2 p[4], mm[4], vv[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const size_t i = q.gi + C::step(e0 + k);
      p[k] = mm[k] = vv[k] = make_float2(0.f, 0.f);
      if (OUTSIDE || s[e0 + k] > 0) {
        p[k] = rho[i];
        if (!fresh) {
          mm[k] = m[i];
          vv[k] = v[i];
        }
      }
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const size_t i = q.gi + C::step(e0 + k);
      if (OUTSIDE || s[e0 + k] > 0) {
        ap.step(g[e0 + k], s[e0 + k], mm[k], vv[k], p[k]);
        m[i] = mm[k];
        v[i] = vv[k];
        rho[i] = p[k];
      }
      g[e0 + k] = s[e0 + k] > 0 ? p[k] : make_float2(0.f, 0.f);
    }
  }
  if (!any || !next) return;
  fft_x<N, Lay, +1, 1, 0>(g, xb, tw, q.c, q.j);
#pragma unroll
  for (int e = 0; e < E; ++e) T[q.ti + (size_t)C::step(e) * LossT<N>::XS] = g[e];
}

}  // namespace spe
