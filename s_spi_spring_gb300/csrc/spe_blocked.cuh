// Iteration kernels over a blocked transform scratch.
//
// T, the array between the row and the column passes, is private to a call,
// so it need not be row-major.  Here the BC columns that a column-pass CTA
// transforms lie next to each other (Blocked<N>): with BC = 4 (32 bytes of a
// row) one warp-wide 8-byte access of the column pass covers 256 contiguous
// bytes, two 128-byte lines, where four columns of a row-major T touch eight.
// The L1's rate of line requests is what kept the row-major column pass from
// using CTAs that narrow; narrow CTAs in turn mean more and smaller barrier
// groups per SM.  Measured on GB300 (one pass over 16.7 M pixels, 8-column
// row-major kernel before -> blocked after): column pass at 512 87 -> 70 us,
// at 1024 129 -> 92 us, at 2048 167 -> 99 us; column + row pass at 256 172 ->
// 155 us, 384 222 -> 187, 512 184 -> 152, 768 240 -> 200, 1024 233 -> 187,
// 2048 265 -> 223.
//
// The column pass reads T straight into registers (no staging through shared
// memory; the next tile's elements are loaded while this one's inverse
// transform runs).  The row pass maps threads like the column pass, (row,
// position) = (t % WR, t / WR), so that its accesses to T are whole lines as
// well, and stages T and the previous iterate with cp.async.  Both are then
// bound by the shared-memory pipe (61% / 72% of its wavefront rate at 512;
// the exchanges of the transforms are 60% of them) with 58% / 40% of the issue
// slots used, not by DRAM.
//
// Two more things are laid out for these kernels:
//   * the support as one bit per pixel, packed by the call's first pass in
//     the order in which the row pass's threads hold their elements (a
//     thread's bits are one byte or one 16-bit word): 1/32 of the int32 array
//     that every iteration read.  A row tile whose support holds anything but
//     0 and 1 is flagged by the packing pass and read as integers instead.
//   * the amplitudes in the order of the column pass's registers (At), so
//     that a thread's E values are E / 4 16-byte loads; made when the
//     amplitudes are set.
//
// Passes alternate their direction over the population (rows upward, columns
// downward): each starts with the individuals that the previous one left in
// L2 (2-3% at 512^2 x 64, 10% at 256^2 x 256).
//
// Per-element arithmetic, radix plans and twiddles are those of the row-major
// kernels (spe_pipe.cuh): bit-identical results.
#pragma once
#include "spe_pipe.cuh"

namespace spe {

// Layout of T and launch shapes per side.  BC: columns of a block (and of a
// column-pass CTA); WR: rows of a row-pass CTA.
// ROWS_TOGETHER: blocks of BR x BC pixels (128 bytes), the blocks of BR rows
// one after the other, so that a row tile is contiguous (equal in speed to
// whole columns of blocks up to 512); otherwise a block's column runs over all
// N rows (5-7% faster at 1024 and 2048).
// NXC / NXR: exchange buffers used in turn (two need one barrier per exchange
// instead of two); ST: stages of the row pass; MBC / MBR: resident CTAs per
// SM the registers must allow.  At 768 and above a 4-row tile of the row pass
// would leave one or two CTAs per SM: two rows.  At 2048 (16 elements per
// thread) two columns: two 256-thread CTAs per SM instead of one of 512.
template <int N>
struct Blocked {
  static constexpr bool ok = N == 256 || N == 384 || N == 512 || N == 768 || N == 1024 || N == 2048;
  static constexpr int BC = N == 2048 ? 2 : 4;
  static constexpr int WR = N <= 512 ? 4 : 2;
  static constexpr bool ROWS_TOGETHER = N <= 512;
  static constexpr int BR = ROWS_TOGETHER ? 4 : 1;
  static constexpr int NXC = 2;
  static constexpr int NXR = N == 2048 ? 1 : 2;
  static constexpr int ST = N == 512 ? 2 : 1;
  static constexpr bool PREFETCH = N != 2048;
  static constexpr int MBC = N == 256 ? 8 : (N == 384 || N == 512 ? 4 : 2);
  static constexpr int MBR = N == 256 ? 6 : N == 384 ? 4 : N == 512 ? 2 : N == 768 ? 4 : N == 1024 ? 3 : 2;
  // offset of pixel (y, x) of an individual; linear in steps of y that are
  // multiples of BR (YS per row) and steps of x that are multiples of BC
  // (XS per BC columns)
  static constexpr int YS = ROWS_TOGETHER ? N : BC;
  static constexpr int XS = ROWS_TOGETHER ? BR * BC : N * BC;
  __host__ __device__ static constexpr int at(int y, int x) {
    return (y / BR) * (BR * YS) + (y % BR) * BC + (x / BC) * XS + x % BC;
  }
};

// a thread's support bits of one row
template <int N>
using SpBits = typename std::conditional<(Elems<N>::value > 8), uint16_t, uint8_t>::type;

// The transform of fft_reg with NX exchange buffers of Lay::SIZE elements.
// With two, consecutive exchanges alternate between them: a thread that
// stores into one has passed the barrier of the other's exchange, which every
// thread reaches after its loads from this one, so the barrier after the
// loads is not needed.  X0: exchanges done before this transform (the buffer
// of its first one); the transforms of a tile must leave an even number in
// all.
template <int L, int S, class Lay, int P, int NS, int NX, int X0>
__device__ __forceinline__ void fft_pass_x(float2* v, float2* __restrict__ buf, const float2* __restrict__ tw, int c,
                                           int j) {
  using Rad = typename Plan<L>::R;
  constexpr int R = Rad::value[P];
  constexpr int TPT = Plan<L>::TPT;
  constexpr int U = L / R / TPT;
  constexpr int OFF = TwiddleTable<L>::offset(P);
#pragma unroll
  for (int u = 0; u < U; ++u) {
    const int b = j + TPT * u;
    const int k = (NS == 1) ? 0 : (b % NS);
    if constexpr (NS > 1) {
#pragma unroll
      for (int r = 1; r < R; ++r) {
        float2 w = tw[OFF + (r - 1) * NS + k];
        if (S < 0) w.y = -w.y;
        v[u * R + r] = cmul(v[u * R + r], w);
      }
    }
    dft<R, S>(v + u * R);
  }
  if constexpr (P + 1 < Rad::count) {
    float2* xb = buf + ((NX == 2 && ((P + X0) & 1)) ? Lay::SIZE : 0);
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int b = j + TPT * u;
      const int k = (NS == 1) ? 0 : (b % NS);
      const int base = (b / NS) * NS * R + k;
#pragma unroll
      for (int q = 0; q < R; ++q) xb[store_addr<Lay, NS, R>(base, q, c)] = v[u * R + q];
    }
    __syncthreads();
    constexpr int R2 = Rad::value[P + 1];
    constexpr int NB2 = L / R2;
    constexpr int U2 = NB2 / TPT;
    static_assert(U2 * R2 == U * R, "every pass must keep E elements per thread");
#pragma unroll
    for (int u = 0; u < U2; ++u) {
      const int b = j + TPT * u;
#pragma unroll
      for (int r = 0; r < R2; ++r) v[u * R2 + r] = xb[load_addr_x<Lay, NB2, NS>(b, r, c)];
    }
    if constexpr (NX == 1) __syncthreads();
    fft_pass_x<L, S, Lay, P + 1, NS * R, NX, X0>(v, buf, tw, c, j);
  }
}
template <int L, class Lay, int S, int NX, int X0>
__device__ __forceinline__ void fft_x(float2* v, float2* buf, const float2* tw, int c, int j) {
  fft_pass_x<L, S, Lay, 0, 1, NX, X0>(v, buf, tw, c, j);
}

// W sequences of N per CTA: thread t holds positions elem_pos(e, t / W) of
// sequence t % W
template <int N, int W, int NX>
struct BlkCfg {
  static constexpr int TPT = Plan<N>::TPT;
  static constexpr int E = Elems<N>::value;
  static constexpr int R0 = Plan<N>::R::value[0];
  static constexpr int NB = N / R0;
  static constexpr int EX = Plan<N>::R::count - 1;  // exchanges of a transform
  static constexpr int NT = W * TPT;
  static constexpr int TWB = align128(TwiddleTable<N>::size() * 8);
  using Lay = LayCol<N, W>;
  static constexpr int XB = align128(NX * Lay::SIZE * 8);
  static constexpr size_t SMEM = (size_t)TWB + XB;
  static_assert(NT % 32 == 0 && NT <= 1024, "whole warps");
  // position of element e relative to element 0
  __host__ __device__ static constexpr int step(int e) { return (e / R0) * TPT + (e % R0) * NB; }
};

// Row tiles of an ER call.  The update multiplies by the support, so that
// outside the row tiles that hold any the density, and its row transform, are
// zeros, and of the projected column transform only those tiles' rows are
// used.  A support is compact (a quarter of the rows or less, from the
// oversampling that phase retrieval needs): the passes between the first and
// the last column pass leave the other tiles out.  `odd` carries the tiles'
// state, `live` the list of those with support: its length, a counter per
// individual (tiles seen, and 2^16 times those with support), the tiles.
// (A tile that is not finite counts as one with support: 0 times it is not 0.
// An individual without any support has all its tiles in the list: its density
// is zeros of either sign, and the projection of an all-zero transform goes by
// their signs.  Not with a phase gate, which may empty a support.)
// The flags and the list cost a dependent read each before a tile's own; from
// 3/8 of the tiles on that is more than the rest saves, and every tile runs (20
// iterations, us, support over 25 / 36 / 45% of the rows; no live tiles:
// 512^2 x 64 2127 / 2342 / 3208; 3214, 1024^2 x 4 890 / 930 / 1048; 1024; live
// tiles whatever the support, over all rows: 3607 and 1265).
enum { TILE_ODD = 1, TILE_LIVE = 2 };
__device__ __forceinline__ bool every_tile(const int* live, int tiles) { return __ldcg(live) > tiles / 8 * 3; }

// column pass: T -> FFT+ (y) -> P_M with A -> FFT- (y) -> T.  IN / OUT: only
// the rows of live tiles are read (the others are zeros) / written.
template <int N, bool IN, bool OUT>
__global__ void __launch_bounds__(BlkCfg<N, Blocked<N>::BC, Blocked<N>::NXC>::NT, Blocked<N>::MBC)
    k_cols_blocked(float2* __restrict__ T, const float* __restrict__ At, const unsigned char* __restrict__ odd,
                   const int* __restrict__ live, int ipp, int first, int count, const float2* __restrict__ twg) {
  using B = Blocked<N>;
  constexpr int W = B::BC, NX = B::NXC;
  using C = BlkCfg<N, W, NX>;
  using Lay = typename C::Lay;
  constexpr int NT = C::NT, E = C::E, TPI = N / W;
  constexpr bool PF = B::PREFETCH;
  static_assert(C::TPT % B::WR == 0 && C::NB % B::WR == 0, "a thread's rows are tiles apart");
  extern __shared__ __align__(128) unsigned char sm[];
  float2* tw = reinterpret_cast<float2*>(sm);
  float2* xb = reinterpret_cast<float2*>(sm + C::TWB);
  pdl_enter();
  load_twiddles<N>(tw, twg, NT);
  __syncthreads();
  pdl_wait();
  const int t = threadIdx.x;
  const int c = t % W, j = t / W;
  const int ntiles = count * TPI;
  const bool all = (!IN && !OUT) || every_tile(live, count * (N / B::WR));
  // tiles run downward (see the head of the file); T is written by other
  // SMs between the launches: loads go to L2 (__ldcg)
  const size_t off = (size_t)first * N * N + B::at(j, c);
  auto tile_ptr = [&](int k) {
    const int tile = ntiles - 1 - k;
    return T + off + (size_t)(tile / TPI) * N * N + (size_t)(tile % TPI) * B::XS;
  };
  // the thread's rows of live tiles, as bits
  auto rows_of = [&](int k) {
    if (all) return 0xffffffffu;
    const unsigned char* f = odd + (size_t)(first + (ntiles - 1 - k) / TPI) * (N / B::WR) + j / B::WR;
    unsigned r = 0;
#pragma unroll
    for (int e = 0; e < E; ++e) r |= (__ldcg(f + C::step(e) / B::WR) & TILE_LIVE) ? 1u << e : 0u;
    return r;
  };
  auto fetch = [&](float2* v, int k, unsigned rows) {
    const float2* g = tile_ptr(k);
#pragma unroll
    for (int e = 0; e < E; ++e)
      v[e] = !IN || ((rows >> e) & 1u) ? __ldcg(g + (size_t)C::step(e) * B::YS) : make_float2(0.f, 0.f);
  };
  float2 v[E], nx[PF ? E : 1];
  int k = blockIdx.x;
  unsigned rows = 0, nrows = 0;
  if (k < ntiles) {
    rows = rows_of(k);
    if (PF) fetch(nx, k, rows);
    nrows = k + (int)gridDim.x < ntiles ? rows_of(k + gridDim.x) : rows;
  }
  for (; k < ntiles; k += gridDim.x) {
    const int nk = k + gridDim.x;
    if (PF) {
#pragma unroll
      for (int e = 0; e < E; ++e) v[e] = nx[PF ? e : 0];
    } else {
      fetch(v, k, rows);
    }
    const int tile = ntiles - 1 - k;
    const int p = first + tile / TPI;
    const float4* A4 = reinterpret_cast<const float4*>(At + (ipp > 0 ? (size_t)(p / ipp) * N * N : 0)) +
                       (size_t)((tile % TPI) * NT + t) * (E / 4);
    float4 a[E / 4];
#pragma unroll
    for (int i = 0; i < E / 4; ++i) a[i] = __ldg(A4 + i);
    fft_x<N, Lay, +1, NX, 0>(v, xb, tw, c, j);
#pragma unroll
    for (int i = 0; i < E / 4; ++i) {
      v[4 * i + 0] = project(v[4 * i + 0], a[i].x);
      v[4 * i + 1] = project(v[4 * i + 1], a[i].y);
      v[4 * i + 2] = project(v[4 * i + 2], a[i].z);
      v[4 * i + 3] = project(v[4 * i + 3], a[i].w);
    }
    if (PF) fetch(nx, nk < ntiles ? nk : k, nk < ntiles ? nrows : rows);
    fft_x<N, Lay, -1, NX, C::EX>(v, xb, tw, c, j);
    float2* g = tile_ptr(k);
#pragma unroll
    for (int e = 0; e < E; ++e)
      if (!OUT || ((rows >> e) & 1u)) g[(size_t)C::step(e) * B::YS] = v[e];
    rows = nrows;
    if (nk + (int)gridDim.x < ntiles) nrows = rows_of(nk + gridDim.x);
  }
}

template <int N>
struct BlkRowCfg : BlkCfg<N, Blocked<N>::WR, Blocked<N>::NXR> {
  using C = BlkCfg<N, Blocked<N>::WR, Blocked<N>::NXR>;
  static constexpr int WR = Blocked<N>::WR;
  // a staged row of the iterate is padded by 16 / WR elements: the WR rows of
  // a half-warp's accesses fall into different banks
  static constexpr int RS = N + 16 / WR;
  static constexpr int R_T = align128(N * WR * 8);
  static constexpr int R_R = align128(WR * RS * 8);
  static constexpr int STAGE = R_T + R_R;
  static constexpr size_t SMEM = C::SMEM + (size_t)Blocked<N>::ST * STAGE;
};

// row pass: T -> FFT- (x) -> /N^2 -> update with (rho, support) -> rho -> FFT+ (x) -> T
template <int N, int UPD, bool LIST>
__global__ void __launch_bounds__(BlkRowCfg<N>::NT, Blocked<N>::MBR)
    k_rows_blocked(float2* __restrict__ T, float2* __restrict__ rho, const int* __restrict__ S,
                   const SpBits<N>* __restrict__ sp, const unsigned char* __restrict__ odd,
                   const int* __restrict__ live, int first, int count, float scale, float beta, Gate g,
                   const float2* __restrict__ twg) {
  using B = Blocked<N>;
  using C = BlkRowCfg<N>;
  using Lay = typename C::Lay;
  constexpr int NT = C::NT, E = C::E, TPT = C::TPT, W = B::WR, TPI = N / W, RS = C::RS, ST = B::ST, NX = B::NXR;
  constexpr int CB = W * B::BC / 2;  // 16-byte chunks of the tile's part of a column of blocks
  static_assert(NT % CB == 0 && (N * W / 2) % NT == 0 && TPT % B::BC == 0 && (B::BR == 1 || B::BR == W), "tile shape");
  constexpr bool NEED_PREV = (UPD != UPD_ER);
  extern __shared__ __align__(128) unsigned char sm[];
  float2* tw = reinterpret_cast<float2*>(sm);
  float2* xb = reinterpret_cast<float2*>(sm + C::TWB);
  unsigned char* stages = sm + C::C::SMEM;
  pdl_enter();
  load_twiddles<N>(tw, twg, NT);
  pdl_wait();
  const int t = threadIdx.x;
  const int c = t % W, j = t / W;
  // the tiles of the pass: all, or (LIST) the live ones by their list
  const bool all = !LIST || every_tile(live, count * TPI);
  const int ntiles = all ? count * TPI : __ldcg(live);
  auto tile_at = [&](int k) { return all ? k : __ldcg(live + 1 + count + k); };
  // offset of a tile's first row in T (blocked), rho and S (row-major)
  auto t_base = [&](int tile) {
    return (size_t)(first + tile / TPI) * N * N + (size_t)(tile % TPI) * (W * B::YS);
  };
  auto r_base = [&](int tile) { return ((size_t)first * N + (size_t)tile * W) * N; };
  // staged T: [columns of blocks][W rows][BC]
  auto stage_T = [&](int tile, int s) {
    float2* sT = reinterpret_cast<float2*>(stages + s * C::STAGE) + 2 * t;
    const int r = 2 * (t % CB);  // (row of the tile, column of the block) = (r / BC, r % BC)
    const float2* src = T + t_base(tile) + (size_t)(t / CB) * B::XS + r;
#pragma unroll
    for (int i = 0; i < N * W / 2 / NT; ++i) cp_async16(sT + i * 2 * NT, src + (size_t)i * (NT / CB) * B::XS);
  };
  auto stage_R = [&](int tile, int s) {
    if (!NEED_PREV) return;
    float2* sR = reinterpret_cast<float2*>(stages + s * C::STAGE + C::R_T);
    const float2* src = rho + r_base(tile);
#pragma unroll
    for (int i = 0; i < N * W / 2 / NT; ++i) {
      const int q = t + i * NT;
      cp_async16(&sR[(q / (N / 2)) * RS + 2 * (q % (N / 2))], src + 2 * q);
    }
  };
  // the thread's support bits of a tile, bit 16: the tile's support is not 0 / 1
  auto bits_of = [&](int tile) {
    const unsigned b = sp[((size_t)first * N + (size_t)tile * W + c) * TPT + j];
    return b | ((unsigned)(odd[(size_t)first * TPI + tile] & TILE_ODD) << 16);
  };
  int i = blockIdx.x, listed = 0;
  unsigned nbits = 0;
  if (i < ntiles) {
    listed = tile_at(i);
    stage_T(listed, 0);
    stage_R(listed, 0);
    nbits = bits_of(listed);
  }
  cp_async_commit();
  for (int k = 0; i < ntiles; ++k, i += gridDim.x) {
    const int tile = LIST ? listed : i;
    const bool more = i + (int)gridDim.x < ntiles;
    const int nxt = LIST && !more ? 0 : tile_at(i + gridDim.x);
    listed = nxt;
    const int s = ST == 2 ? (k & 1) : 0;
    const unsigned bits = nbits;
    if constexpr (ST == 2) {
      if (more) {
        stage_T(nxt, s ^ 1);
        stage_R(nxt, s ^ 1);
        nbits = bits_of(nxt);
      }
      cp_async_commit();
      cp_async_wait_prev();
    } else {
      cp_async_wait_all();
    }
    __syncthreads();  // this tile is in the stage
    const float2* sT = reinterpret_cast<const float2*>(stages + s * C::STAGE) + (j / B::BC) * (W * B::BC) + c * B::BC +
                       j % B::BC;
    const float2* sR = reinterpret_cast<const float2*>(stages + s * C::STAGE + C::R_T) + c * RS + j;
    const size_t rb = r_base(tile) + (size_t)c * N + j;
    float2 v[E];
#pragma unroll
    for (int e = 0; e < E; ++e) v[e] = sT[C::step(e) * W];
    if constexpr (ST == 1) {
      __syncthreads();  // every thread has read its elements of T
      if (more) stage_T(nxt, 0);
      cp_async_commit();
    }
    fft_x<N, Lay, -1, NX, 0>(v, xb, tw, c, j);
    const bool plain = (bits >> 16) != 0;  // (the same for every thread of a tile)
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const float2 rp = __fmul2_rn(v[e], make_float2(scale, scale));
      const float2 prev = NEED_PREV ? sR[C::step(e)] : make_float2(0.f, 0.f);
      int m = (int)((bits >> e) & 1u);
      if (plain) m = S[rb + C::step(e)];
      const float2 r = update<UPD>(rp, prev, m, beta, g);
      if (NEED_PREV) rho[rb + C::step(e)] = r;  // (ER reads no previous iterate, and the last pass writes the result)
      v[e] = r;
    }
    if constexpr (ST == 1) {
      if (NEED_PREV) __syncthreads();  // every thread has read its elements of the previous iterate
      if (more) {
        stage_R(nxt, 0);
        nbits = bits_of(nxt);
      }
      cp_async_commit();
    }
    fft_x<N, Lay, +1, NX, C::EX>(v, xb, tw, c, j);
    float2* gt = T + t_base(tile) + B::at(c, j);
#pragma unroll
    for (int e = 0; e < E; ++e) gt[(size_t)(C::step(e) / B::BC) * B::XS] = v[e];
    if constexpr (ST == 2) __syncthreads();  // stage s is refilled by the next iteration's copies
  }
  cp_async_wait_all();  // no copy outlives the CTA
}

// First pass of a call: rho -> FFT+ (x) -> T; packs the support and, with LIST,
// lists the live tiles (length and counters: 0 before).  One tile per CTA, loads
// in flight over many CTAs per SM.
template <int N, bool LIST>
__global__ void __launch_bounds__(BlkRowCfg<N>::NT, BlkCfg<N, Blocked<N>::WR, 1>::E <= 8 ? 1024 / BlkRowCfg<N>::NT : 2)
    k_rows_blocked_first(const float2* __restrict__ rho, const int* __restrict__ S, float2* __restrict__ T,
                         SpBits<N>* __restrict__ sp, unsigned char* __restrict__ odd, int* __restrict__ live,
                         int first, int count, const float2* __restrict__ twg) {
  using B = Blocked<N>;
  using C = BlkCfg<N, B::WR, 1>;
  using Lay = typename C::Lay;
  constexpr int NT = C::NT, E = C::E, TPT = C::TPT, W = B::WR, TPI = N / W;
  extern __shared__ __align__(128) unsigned char sm[];
  float2* tw = reinterpret_cast<float2*>(sm);
  float2* xb = reinterpret_cast<float2*>(sm + C::TWB);
  const int t = threadIdx.x;
  const int c = t % W, j = t / W;
  const int tile = blockIdx.x;
  const size_t rb = ((size_t)first * N + (size_t)tile * W + c) * N + j;
  float2 v[E];
  int m[E];
#pragma unroll
  for (int e = 0; e < E; ++e) v[e] = __ldcg(rho + rb + C::step(e));
#pragma unroll
  for (int e = 0; e < E; ++e) m[e] = __ldcg(S + rb + C::step(e));
  load_twiddles<N>(tw, twg, NT);
  unsigned bits = 0;
  int other = 0;
#pragma unroll
  for (int e = 0; e < E; ++e) {
    bits |= m[e] != 0 ? 1u << e : 0u;
    other |= m[e] & ~1;
  }
  sp[((size_t)first * N + (size_t)tile * W + c) * TPT + j] = (SpBits<N>)bits;
  int state = other != 0 ? TILE_ODD : 0;
  if (LIST) {
    float chk = 0.f;
#pragma unroll
    for (int e = 0; e < E; ++e) chk += 0.f * v[e].x + 0.f * v[e].y;
    if (bits != 0 || chk != 0.f) state |= TILE_LIVE;
  }
  // (also: the twiddles are in shared memory)
  state = (__syncthreads_or(state & TILE_ODD) ? TILE_ODD : 0) |
          (LIST && __syncthreads_or(state & TILE_LIVE) ? TILE_LIVE : 0);
  if (t == 0) {
    odd[(size_t)first * TPI + tile] = (unsigned char)state;
    if (LIST) {
      int* list = live + 1 + count;
      if (state & TILE_LIVE) list[atomicAdd(live, 1)] = tile;
      // the individual's last tile sees whether it has any support
      __threadfence();
      const int add = 1 + (state & TILE_LIVE ? 1 << 16 : 0);
      if (atomicAdd(live + 1 + tile / TPI, add) + add == TPI) {
        __threadfence();
        const int t0 = tile / TPI * TPI, at = atomicAdd(live, TPI);
        for (int k = 0; k < TPI; ++k) {
          unsigned char* f = odd + (size_t)first * TPI + t0 + k;
          *f = (unsigned char)(__ldcg(f) | TILE_LIVE);
          list[at + k] = t0 + k;
        }
      }
    }
  }
  fft_x<N, Lay, +1, 1, 0>(v, xb, tw, c, j);
  float2* gt = T + (size_t)(first + tile / TPI) * N * N + (size_t)(tile % TPI) * (W * B::YS) + B::at(c, j);
#pragma unroll
  for (int e = 0; e < E; ++e) gt[(size_t)(C::step(e) / B::BC) * B::XS] = v[e];
}

// Last pass of a call: T -> FFT- (x) -> /N^2 -> rho (the trailing modulus
// projection of GPU_context::HIO/RAAR/ER, gpu_context.cu:803-812)
template <int N>
__global__ void __launch_bounds__(BlkRowCfg<N>::NT, BlkCfg<N, Blocked<N>::WR, 1>::E <= 8 ? 1024 / BlkRowCfg<N>::NT : 2)
    k_rows_blocked_last(const float2* __restrict__ T, float2* __restrict__ rho, int first, float scale,
                        const float2* __restrict__ twg) {
  using B = Blocked<N>;
  using C = BlkCfg<N, B::WR, 1>;
  using Lay = typename C::Lay;
  constexpr int NT = C::NT, E = C::E, W = B::WR, TPI = N / W;
  extern __shared__ __align__(128) unsigned char sm[];
  float2* tw = reinterpret_cast<float2*>(sm);
  float2* xb = reinterpret_cast<float2*>(sm + C::TWB);
  const int t = threadIdx.x;
  const int c = t % W, j = t / W;
  const int tile = blockIdx.x;
  const float2* gt = T + (size_t)(first + tile / TPI) * N * N + (size_t)(tile % TPI) * (W * B::YS) + B::at(c, j);
  float2 v[E];
#pragma unroll
  for (int e = 0; e < E; ++e) v[e] = __ldcg(gt + (size_t)(C::step(e) / B::BC) * B::XS);
  load_twiddles<N>(tw, twg, NT);
  __syncthreads();
  fft_x<N, Lay, -1, 1, 0>(v, xb, tw, c, j);
  float2* gr = rho + ((size_t)first * N + (size_t)tile * W + c) * N + j;
#pragma unroll
  for (int e = 0; e < E; ++e) gr[C::step(e)] = make_float2(v[e].x * scale, v[e].y * scale);
}

// Any op (spe_kernels.cuh) on the blocked scratch: one tile per CTA, W = WR
// rows or BC columns, elements straight between memory and registers.  Row
// passes read and write the row-major arrays in runs of 32 / WR pixels.  An
// op's per-pixel operand comes in the order of k_block_amplitudes.
template <int N, int AXIS, class Op>
struct BlkPassCfg : BlkCfg<N, AXIS == AX_ROWS ? Blocked<N>::WR : Blocked<N>::BC, 2> {
  static constexpr int W = AXIS == AX_ROWS ? Blocked<N>::WR : Blocked<N>::BC;
  using C = BlkCfg<N, W, 2>;
  // registers a thread: 64 (a pair of arrays: 80) per 8 elements
  static constexpr int REGS = C::E <= 8 ? (Op::PAIR ? 80 : 64) : 128;
  static constexpr int MINB = 65536 / (C::NT * REGS) < 1 ? 1 : 65536 / (C::NT * REGS);
};
template <int N, int AXIS, class Op>
__global__ void __launch_bounds__(BlkPassCfg<N, AXIS, Op>::NT, BlkPassCfg<N, AXIS, Op>::MINB)
    k_blocked_pass(const Op op, const float2* __restrict__ twg) {
  using B = Blocked<N>;
  using C = BlkPassCfg<N, AXIS, Op>;
  using Lay = typename C::Lay;
  constexpr int NT = C::NT, E = C::E, W = C::W, TPI = N / W;
  static_assert(!Op::AMP || (AXIS == AX_COLS && E % 4 == 0), "operands are in column order");
  extern __shared__ __align__(128) unsigned char sm[];
  float2* tw = reinterpret_cast<float2*>(sm);
  float2* xb = reinterpret_cast<float2*>(sm + C::TWB);
  pdl_enter();
  load_twiddles<N>(tw, twg, NT);
  const int t = threadIdx.x;
  const int c = t % W, j = t / W;
  const int p = op.first + blockIdx.x / TPI;
  const int fixed = (blockIdx.x % TPI) * W + c;
  const int y0 = AXIS == AX_ROWS ? fixed : j, x0 = AXIS == AX_ROWS ? j : fixed;
  const size_t g0 = (size_t)p * N * N + (size_t)y0 * N + x0, t0 = (size_t)p * N * N + B::at(y0, x0);
  typename Op::Acc acc;
  pdl_wait();
  __syncthreads();
  float4 a[Op::AMP ? E / 4 : 1];
  if constexpr (Op::AMP) {
    const float4* A4 = reinterpret_cast<const float4*>(op.amp(p, N)) + (size_t)((blockIdx.x % TPI) * NT + t) * (E / 4);
#pragma unroll
    for (int i = 0; i < E / 4; ++i) a[i] = __ldg(A4 + i);
  }
  auto px = [&](int e) {
    const int d = C::step(e);
    Px q;
    q.p = p;
    q.y = AXIS == AX_ROWS ? y0 : y0 + d;
    q.x = AXIS == AX_ROWS ? x0 + d : x0;
    q.gi = g0 + (AXIS == AX_ROWS ? (size_t)d : (size_t)d * N);
    q.ti = t0 + (AXIS == AX_ROWS ? (size_t)(d / B::BC) * B::XS : (size_t)d * B::YS);
    q.a = 0.f;
    if constexpr (Op::AMP) q.a = e % 4 == 0 ? a[e / 4].x : e % 4 == 1 ? a[e / 4].y : e % 4 == 2 ? a[e / 4].z : a[e / 4].w;
    return q;
  };
  // (two exchange buffers in turn: one barrier per exchange)
  pass_elements<N, E, Lay, Op>(op, px, acc, [&](float2* v, auto sign, auto nth) {
    fft_x<N, Lay, decltype(sign)::value, 2, decltype(nth)::value * C::EX>(v, xb, tw, c, j);
  });
  if constexpr (Op::NSUM + Op::NMAX > 0) {
    float r[NRED];
    acc.values(r);
    block_reduce_store<NT, Op::NSUM, Op::NMAX>(op.partials, blockIdx.x, r);
  }
  if constexpr (Op::PEAK) block_argmax_store<NT>(op.partials, acc.mx, acc.idx);
}

// ---- the column pass of the Fourier-space crossover
// The pixels that child w takes from the crossed parents, as a bit per element
// of the column pass's threads (SpBits): the polar coordinates of a pixel cost
// more than its share of the pass, and here one thread has nothing else to
// hold.
template <int N>
__global__ void k_cross_bits(const CrossArgs a) {
  constexpr int W = Blocked<N>::BC, TPT = Plan<N>::TPT, NT = W * TPT, E = Elems<N>::value;
  const CrossChild c = a.children[blockIdx.y];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;  // (tile, thread)
  if (i >= N * TPT) return;
  const int tile = i / NT, t = i % NT;
  unsigned bits = 0;
#pragma unroll
  for (int e = 0; e < E; ++e)
    bits |= cross_pixel(tile * W + t % W, elem_pos<N>(e, t / W), N, c, a.crosssym, a.cmaps, a.cmap_total) ? 1u << e : 0u;
  reinterpret_cast<SpBits<N>*>(a.bits)[(size_t)blockIdx.y * N * TPT + i] = (SpBits<N>)bits;
}

// row pass of the children's parents: gathered copy of item blockIdx / TPI ->
// FFT+ (x) -> W; the shifted supports of self, p2 and p3 into Ws.  (450 us at
// 512^2 x 64, four parents a child: the reads at any shift and the int32
// supports take twice the L1 line requests of the plain forward pass.)
template <int N>
__global__ void __launch_bounds__(BlkCfg<N, Blocked<N>::WR, 1>::NT,
                                  BlkCfg<N, Blocked<N>::WR, 1>::E <= 8 ? 1024 / BlkCfg<N, Blocked<N>::WR, 1>::NT : 2)
    k_cross_rows(const CrossArgs a, Gate g, const float2* __restrict__ twg) {
  using B = Blocked<N>;
  constexpr int W = B::WR;
  using C = BlkCfg<N, W, 1>;
  constexpr int E = C::E, TPI = N / W;
  constexpr size_t npix = (size_t)N * N;
  extern __shared__ __align__(128) unsigned char sm[];
  float2* tw = reinterpret_cast<float2*>(sm);
  float2* xb = reinterpret_cast<float2*>(sm + C::TWB);
  pdl_enter();
  load_twiddles<N>(tw, twg, C::NT);
  const int c = threadIdx.x % W, j = threadIdx.x / W;
  const int p = blockIdx.x / TPI, y = (blockIdx.x % TPI) * W + c;
  pdl_wait();
  __syncthreads();
  const ShiftItem it = load_item(a.items + p);
  const int row = shift_source(it, j, y, N) / N;  // of the source: the same for the whole row
  const int x0 = (it.flip ? N - 1 - j : j) - it.sx, dir = it.flip ? -1 : 1;
  const float2* src = a.rho + (size_t)it.src * npix + (size_t)row * N;
  // (an item without a support of its own is gated with gsrc, unshifted: only
  // the plain copy, whose shift is 0)
  const int ss = it.ssrc >= 0 ? it.ssrc : it.gsrc;
  const int* sup = a.S + (size_t)max(ss, 0) * npix + (size_t)row * N;
  float2 v[E];
  int s[E];
#pragma unroll
  for (int e = 0; e < E; ++e) {
    int x = x0 + dir * C::step(e);
    x += x < 0 ? N : (x >= N ? -N : 0);
    v[e] = __ldcg(src + x);
    s[e] = ss >= 0 ? __ldcg(sup + x) : 0;
  }
  if (it.sdst >= 0) {
    int* ws = a.Ws + (size_t)it.sdst * npix + (size_t)y * N + j;
#pragma unroll
    for (int e = 0; e < E; ++e) ws[C::step(e)] = s[e];
  }
#pragma unroll
  for (int e = 0; e < E; ++e) {
    v[e] = shift_value(it, v[e]);
    if (it.gate) {
      const float t = s[e] == 0 || phase_out(v[e], g) ? 0.f : (float)s[e];
      v[e] = make_float2(v[e].x * t, v[e].y * t);
    }
  }
  fft_x<N, typename C::Lay, +1, 1, 0>(v, xb, tw, c, j);
  float2* o = a.W + (size_t)p * npix + B::at(y, j);
#pragma unroll
  for (int e = 0; e < E; ++e) o[(size_t)(C::step(e) / B::BC) * B::XS] = v[e];
}

// W[per w + k] (row transforms) -> FFT+ (y) -> crossed child -> FFT- (y) -> C[w].
// Each parent is transformed in turn and only its share kept, so the parents'
// spectra never reach memory (they were written once and read twice).
template <int N, bool AVG>
__global__ void __launch_bounds__(BlkCfg<N, Blocked<N>::BC, 1>::NT,
                                  BlkCfg<N, Blocked<N>::BC, 1>::E <= 8 ? 768 / BlkCfg<N, Blocked<N>::BC, 1>::NT : 1)
    k_cross_cols(const CrossArgs a, const float* __restrict__ At, const float2* __restrict__ twg) {
  using B = Blocked<N>;
  constexpr int W = B::BC;
  using C = BlkCfg<N, W, 1>;
  using Lay = typename C::Lay;
  constexpr int NT = C::NT, E = C::E, TPI = N / W;
  extern __shared__ __align__(128) unsigned char sm[];
  float2* tw = reinterpret_cast<float2*>(sm);
  float2* xb = reinterpret_cast<float2*>(sm + C::TWB);
  pdl_enter();
  load_twiddles<N>(tw, twg, NT);
  const int t = threadIdx.x, c = t % W, j = t / W;
  const int w = blockIdx.x / TPI, tile = blockIdx.x % TPI;
  constexpr size_t npix = (size_t)N * N;
  const size_t t0 = B::at(j, tile * W + c);
  pdl_wait();
  __syncthreads();
  const unsigned bits = reinterpret_cast<const SpBits<N>*>(a.bits)[((size_t)w * TPI + tile) * NT + t];
  auto spectrum = [&](float2* v, int k) {
    const float2* g = a.W + ((size_t)a.per * w + k) * npix + t0;
#pragma unroll
    for (int e = 0; e < E; ++e) v[e] = __ldcg(g + (size_t)C::step(e) * B::YS);
    fft_x<N, Lay, +1, 1, 0>(v, xb, tw, c, j);
  };
  float2 out[E], d[E], v[E];
  spectrum(out, 0);
  spectrum(d, 2);
  spectrum(v, 3);
#pragma unroll
  for (int e = 0; e < E; ++e) d[e] = make_float2(d[e].x - v[e].x, d[e].y - v[e].y);
  float amod[AVG ? E : 1];
  if (AVG) {
    spectrum(v, 4);
#pragma unroll
    for (int e = 0; e < E; ++e) amod[AVG ? e : 0] = sqrtf(v[e].x * v[e].x + v[e].y * v[e].y);
  }
  spectrum(v, 1);
#pragma unroll
  for (int e = 0; e < E; ++e) {
    float2 d1 = v[e];
    if (AVG && ((bits >> e) & 1u) && At[((size_t)tile * NT + t) * E + e] < 0.f)
      d1 = cross_average(d1, a.avg_mod[(size_t)(j + C::step(e)) * N + tile * W + c], amod[AVG ? e : 0], a.use_average);
    if ((bits >> e) & 1u) out[e] = make_float2(d1.x + a.crossdiff * d[e].x, d1.y + a.crossdiff * d[e].y);
  }
  fft_x<N, Lay, -1, 1, 0>(out, xb, tw, c, j);
  float2* o = a.C + (size_t)w * npix + t0;
#pragma unroll
  for (int e = 0; e < E; ++e) o[(size_t)C::step(e) * B::YS] = out[e];
}

// amplitudes in the order of the column pass's registers: At[(tile of BC
// columns) * NT + thread][e]; with BAND, the correlation ops' weights
// (band_weight) of the band [minr, maxr] instead
template <int N, bool BAND>
__global__ void k_block_amplitudes(const float* __restrict__ A, float* __restrict__ At, int npatterns, float minr,
                                   float maxr) {
  using C = BlkCfg<N, Blocked<N>::BC, 1>;
  constexpr int W = Blocked<N>::BC, NT = C::NT, E = C::E;
  const size_t total = (size_t)npatterns * N * N;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
    const size_t pat = i / ((size_t)N * N);
    const int q = (int)(i % ((size_t)N * N));
    const int e = q % E, t = (q / E) % NT, tile = q / (E * NT);
    const int y = elem_pos<N>(e, t / W), x = tile * W + t % W;
    const float a = A[pat * N * N + (size_t)y * N + x];
    At[i] = BAND ? band_weight(a, x, y, N, minr, maxr) : a;
  }
}

}  // namespace spe
