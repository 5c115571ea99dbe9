// Size-specialised op sequences.  Each spe_size_<N>.cu instantiates this for
// one pattern side so that the sizes compile in parallel.
#pragma once
#include <atomic>

#include "spe_internal.h"
#include "spe_kernels.cuh"
#include "spe_pipe.cuh"
#include "spe_blocked.cuh"
#include "spe_cluster.cuh"
#include "spe_support.cuh"
#include "spe_pairs.cuh"
#include "spe_tma.cuh"

namespace spe {

// Per-device caches below are shared by every engine and host thread: they
// are atomics, and what they cache (an attribute set, a count queried) is
// the same whichever thread fills it first.
inline int sm_count() {
  static std::atomic<int> count[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 64) {
    int c = 0;
    cudaDeviceGetAttribute(&c, cudaDevAttrMultiProcessorCount, dev);
    return c > 0 ? c : 148;
  }
  int c = count[dev].load(std::memory_order_acquire);
  if (c == 0) {
    cudaDeviceGetAttribute(&c, cudaDevAttrMultiProcessorCount, dev);
    count[dev].store(c, std::memory_order_release);
  }
  return c;
}

// Shared-memory opt-in of one kernel, once per device.  `configured` must be
// distinct per kernel instantiation: callers pass their own flag word.  Two
// threads may both set the (idempotent) attributes; a thread that sees the
// device's bit knows they are set.
template <class K>
cudaError_t configure(K kern, size_t smem, std::atomic<unsigned long long>& configured) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const unsigned long long bit = dev < 64 ? (1ull << dev) : 0ull;
  if (!bit || !(configured.load(std::memory_order_acquire) & bit)) {
    e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
    if (e != cudaSuccess) return e;
    if (bit) configured.fetch_or(bit, std::memory_order_release);
  }
  return cudaSuccess;
}

// launch with programmatic stream serialisation (the kernel's prologue
// overlaps the previous kernel's drain; see pdl_wait)
template <class K, class... Args>
cudaError_t launch_pdl(K kern, int grid, int threads, size_t smem, cudaStream_t st, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, args...);
}

template <int N, int AXIS, class Op>
cudaError_t launch_pass(const Op& op, int count, cudaStream_t st, const float2* tw) {
  using C = PassCfg<N, AXIS>;
  constexpr int W = C::W;
  constexpr int NT = C::NT;
  // the block reductions shuffle with a full warp mask
  static_assert(NT % 32 == 0, "pass kernels need whole warps");
  const size_t smem = C::SMEM;
  auto kern = pass_kernel<N, AXIS, Op>;
  // the dynamic shared-memory opt-in is per device and per kernel
  static std::atomic<unsigned long long> configured{0ull};
  cudaError_t e = configure(kern, smem, configured);
  if (e != cudaSuccess) return e;
  if (count <= 0) return cudaSuccess;
  return launch_pdl(kern, (int)((unsigned)count * (N / W)), NT, smem, st, op, tw);
}

// an op on the blocked scratch where the side has one, else row-major
template <int N, int AXIS, class Op>
cudaError_t run_pass(const Op& op, int count, cudaStream_t st, const float2* tw) {
  if constexpr (Blocked<N>::ok) {
    using C = BlkPassCfg<N, AXIS, Op>;
    auto kern = k_blocked_pass<N, AXIS, Op>;
    static std::atomic<unsigned long long> configured{0ull};
    cudaError_t e = configure(kern, C::SMEM, configured);
    if (e != cudaSuccess || count <= 0) return e;
    return launch_pdl(kern, (int)((unsigned)count * (N / C::W)), C::NT, C::SMEM, st, op, tw);
  } else {
    return launch_pass<N, AXIS>(op, count, st, tw);
  }
}

// tile-width variants compiled per size: those whose tile fits in shared
// memory with whole warps
constexpr size_t kMaxSmem = 232448;  // 227 KB per CTA
template <int N, int W>
constexpr bool col_ok() {
  return W <= N && N % W == 0 && ColCfg<N, W>::NT % 32 == 0 && ColCfg<N, W>::NT <= 1024 &&
         ColCfg<N, W>::SMEM <= kMaxSmem;
}
template <int N, int W, class XLay = LayPad<N, W>>
constexpr bool row_ok() {
  return W <= N && N % W == 0 && RowCfg<N, W, XLay>::NT % 32 == 0 && RowCfg<N, W, XLay>::NT <= 1024 &&
         RowCfg<N, W, XLay>::SMEM <= kMaxSmem;
}
// the one-stage row pass (k_rows_iterate1): where the two-stage one fits
// fewer CTAs per SM than it would
template <int N, int W>
constexpr bool row1_ok() {
  return row_ok<N, W>() && Row1Cfg<N, W>::SMEM <= kMaxSmem;
}
// the row pass with per-exchange paddings (LayRowX), where they differ from
// the plain l + l/16 layout
template <int N, int W>
constexpr bool xrow_ok() {
  return RowPads<N>::n > 0 && row_ok<N, W, LayRowX<N, W>>();
}
// two-columns-per-thread variants (registers for 2E elements): E <= 8 only
template <int N, int W>
constexpr bool pair_ok() {
  return W % 4 == 0 && W <= N && N % W == 0 && Elems<N>::value <= 8 && PairCfg<N, W / 2>::NT % 32 == 0 &&
         PairCfg<N, W / 2>::NT <= 1024 && PairCfg<N, W / 2>::SMEM <= kMaxSmem;
}
// column-major variants (TPT consecutive threads per column): every pass's
// butterflies divide over TPT threads, at most 16 elements per thread, and
// with barrier groups (TPT > 32) at most 15 columns per tile
template <int N, int TPT>
constexpr bool cm_plan_ok() {
  using Rad = typename Plan<N>::R;
  for (int p = 0; p < Rad::count; ++p)
    if ((N / Rad::value[p]) % TPT != 0) return false;
  return N / TPT <= 16;
}
template <int N, int W, int TPT>
constexpr bool cm_ok() {
  return cm_plan_ok<N, TPT>() && W <= N && N % W == 0 && W % 2 == 0 && (TPT <= 32 || W <= 15) &&
         WarpCfg<N, W, TPT>::NT <= 1024 && WarpCfg<N, W, TPT>::SMEM <= kMaxSmem;
}
template <int N, int W>
constexpr bool warpcol_ok() {
  return cm_ok<N, W, 32>();
}
// the column pass with the padded (affine) exchange layout
template <int N, int W>
constexpr bool padcol_ok() {
  return col_ok<N, W>() && ColCfg<N, W, LayColPad<N, W>>::SMEM <= kMaxSmem;
}
// the plan's own threads per column, when that is more than a warp
template <int N, int W>
constexpr bool groupcol_ok() {
  return Plan<N>::TPT > 32 && cm_ok<N, W, Plan<N>::TPT>();
}
// paired-line variants (spe_pairs.cuh): sides 256, 512, 1024 (first radix 8,
// at most 8 elements per thread); WP column pairs / WR row pairs per tile
template <int N>
constexpr bool pairs_side_ok() {
  return N == 256 || N == 512 || N == 1024;
}
template <int N, int WP>
constexpr bool paircolst_ok() {
  return pairs_side_ok<N>() && WP >= 4 && N % (2 * WP) == 0 && PairColStCfg<N, WP>::NT <= 1024 &&
         PairColStCfg<N, WP>::SMEM <= kMaxSmem;
}
// TMA row pass (spe_tma.cuh): sides 256, 512, 1024 (whose tensor maps the
// engine builds), W = 2, 4, 8 rows per tile
template <int N, int W, class XLay>
constexpr bool tmarow_ok() {
  return (N == 256 || N == 512 || N == 1024) && N % W == 0 && TmaRowCfg<N, W, XLay>::NT % 32 == 0 &&
         TmaRowCfg<N, W, XLay>::NT <= 1024 && TmaRowCfg<N, W, XLay>::SMEM <= kMaxSmem;
}
template <int N, int WR>
constexpr bool pairrow_ok() {
  return pairs_side_ok<N>() && N % (2 * WR) == 0 && PairRowCfg<N, WR>::NT % 32 == 0 &&
         PairRowCfg<N, WR>::NT <= 1024 && PairRowCfg<N, WR>::SMEM <= kMaxSmem;
}
constexpr int kColWidths[3] = {4, 8, 16};
constexpr int kRowWidths[5] = {1, 2, 4, 8, 16};

// default widths (before any tuning)
template <int N>
struct DefaultTiles {  // what the autotuner picks for a population of ~32 M pixels
  static constexpr int cols = (N >= 2048) ? 4 : (N >= 512 || N == 256 ? 8 : 16);
  // (16 at side 16: two threads a row, and a CTA is whole warps)
  static constexpr int rows = (N == 16) ? 16 : (N <= 256) ? 8 : (N == 384 ? 2 : (N <= 512 ? 4 : 1));
};

// persistent grid size: the CTAs that fit on all SMs at once (occupancy
// queried once per kernel and device), never more than the tiles
template <class K>
int resident_ctas(K kern, int threads, size_t smem, std::atomic<int>* cache) {
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 64) dev = 63;
  int r = cache[dev].load(std::memory_order_acquire);
  if (r == 0) {
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, smem) != cudaSuccess || per_sm < 1)
      per_sm = 1;
    r = per_sm * sm_count();
    cache[dev].store(r, std::memory_order_release);
  }
  return r;
}

// the resident CTAs a persistent launch takes when `div` kernels share the GPU
inline int share(int slots, int div) {
  const int s = div > 1 ? slots / div : slots;
  return s < 1 ? 1 : s;
}

template <int N, int W, class Lay = LayCol<N, W>>
cudaError_t launch_cols_project(const Ctx& c) {
  using P = ColCfg<N, W, Lay>;
  auto kern = k_cols_project<N, W, Lay>;
  static std::atomic<unsigned long long> configured{0ull};
  static std::atomic<int> resident[64] = {};
  cudaError_t e = configure(kern, P::SMEM, configured);
  if (e != cudaSuccess || c.count <= 0) return e;
  const int tiles = c.count * (N / W);
  const int slots = share(resident_ctas(kern, P::NT, P::SMEM, resident), c.grid_div);
  const int grid = tiles < slots ? tiles : slots;
  return launch_pdl(kern, grid, P::NT, P::SMEM, c.st, c.T, c.A, c.ipp, c.first, c.count, c.tw);
}

template <int N, int W, int UPD, class XLay = LayPad<N, W>>
cudaError_t launch_rows_iterate(const Ctx& c, float scale, float beta, Gate g) {
  using P = RowCfg<N, W, XLay>;
  auto kern = k_rows_iterate<N, W, UPD, XLay>;
  static std::atomic<unsigned long long> configured{0ull};
  static std::atomic<int> resident[64] = {};
  cudaError_t e = configure(kern, P::SMEM, configured);
  if (e != cudaSuccess || c.count <= 0) return e;
  const int tiles = c.count * (N / W);
  const int slots = share(resident_ctas(kern, P::NT, P::SMEM, resident), c.grid_div);
  const int grid = tiles < slots ? tiles : slots;
  return launch_pdl(kern, grid, P::NT, P::SMEM, c.st, c.T, c.rho, static_cast<const int*>(c.S), c.first, c.count,
                    scale, beta, g, c.tw);
}

template <int N, int W, int UPD>
cudaError_t launch_rows_iterate1(const Ctx& c, float scale, float beta, Gate g) {
  using P = Row1Cfg<N, W>;
  auto kern = k_rows_iterate1<N, W, UPD>;
  static std::atomic<unsigned long long> configured{0ull};
  static std::atomic<int> resident[64] = {};
  cudaError_t e = configure(kern, P::SMEM, configured);
  if (e != cudaSuccess || c.count <= 0) return e;
  const int tiles = c.count * (N / W);
  const int slots = share(resident_ctas(kern, P::NT, P::SMEM, resident), c.grid_div);
  const int grid = tiles < slots ? tiles : slots;
  return launch_pdl(kern, grid, P::NT, P::SMEM, c.st, c.T, c.rho, static_cast<const int*>(c.S), c.first, c.count,
                    scale, beta, g, c.tw);
}

// ---- the blocked-scratch kernels (spe_blocked.cuh), tile codes 800 + W
template <int N>
constexpr int blocked_cols_code() {
  return Blocked<N>::ok ? 800 + Blocked<N>::BC : 0;
}
template <int N>
constexpr int blocked_rows_code() {
  return Blocked<N>::ok ? 800 + Blocked<N>::WR : 0;
}
// the list of an ER call's live row tiles, in the magnitudes' memory of its
// individuals (free during an iteration; a tile is at least two rows): length,
// counters, tiles
template <int N>
int* live_tiles(const Ctx& c) {
  return reinterpret_cast<int*>(c.M + (size_t)c.first * N * N);
}
template <int N, bool IN, bool OUT>
cudaError_t launch_cols_blocked(const Ctx& c) {
  using P = BlkCfg<N, Blocked<N>::BC, Blocked<N>::NXC>;
  auto kern = k_cols_blocked<N, IN, OUT>;
  static std::atomic<unsigned long long> configured{0ull};
  static std::atomic<int> resident[64] = {};
  cudaError_t e = configure(kern, P::SMEM, configured);
  if (e != cudaSuccess || c.count <= 0) return e;
  const int tiles = c.count * (N / Blocked<N>::BC);
  const int slots = share(resident_ctas(kern, P::NT, P::SMEM, resident), c.grid_div);
  return launch_pdl(kern, tiles < slots ? tiles : slots, P::NT, P::SMEM, c.st, c.T, c.At,
                    static_cast<const unsigned char*>(c.odd),
                    static_cast<const int*>(IN || OUT ? live_tiles<N>(c) : nullptr), c.ipp, c.first, c.count, c.tw);
}
template <int N, int UPD, bool LIST>
cudaError_t launch_rows_blocked(const Ctx& c, float scale, float beta, Gate g) {
  using P = BlkRowCfg<N>;
  static_assert(P::SMEM <= kMaxSmem, "row tile");
  auto kern = k_rows_blocked<N, UPD, LIST>;
  static std::atomic<unsigned long long> configured{0ull};
  static std::atomic<int> resident[64] = {};
  cudaError_t e = configure(kern, P::SMEM, configured);
  if (e != cudaSuccess || c.count <= 0) return e;
  const int tiles = c.count * (N / Blocked<N>::WR);
  const int slots = share(resident_ctas(kern, P::NT, P::SMEM, resident), c.grid_div);
  return launch_pdl(kern, tiles < slots ? tiles : slots, P::NT, P::SMEM, c.st, c.T, c.rho, static_cast<const int*>(c.S),
                    static_cast<const SpBits<N>*>(c.sp), static_cast<const unsigned char*>(c.odd),
                    static_cast<const int*>(LIST ? live_tiles<N>(c) : nullptr), c.first, c.count, scale, beta, g, c.tw);
}
template <int N, bool LIST>
cudaError_t launch_rows_blocked_first(const Ctx& c) {
  using P = BlkCfg<N, Blocked<N>::WR, 1>;
  auto kern = k_rows_blocked_first<N, LIST>;
  static std::atomic<unsigned long long> configured{0ull};
  cudaError_t e = configure(kern, P::SMEM, configured);
  if (e != cudaSuccess || c.count <= 0) return e;
  int* live = LIST ? live_tiles<N>(c) : nullptr;
  if (LIST && (e = cudaMemsetAsync(live, 0, (size_t)(1 + c.count) * sizeof(int), c.st)) != cudaSuccess)
    return e;
  kern<<<(unsigned)c.count * (N / Blocked<N>::WR), P::NT, P::SMEM, c.st>>>(
      c.rho, c.S, c.T, static_cast<SpBits<N>*>(c.sp), c.odd, live, c.first, c.count, c.tw);
  return cudaGetLastError();
}
template <int N>
cudaError_t launch_rows_blocked_last(const Ctx& c, float scale) {
  using P = BlkCfg<N, Blocked<N>::WR, 1>;
  auto kern = k_rows_blocked_last<N>;
  static std::atomic<unsigned long long> configured{0ull};
  cudaError_t e = configure(kern, P::SMEM, configured);
  if (e != cudaSuccess || c.count <= 0) return e;
  kern<<<(unsigned)c.count * (N / Blocked<N>::WR), P::NT, P::SMEM, c.st>>>(c.T, c.rho, c.first, scale, c.tw);
  return cudaGetLastError();
}

// ---- one cluster per individual (spe_cluster.cuh)
template <int N, int UPD>
cudaError_t launch_cluster(const Ctx& c, int iters, float scale, float beta, Gate g) {
  using P = ClusterCfg<N>;
  auto kern = k_cluster_iterate<N, UPD>;
  static std::atomic<unsigned long long> configured{0ull};
  cudaError_t e = configure(kern, P::SMEM, configured);
  if (e != cudaSuccess || c.count <= 0) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)c.count * P::CL);
  cfg.blockDim = dim3(P::NT);
  cfg.dynamicSmemBytes = P::SMEM;
  cfg.stream = c.st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim = {P::CL, 1, 1};
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kern, c.rho, static_cast<const int*>(c.S), c.A, c.ipp, c.first, iters, scale, beta,
                            g, c.tw);
}

template <int N, int WP>
cudaError_t launch_cols_pairs_st(const Ctx& c) {
  using P = PairColStCfg<N, WP>;
  auto kern = k_cols_pairs_st<N, WP>;
  static std::atomic<unsigned long long> configured{0ull};
  static std::atomic<int> resident[64] = {};
  cudaError_t e = configure(kern, P::SMEM, configured);
  if (e != cudaSuccess || c.count <= 0) return e;
  const int tiles = c.count * (N / P::W);
  const int slots = share(resident_ctas(kern, P::NT, P::SMEM, resident), c.grid_div);
  const int grid = tiles < slots ? tiles : slots;
  return launch_pdl(kern, grid, P::NT, P::SMEM, c.st, c.T, c.A, c.ipp, c.first, c.count, c.tw);
}

template <int N, int W, int UPD, class XLay>
cudaError_t launch_rows_tma(const Ctx& c, float scale, float beta, Gate g) {
  if (!c.tma || !c.err) return cudaErrorInvalidValue;  // no tensor maps for these arrays
  using P = TmaRowCfg<N, W, XLay>;
  auto kern = k_rows_tma<N, W, UPD, XLay>;
  static std::atomic<unsigned long long> configured{0ull};
  static std::atomic<int> resident[64] = {};
  cudaError_t e = configure(kern, P::SMEM, configured);
  if (e != cudaSuccess || c.count <= 0) return e;
  const int tiles = c.count * (N / W);
  const int slots = share(resident_ctas(kern, P::NT, P::SMEM, resident), c.grid_div);
  const int grid = tiles < slots ? tiles : slots;
  constexpr int slot = W == 1 ? 0 : (W == 2 ? 1 : (W == 4 ? 2 : 3));
  const RowMaps& maps = static_cast<const RowMaps*>(c.tma)[slot];
  return launch_pdl(kern, grid, P::NT, P::SMEM, c.st, maps, c.T, c.rho, c.first, c.count, scale, beta, g, c.tw,
                    c.err);
}

template <int N, int WR, int UPD>
cudaError_t launch_rows_pairs(const Ctx& c, float scale, float beta, Gate g) {
  using P = PairRowCfg<N, WR>;
  auto kern = k_rows_pairs<N, WR, UPD>;
  static std::atomic<unsigned long long> configured{0ull};
  static std::atomic<int> resident[64] = {};
  cudaError_t e = configure(kern, P::SMEM, configured);
  if (e != cudaSuccess || c.count <= 0) return e;
  const int tiles = c.count * (N / P::ROWS);
  const int slots = share(resident_ctas(kern, P::NT, P::SMEM, resident), c.grid_div);
  const int grid = tiles < slots ? tiles : slots;
  return launch_pdl(kern, grid, P::NT, P::SMEM, c.st, c.T, c.rho, static_cast<const int*>(c.S), c.first, c.count,
                    scale, beta, g, c.tw);
}

template <int N, int W>
cudaError_t launch_cols_pair(const Ctx& c) {
  using P = PairCfg<N, W / 2>;
  auto kern = k_cols_pair<N, W / 2>;
  static std::atomic<unsigned long long> configured{0ull};
  static std::atomic<int> resident[64] = {};
  cudaError_t e = configure(kern, P::SMEM, configured);
  if (e != cudaSuccess || c.count <= 0) return e;
  const int tiles = c.count * (N / W);
  const int slots = share(resident_ctas(kern, P::NT, P::SMEM, resident), c.grid_div);
  const int grid = tiles < slots ? tiles : slots;
  return launch_pdl(kern, grid, P::NT, P::SMEM, c.st, c.T, c.A, c.ipp, c.first, c.count, c.tw);
}

template <int N, int W, int TPT>
cudaError_t launch_cols_warp(const Ctx& c) {
  using P = WarpCfg<N, W, TPT>;
  auto kern = k_cols_warp<N, W, TPT>;
  static std::atomic<unsigned long long> configured{0ull};
  static std::atomic<int> resident[64] = {};
  cudaError_t e = configure(kern, P::SMEM, configured);
  if (e != cudaSuccess || c.count <= 0) return e;
  const int tiles = c.count * (N / W);
  const int slots = share(resident_ctas(kern, P::NT, P::SMEM, resident), c.grid_div);
  const int grid = tiles < slots ? tiles : slots;
  return launch_pdl(kern, grid, P::NT, P::SMEM, c.st, c.T, c.A, c.ipp, c.first, c.count, c.tw);
}

// ---- the loss passes (spe_support.cuh): one row tile or BC columns per CTA
template <class K, class... Args>
cudaError_t launch_loss(K kern, size_t smem, std::atomic<unsigned long long>& configured, int grid, int threads,
                        cudaStream_t st, Args... args) {
  cudaError_t e = configure(kern, smem, configured);
  if (e != cudaSuccess || grid <= 0) return e;
  return launch_pdl(kern, grid, threads, smem, st, args...);
}
template <int N, class L>
cudaError_t launch_loss_rows_in(const Ctx& c) {
  using P = LossRows<N>;
  static std::atomic<unsigned long long> configured{0ull};
  return launch_loss(k_loss_rows_in<N, L>, P::SMEM, configured, c.count * (N / Blocked<N>::WR), P::NT, c.st,
                     static_cast<const float2*>(c.rho), static_cast<const int*>(c.S), c.T, c.flags, c.bad, c.first,
                     c.tw);
}
template <int N, int LOSS, bool GRAD, class L, bool MARK>
cudaError_t launch_loss_cols(const Ctx& c, float eps, double* partials) {
  using P = LossCols<N>;
  auto kern = k_loss_cols<N, LOSS, GRAD, L, MARK>;
  static std::atomic<unsigned long long> configured{0ull};
  static std::atomic<int> resident[64] = {};
  cudaError_t e = configure(kern, P::SMEM, configured);
  if (e != cudaSuccess || c.count <= 0) return e;
  const int tiles = c.count * (N / Blocked<N>::BC);
  const int slots = resident_ctas(kern, P::NT, P::SMEM, resident);
  return launch_pdl(kern, tiles < slots ? tiles : slots, P::NT, P::SMEM, c.st, c.T, c.At, c.ipp,
                    static_cast<const unsigned char*>(c.flags), c.bad, c.first, c.count, eps, partials, c.tw);
}
template <int N, class L>
cudaError_t launch_loss_rows_out(const Ctx& c, float2* grad, const float* scale) {
  using P = LossRows<N>;
  static std::atomic<unsigned long long> configured{0ull};
  return launch_loss(k_loss_rows_out<N, L>, P::SMEM, configured, c.count * (N / Blocked<N>::WR), P::NT, c.st,
                     static_cast<const float2*>(c.T), static_cast<const int*>(c.S), grad, scale,
                     static_cast<const unsigned char*>(c.flags), static_cast<const unsigned*>(c.bad), c.first, c.tw);
}
template <int N, bool OUTSIDE>
cudaError_t launch_adam_rows(const Ctx& c, float2* m, float2* v, const AdamParams& ap, int fresh, int next) {
  using P = LossRows<N>;
  static std::atomic<unsigned long long> configured{0ull};
  return launch_loss(k_adam_rows<N, OUTSIDE>, P::SMEM, configured, c.count * (N / Blocked<N>::WR), P::NT, c.st, c.T,
                     static_cast<const unsigned char*>(c.flags), static_cast<const int*>(c.S), c.rho, m, v, ap, fresh,
                     next, c.first, c.tw);
}

// column-pass variant code: W > 0 one column per thread, W columns per tile;
// W < 0 two columns per thread, -W columns per tile; 100 + W one warp per
// column, 200 + W the plan's threads per column (column-major tile, barrier
// per column), 300 + W one column per thread with the padded layout, W
// columns per tile; 600 + W column pairs with split real / imaginary parts
// (spe_pairs.cuh), W columns per tile
template <int N>
cudaError_t launch_cols_w(const Ctx& c, int w) {
  switch (w) {
    case 608: if constexpr (paircolst_ok<N, 4>()) return launch_cols_pairs_st<N, 4>(c); break;
    case 616: if constexpr (paircolst_ok<N, 8>()) return launch_cols_pairs_st<N, 8>(c); break;
    case 104: if constexpr (warpcol_ok<N, 4>()) return launch_cols_warp<N, 4, 32>(c); break;
    case 108: if constexpr (warpcol_ok<N, 8>()) return launch_cols_warp<N, 8, 32>(c); break;
    case 116: if constexpr (warpcol_ok<N, 16>()) return launch_cols_warp<N, 16, 32>(c); break;
    case 304: if constexpr (padcol_ok<N, 4>()) return launch_cols_project<N, 4, LayColPad<N, 4>>(c); break;
    case 308: if constexpr (padcol_ok<N, 8>()) return launch_cols_project<N, 8, LayColPad<N, 8>>(c); break;
    case 204: if constexpr (groupcol_ok<N, 4>()) return launch_cols_warp<N, 4, Plan<N>::TPT>(c); break;
    case 208: if constexpr (groupcol_ok<N, 8>()) return launch_cols_warp<N, 8, Plan<N>::TPT>(c); break;
    case -4: if constexpr (pair_ok<N, 4>()) return launch_cols_pair<N, 4>(c); break;
    case -8: if constexpr (pair_ok<N, 8>()) return launch_cols_pair<N, 8>(c); break;
    case -16: if constexpr (pair_ok<N, 16>()) return launch_cols_pair<N, 16>(c); break;
    case 4: if constexpr (col_ok<N, 4>()) return launch_cols_project<N, 4>(c); break;
    case 8: if constexpr (col_ok<N, 8>()) return launch_cols_project<N, 8>(c); break;
    case 16: if constexpr (col_ok<N, 16>()) return launch_cols_project<N, 16>(c); break;
    default: break;
  }
  return cudaErrorInvalidValue;
}

// row-pass variant code: W rows per tile; 100 + W the per-exchange
// padding; 400 + W row pairs with split real / imaginary parts
// (spe_pairs.cuh); 500 + W / 600 + W tiles moved by the TMA (spe_tma.cuh)
// with the plain / the per-exchange padding; 700 + W one stage instead of
// two (k_rows_iterate1)
template <int N, int UPD>
cudaError_t launch_rows_w(const Ctx& c, int w, float scale, float beta, Gate g) {
  switch (w) {
    case 502: if constexpr (tmarow_ok<N, 2, LayPad<N, 2>>()) return launch_rows_tma<N, 2, UPD, LayPad<N, 2>>(c, scale, beta, g); break;
    case 504: if constexpr (tmarow_ok<N, 4, LayPad<N, 4>>()) return launch_rows_tma<N, 4, UPD, LayPad<N, 4>>(c, scale, beta, g); break;
    case 508: if constexpr (tmarow_ok<N, 8, LayPad<N, 8>>()) return launch_rows_tma<N, 8, UPD, LayPad<N, 8>>(c, scale, beta, g); break;
    case 602: if constexpr (RowPads<N>::n > 0 && tmarow_ok<N, 2, LayRowX<N, 2>>()) return launch_rows_tma<N, 2, UPD, LayRowX<N, 2>>(c, scale, beta, g); break;
    case 604: if constexpr (RowPads<N>::n > 0 && tmarow_ok<N, 4, LayRowX<N, 4>>()) return launch_rows_tma<N, 4, UPD, LayRowX<N, 4>>(c, scale, beta, g); break;
    case 608: if constexpr (RowPads<N>::n > 0 && tmarow_ok<N, 8, LayRowX<N, 8>>()) return launch_rows_tma<N, 8, UPD, LayRowX<N, 8>>(c, scale, beta, g); break;
    case 402: if constexpr (pairrow_ok<N, 1>()) return launch_rows_pairs<N, 1, UPD>(c, scale, beta, g); break;
    case 404: if constexpr (pairrow_ok<N, 2>()) return launch_rows_pairs<N, 2, UPD>(c, scale, beta, g); break;
    case 408: if constexpr (pairrow_ok<N, 4>()) return launch_rows_pairs<N, 4, UPD>(c, scale, beta, g); break;
    case 1: if constexpr (row_ok<N, 1>()) return launch_rows_iterate<N, 1, UPD>(c, scale, beta, g); break;
    case 2: if constexpr (row_ok<N, 2>()) return launch_rows_iterate<N, 2, UPD>(c, scale, beta, g); break;
    case 4: if constexpr (row_ok<N, 4>()) return launch_rows_iterate<N, 4, UPD>(c, scale, beta, g); break;
    case 8: if constexpr (row_ok<N, 8>()) return launch_rows_iterate<N, 8, UPD>(c, scale, beta, g); break;
    case 16: if constexpr (row_ok<N, 16>()) return launch_rows_iterate<N, 16, UPD>(c, scale, beta, g); break;
    case 701: if constexpr (row1_ok<N, 1>()) return launch_rows_iterate1<N, 1, UPD>(c, scale, beta, g); break;
    case 702: if constexpr (row1_ok<N, 2>()) return launch_rows_iterate1<N, 2, UPD>(c, scale, beta, g); break;
    case 704: if constexpr (row1_ok<N, 4>()) return launch_rows_iterate1<N, 4, UPD>(c, scale, beta, g); break;
    case 101: if constexpr (xrow_ok<N, 1>()) return launch_rows_iterate<N, 1, UPD, LayRowX<N, 1>>(c, scale, beta, g); break;
    case 102: if constexpr (xrow_ok<N, 2>()) return launch_rows_iterate<N, 2, UPD, LayRowX<N, 2>>(c, scale, beta, g); break;
    case 104: if constexpr (xrow_ok<N, 4>()) return launch_rows_iterate<N, 4, UPD, LayRowX<N, 4>>(c, scale, beta, g); break;
    case 108: if constexpr (xrow_ok<N, 8>()) return launch_rows_iterate<N, 8, UPD, LayRowX<N, 8>>(c, scale, beta, g); break;
    default: break;
  }
  return cudaErrorInvalidValue;
}

template <int N>
cudaError_t launch_cross_rows(const Ctx& c, const CrossArgs& a, Gate g) {
  using P = BlkCfg<N, Blocked<N>::WR, 1>;
  auto kern = k_cross_rows<N>;
  static std::atomic<unsigned long long> configured{0ull};
  cudaError_t e = configure(kern, P::SMEM, configured);
  if (e != cudaSuccess || a.count <= 0) return e;
  return launch_pdl(kern, a.per * a.count * (N / Blocked<N>::WR), P::NT, P::SMEM, c.st, a, g, c.tw);
}
template <int N, bool AVG>
cudaError_t launch_cross_cols(const Ctx& c, const CrossArgs& a) {
  using P = BlkCfg<N, Blocked<N>::BC, 1>;
  auto kern = k_cross_cols<N, AVG>;
  static std::atomic<unsigned long long> configured{0ull};
  cudaError_t e = configure(kern, P::SMEM, configured);
  if (e != cudaSuccess || a.count <= 0) return e;
  return launch_pdl(kern, a.count * (N / Blocked<N>::BC), P::NT, P::SMEM, c.st, a, c.At, c.tw);
}

#define SPE_TRY(x)                         \
  do {                                     \
    cudaError_t e_ = (x);                  \
    if (e_ != cudaSuccess) return e_;      \
  } while (0)

template <int N>
void fill_twiddles_n(float2* out, int) {
  fill_twiddles<N>(out);
}

template <int N>
struct SizeImpl {
  static float scale() { return (float)(1.0 / ((double)N * (double)N)); }

  template <int SRC>
  static OpRowsForward<SRC> rows_forward(const Ctx& c, const float2* src, float2* dst, double* partials) {
    OpRowsForward<SRC> op;
    op.first = c.first;
    op.partials = partials;
    op.rho = src;
    op.T = dst;
    return op;
  }

  // amplitudes in the order of run_pass's column passes
  static const float* amps(const Ctx& c) { return Blocked<N>::ok ? c.At : c.A; }

  static OpColsProject cols_project(const Ctx& c) {
    OpColsProject op;
    op.first = c.first;
    op.T = c.T;
    op.A = amps(c);
    op.ipp = c.ipp;
    return op;
  }

  template <int UPD>
  static cudaError_t iterate_t(const Ctx& c, int iters, float beta, Gate g, int wc, int wr) {
    SPE_TRY((launch_pass<N, AX_ROWS>(rows_forward<SRC_RHO>(c, c.rho, c.T, nullptr), c.count, c.st, c.tw)));
    for (int i = 0; i < iters; ++i) {
      SPE_TRY(launch_cols_w<N>(c, wc));
      if (i == 0 && c.mark) SPE_TRY(cudaEventRecord(c.mark, c.st));
      SPE_TRY((launch_rows_w<N, UPD>(c, wr, scale(), beta, g)));
    }
    SPE_TRY(launch_cols_w<N>(c, wc));
    if (iters == 0 && c.mark) SPE_TRY(cudaEventRecord(c.mark, c.st));
    OpRowsFinal fin;
    fin.first = c.first;
    fin.T = c.T;
    fin.out = c.rho;
    fin.scale = scale();
    return launch_pass<N, AX_ROWS>(fin, c.count, c.st, c.tw);
  }

  // the same sequence on the blocked scratch; LIVE: only the support's row
  // tiles between the ends (ER)
  template <int UPD, bool LIVE>
  static cudaError_t iterate_blocked(const Ctx& c, int iters, float beta, Gate g) {
    SPE_TRY((launch_rows_blocked_first<N, LIVE>(c)));
    for (int i = 0; i < iters; ++i) {
      SPE_TRY((i == 0 ? launch_cols_blocked<N, false, LIVE>(c) : launch_cols_blocked<N, LIVE, LIVE>(c)));
      if (i == 0 && c.mark) SPE_TRY(cudaEventRecord(c.mark, c.st));
      SPE_TRY((launch_rows_blocked<N, UPD, LIVE>(c, scale(), beta, g)));
    }
    SPE_TRY((iters == 0 ? launch_cols_blocked<N, false, false>(c) : launch_cols_blocked<N, LIVE, false>(c)));
    if (iters == 0 && c.mark) SPE_TRY(cudaEventRecord(c.mark, c.st));
    return launch_rows_blocked_last<N>(c, scale());
  }

  // wc / wr: tile codes of the column / row pass (<= 0: defaults).  The
  // defaults are the blocked-scratch kernels where the side has them and the
  // caller holds their operands (an engine does, the allocation-free entry
  // point does not)
  static cudaError_t iterate(const Ctx& c, int upd, int iters, float beta, Gate g, int wc, int wr) {
    if constexpr (ClusterCfg<N>::ok) {
      if (wc == 0 && wr <= 0 && c.count <= ClusterCfg<N>::MOST && !c.mark && c.grid_div <= 1) {
        switch (upd) {
          case 0: return launch_cluster<N, UPD_HIO>(c, iters, scale(), beta, g);
          case 1: return launch_cluster<N, UPD_RAAR>(c, iters, scale(), beta, g);
          default: return launch_cluster<N, UPD_ER>(c, iters, scale(), beta, g);
        }
      }
    }
    if constexpr (Blocked<N>::ok) {
      const bool cols = wc == 0 || wc == blocked_cols_code<N>(), rows = wr <= 0 || wr == blocked_rows_code<N>();
      if (cols && rows && c.At && c.sp && c.odd && c.M) {
        switch (upd) {
          case 0: return iterate_blocked<UPD_HIO, false>(c, iters, beta, g);
          case 1: return iterate_blocked<UPD_RAAR, false>(c, iters, beta, g);
          default:
            // live tiles: with an open gate (reality 0), and from the
            // population on whose passes have the work to hide the flags and
            // the list behind (20 iterations of a support over 25% of the rows,
            // us, live / not: 512^2 x 4 336 / 295, x 8 525 / 510, x 9 490 / 514,
            // x 16 811 / 884; 768^2 x 2 448 / 410, x 4 655 / 690; 1024^2 x 2
            // 612 / 635 but 5 iterations 191 / 187, x 3 758 / 866; 256^2 x 16
            // 319 / 290, x 33 437 / 468).  Several engines' calls at once hide
            // them sooner (512^2 x 4 190 / 207), which a call cannot know.
            return g.hi >= 3.14159f && g.lo >= 3.14159f && (size_t)c.count * N * N > (2u << 20)
                       ? iterate_blocked<UPD_ER, true>(c, iters, beta, g)
                       : iterate_blocked<UPD_ER, false>(c, iters, beta, g);
        }
      }
    }
    if (wc == 0) wc = DefaultTiles<N>::cols;
    if (wr <= 0) wr = DefaultTiles<N>::rows;
    switch (upd) {
      case 0: return iterate_t<UPD_HIO>(c, iters, beta, g, wc, wr);
      case 1: return iterate_t<UPD_RAAR>(c, iters, beta, g, wc, wr);
      default: return iterate_t<UPD_ER>(c, iters, beta, g, wc, wr);
    }
  }

  static int col_widths(int* out) {
    int k = 0;
    if constexpr (Blocked<N>::ok) out[k++] = blocked_cols_code<N>();
    if constexpr (paircolst_ok<N, 4>()) out[k++] = 608;
    if constexpr (paircolst_ok<N, 8>()) out[k++] = 616;
    if constexpr (warpcol_ok<N, 4>()) out[k++] = 104;
    if constexpr (warpcol_ok<N, 8>()) out[k++] = 108;
    if constexpr (warpcol_ok<N, 16>()) out[k++] = 116;
    if constexpr (padcol_ok<N, 4>()) out[k++] = 304;
    if constexpr (padcol_ok<N, 8>()) out[k++] = 308;
    if constexpr (groupcol_ok<N, 4>()) out[k++] = 204;
    if constexpr (groupcol_ok<N, 8>()) out[k++] = 208;
    if constexpr (pair_ok<N, 4>()) out[k++] = -4;
    if constexpr (pair_ok<N, 8>()) out[k++] = -8;
    if constexpr (pair_ok<N, 16>()) out[k++] = -16;
    if constexpr (col_ok<N, 4>()) out[k++] = 4;
    if constexpr (col_ok<N, 8>()) out[k++] = 8;
    if constexpr (col_ok<N, 16>()) out[k++] = 16;
    return k;
  }
  static int row_widths(int* out) {
    int k = 0;
    if constexpr (Blocked<N>::ok) out[k++] = blocked_rows_code<N>();
    if constexpr (tmarow_ok<N, 2, LayPad<N, 2>>()) out[k++] = 502;
    if constexpr (tmarow_ok<N, 4, LayPad<N, 4>>()) out[k++] = 504;
    if constexpr (tmarow_ok<N, 8, LayPad<N, 8>>()) out[k++] = 508;
    if constexpr (RowPads<N>::n > 0 && tmarow_ok<N, 2, LayRowX<N, 2>>()) out[k++] = 602;
    if constexpr (RowPads<N>::n > 0 && tmarow_ok<N, 4, LayRowX<N, 4>>()) out[k++] = 604;
    if constexpr (RowPads<N>::n > 0 && tmarow_ok<N, 8, LayRowX<N, 8>>()) out[k++] = 608;
    if constexpr (pairrow_ok<N, 1>()) out[k++] = 402;
    if constexpr (pairrow_ok<N, 2>()) out[k++] = 404;
    if constexpr (pairrow_ok<N, 4>()) out[k++] = 408;
    if constexpr (row1_ok<N, 1>()) out[k++] = 701;
    if constexpr (row1_ok<N, 2>()) out[k++] = 702;
    if constexpr (row1_ok<N, 4>()) out[k++] = 704;
    if constexpr (row_ok<N, 1>()) out[k++] = 1;
    if constexpr (row_ok<N, 2>()) out[k++] = 2;
    if constexpr (row_ok<N, 4>()) out[k++] = 4;
    if constexpr (row_ok<N, 8>()) out[k++] = 8;
    if constexpr (row_ok<N, 16>()) out[k++] = 16;
    if constexpr (xrow_ok<N, 1>()) out[k++] = 101;
    if constexpr (xrow_ok<N, 2>()) out[k++] = 102;
    if constexpr (xrow_ok<N, 4>()) out[k++] = 104;
    if constexpr (xrow_ok<N, 8>()) out[k++] = 108;
    return k;
  }

  static cudaError_t blur_magnitude(const Ctx& c, float sigma_ft) {
    SPE_TRY((run_pass<N, AX_ROWS>(rows_forward<SRC_RHO>(c, c.rho, c.T, nullptr), c.count, c.st, c.tw)));
    SPE_TRY((run_pass<N, AX_COLS>(cols_project(c), c.count, c.st, c.tw)));
    OpRowsModulusForward mf;
    mf.first = c.first;
    mf.T = c.T;
    mf.scale = scale();
    SPE_TRY((run_pass<N, AX_ROWS>(mf, c.count, c.st, c.tw)));
    OpColsBlur bl;
    bl.first = c.first;
    bl.T = c.T;
    bl.n = N;
    bl.sig2 = sigma_ft * sigma_ft;
    SPE_TRY((run_pass<N, AX_COLS>(bl, c.count, c.st, c.tw)));
    OpRowsMagnitude mg;
    mg.first = c.first;
    mg.partials = c.partials;
    mg.T = c.T;
    mg.M = c.M;
    return run_pass<N, AX_ROWS>(mg, c.count, c.st, c.tw);
  }

  static cudaError_t error_terms(const Ctx& c, Gate g, double* p1, double* p2, double* p3) {
    OpRowsEvaluate ev;
    ev.first = c.first;
    ev.partials = p1;
    ev.rho = c.rho;
    ev.S = c.S;
    ev.T = c.T;
    ev.T2 = c.T2;
    ev.g = g;
    SPE_TRY((run_pass<N, AX_ROWS>(ev, c.count, c.st, c.tw)));
    OpColsError ce;
    ce.first = c.first;
    ce.partials = p2;
    ce.T = c.T;
    ce.A = amps(c);
    ce.ipp = c.ipp;
    SPE_TRY((run_pass<N, AX_COLS>(ce, c.count, c.st, c.tw)));
    OpRowsRealError re;
    re.first = c.first;
    re.partials = p3;
    re.T = c.T;
    re.S = c.S;
    re.scale = scale();
    return run_pass<N, AX_ROWS>(re, c.count, c.st, c.tw);
  }

  static cudaError_t symmetry(const Ctx& c, double* psum, double* ppeak) {
    OpColsSymmetry sy;
    sy.first = c.first;
    sy.partials = psum;
    sy.T = c.T2;
    sy.A = c.band;
    sy.ipp = c.ipp;
    SPE_TRY((run_pass<N, AX_COLS>(sy, c.count, c.st, c.tw)));
    return rows_peak(c, c.T2, ppeak);
  }

  static cudaError_t rows_peak(const Ctx& c, const float2* T, double* partials) {
    OpRowsPeak pk;
    pk.first = c.first;
    pk.partials = partials;
    pk.T = T;
    pk.n = N;
    return run_pass<N, AX_ROWS>(pk, c.count, c.st, c.tw);
  }

  // ---- generic transforms over `c.count` items starting at `data` (c.first ignored)
  // (the Fourier-space crossover of the sides without blocked passes)
  static cudaError_t fft2(const Ctx& c, float2* data, int sign) {
    if constexpr (Blocked<N>::ok) {
      return cudaErrorInvalidValue;
    } else {
      if (sign > 0) {
        Ctx z = c;
        z.first = 0;
        SPE_TRY((launch_pass<N, AX_ROWS>(rows_forward<SRC_RHO>(z, data, data, nullptr), c.count, c.st, c.tw)));
        OpColsTransform<+1> ct;
        ct.first = 0;
          ct.src = data;
        ct.dst = data;
        return launch_pass<N, AX_COLS>(ct, c.count, c.st, c.tw);
      }
      OpColsTransform<-1> ct;
      ct.first = 0;
      ct.src = data;
      ct.dst = data;
      SPE_TRY((launch_pass<N, AX_COLS>(ct, c.count, c.st, c.tw)));
      OpRowsFinal fin;
      fin.first = 0;
      fin.T = data;
      fin.out = data;
      fin.scale = scale();
      return launch_pass<N, AX_ROWS>(fin, c.count, c.st, c.tw);
    }
  }

  // M[p] = |FFT+(src[p])| (2D), tmp: scratch of count items
  // (row-major where a blocked column pass has two columns: it would write the
  // magnitudes in 8-byte pieces; an average modulus of 24 of 2048^2 1328 us against
  // 1028)
  static cudaError_t ft_magnitude(const Ctx& c, const float2* src, float2* tmp, float* M) {
    Ctx z = c;
    z.first = 0;
    const auto forward = rows_forward<SRC_RHO>(z, src, tmp, nullptr);
    OpColsMagnitude cm;
    cm.src = tmp;
    cm.M = M;
    if constexpr (Blocked<N>::ok && Blocked<N>::BC < 4) {
      SPE_TRY((launch_pass<N, AX_ROWS>(forward, c.count, c.st, c.tw)));
      return launch_pass<N, AX_COLS>(cm, c.count, c.st, c.tw);
    } else {
      SPE_TRY((run_pass<N, AX_ROWS>(forward, c.count, c.st, c.tw)));
      return run_pass<N, AX_COLS>(cm, c.count, c.st, c.tw);
    }
  }

  // dst[p] = FFT+(|src[p]|) (2D)
  static cudaError_t abs_spectrum_items(const Ctx& c, const float2* src, float2* dst, double* psum) {
    Ctx z = c;
    z.first = 0;
    SPE_TRY((run_pass<N, AX_ROWS>(rows_forward<SRC_ABS_SUM>(z, src, dst, psum), c.count, c.st, c.tw)));
    OpColsTransform<+1> ct;
    ct.src = dst;
    ct.dst = dst;
    return run_pass<N, AX_COLS>(ct, c.count, c.st, c.tw);
  }

  static cudaError_t corr_peaks(const Ctx& c, const float2* D, const float2* Dref, const int* xi, const int* ri,
                                int norm_d, int norm_ref, float2* scratch1, float2* scratch2, double* part1,
                                double* part2) {
    OpColsCrossPower cp;
    cp.A = c.band;
    cp.D = D;
    cp.Dref = Dref;
    cp.xi = xi;
    cp.ri = ri;
    cp.dst = scratch1;
    cp.dst2 = scratch2;
    cp.npix = (size_t)N * N;
    cp.norm_d = norm_d;
    cp.norm_ref = norm_ref;
    SPE_TRY((run_pass<N, AX_COLS>(cp, c.count, c.st, c.tw)));
    Ctx z = c;
    z.first = 0;
    SPE_TRY(rows_peak(z, scratch1, part1));
    return rows_peak(z, scratch2, part2);
  }

  // parents' row transforms, column pass, children's rows
  static cudaError_t cross_fourier(const Ctx& c, const CrossArgs& a, Gate g) {
    if constexpr (Blocked<N>::ok) {
      SPE_TRY(launch_cross_rows<N>(c, a, g));
      k_cross_bits<N><<<dim3((N * Plan<N>::TPT + 127) / 128, (unsigned)a.count), 128, 0, c.st>>>(a);
      SPE_TRY(cudaGetLastError());
      SPE_TRY((a.per == 5 ? launch_cross_cols<N, true>(c, a) : launch_cross_cols<N, false>(c, a)));
      OpRowsChild ch;
      ch.a = a;
      ch.npix = (size_t)N * N;
      ch.scale = scale();
      ch.g = g;
      return run_pass<N, AX_ROWS>(ch, a.count, c.st, c.tw);
    } else {
      return cudaErrorInvalidValue;
    }
  }

  // partials (rows of the column pass): sum_{A>=0} |FFT+(rho)|^2, sum_{A>=0} A^2
  static cudaError_t known_power(const Ctx& c, double* partials) {
    SPE_TRY((run_pass<N, AX_ROWS>(rows_forward<SRC_RHO>(c, c.rho, c.T, nullptr), c.count, c.st, c.tw)));
    OpColsKnownPower kp;
    kp.first = c.first;
    kp.partials = partials;
    kp.T = c.T;
    kp.A = amps(c);
    kp.ipp = c.ipp;
    return run_pass<N, AX_COLS>(kp, c.count, c.st, c.tw);
  }

  // far-field loss per item into partials (column-pass tiles); with grad,
  // grad = scale[p] * 2 S FFT-(dL/dconj F) for items [first, first+count)
  // of c.rho / c.S (c.T is scratch).  Through the support's row tiles where
  // the side has blocked passes (spe_support.cuh), else row-major.
  // S * rho -> FFT+ (x) -> T; whole: row-major, every row after the column pass
  static cudaError_t support_forward(const Ctx& c, bool whole) {
    if constexpr (Blocked<N>::ok) {
      return whole ? launch_loss_rows_in<N, LossRowMajor<N>>(c) : launch_loss_rows_in<N, LossT<N>>(c);
    } else {
      OpRowsSupportForward rf;
      rf.first = c.first;
      rf.rho = c.rho;
      rf.S = c.S;
      rf.T = c.T;
      return launch_pass<N, AX_ROWS>(rf, c.count, c.st, c.tw);
    }
  }
  template <int LOSS, bool GRAD>
  static cudaError_t loss_cols(const Ctx& c, float eps, double* partials, bool whole) {
    if constexpr (Blocked<N>::ok) {
      if constexpr (GRAD) {
        if (whole) return launch_loss_cols<N, LOSS, true, LossRowMajor<N>, false>(c, eps, partials);
        if (c.bad) return launch_loss_cols<N, LOSS, true, LossT<N>, true>(c, eps, partials);
      }
      return launch_loss_cols<N, LOSS, GRAD, LossT<N>, false>(c, eps, partials);
    } else {
      OpColsLoss<LOSS, GRAD> cl;
      cl.first = c.first;
      cl.partials = partials;
      cl.T = c.T;
      cl.A = c.A;
      cl.ipp = c.ipp;
      cl.eps = eps;
      return launch_pass<N, AX_COLS>(cl, c.count, c.st, c.tw);
    }
  }
  // the last pass of the adjoint: T -> FFT- (x) -> grad = scale[p] * S * .
  static cudaError_t grad_rows(const Ctx& c, float2* grad, const float* scale, bool whole) {
    if constexpr (Blocked<N>::ok) {
      return whole ? launch_loss_rows_out<N, LossRowMajor<N>>(c, grad, scale)
                   : launch_loss_rows_out<N, LossT<N>>(c, grad, scale);
    } else {
      OpRowsGradOut go;
      go.first = c.first;
      go.T = c.T;
      go.S = c.S;
      go.G = grad;
      go.scale = scale;
      return launch_pass<N, AX_ROWS>(go, c.count, c.st, c.tw);
    }
  }
  template <int LOSS>
  static cudaError_t loss_grad_t(const Ctx& c, float eps, double* partials, float2* grad, const float* scale,
                                 int stage) {
    const bool whole = stage == GRAD_COLS || stage == GRAD_ROWS;
    if (stage == GRAD_ROWS || stage == GRAD_BACKWARD) return grad_rows(c, grad, scale, whole);
    SPE_TRY(support_forward(c, whole));
    if (!grad && stage == GRAD_ALL) return loss_cols<LOSS, false>(c, eps, partials, false);
    SPE_TRY((loss_cols<LOSS, true>(c, eps, partials, whole)));
    return stage == GRAD_ALL ? grad_rows(c, grad, scale, false) : cudaSuccess;
  }
  // loss (partials) at the current densities, then one Adam step in place
  template <int LOSS>
  static cudaError_t adam_step_t(const Ctx& c, float eps, double* partials, float2* m, float2* v,
                                 const AdamStep& a) {
    const AdamParams ap = {a.b1, a.b2, a.step_size, a.inv_sqrt_bc2, a.eps};
    if (!a.prepared) SPE_TRY(support_forward(c, false));
    SPE_TRY((loss_cols<LOSS, true>(c, eps, partials, false)));
    if constexpr (Blocked<N>::ok) {
      return a.inside ? launch_adam_rows<N, false>(c, m, v, ap, a.fresh, a.next)
                      : launch_adam_rows<N, true>(c, m, v, ap, a.fresh, a.next);
    } else {
      OpRowsGradAdam ad;
      ad.first = c.first;
      ad.T = c.T;
      ad.S = c.S;
      ad.rho = c.rho;
      ad.m = m;
      ad.v = v;
      ad.ap = ap;
      return launch_pass<N, AX_ROWS>(ad, c.count, c.st, c.tw);
    }
  }
  static cudaError_t adam_step(const Ctx& c, int loss, float eps, double* partials, float2* m, float2* v,
                               const AdamStep& a) {
    return loss == LOSS_POISSON ? adam_step_t<LOSS_POISSON>(c, eps, partials, m, v, a)
                                : adam_step_t<LOSS_AMPLITUDE>(c, eps, partials, m, v, a);
  }

  static cudaError_t loss_grad(const Ctx& c, int loss, float eps, double* partials, float2* grad,
                               const float* scale, int stage) {
    return loss == LOSS_POISSON ? loss_grad_t<LOSS_POISSON>(c, eps, partials, grad, scale, stage)
                                : loss_grad_t<LOSS_AMPLITUDE>(c, eps, partials, grad, scale, stage);
  }

  static cudaError_t block_amplitudes(const float* A, float* At, int npatterns, cudaStream_t st) {
    if constexpr (Blocked<N>::ok) {
      k_block_amplitudes<N, false><<<152 * 8, 256, 0, st>>>(A, At, npatterns, 0.f, 0.f);
      return cudaGetLastError();
    } else {
      return cudaSuccess;
    }
  }
  static cudaError_t band_table(const float* A, float* band, int n, int npatterns, float minr, float maxr,
                                cudaStream_t st) {
    if constexpr (Blocked<N>::ok) {
      k_block_amplitudes<N, true><<<152 * 8, 256, 0, st>>>(A, band, npatterns, minr, maxr);
      return cudaGetLastError();
    } else {
      return launch_band_table(A, band, n, npatterns, minr, maxr, st);
    }
  }

  static const SizeOps* table() {
    static const SizeOps t = {N,
                              Blocked<N>::ok ? N / Blocked<N>::WR : N / TileW<N>::rows,
                              Blocked<N>::ok ? N / Blocked<N>::BC : N / TileW<N>::cols,
                              TwiddleTable<N>::size(),
                              &fill_twiddles_n<N>,
                              &SizeImpl<N>::iterate,
                              &SizeImpl<N>::blur_magnitude,
                              &SizeImpl<N>::error_terms,
                              &SizeImpl<N>::symmetry,
                              &SizeImpl<N>::fft2,
                              &SizeImpl<N>::ft_magnitude,
                              &SizeImpl<N>::abs_spectrum_items,
                              &SizeImpl<N>::corr_peaks,
                              Blocked<N>::ok ? &SizeImpl<N>::cross_fourier : nullptr,
                              &SizeImpl<N>::band_table,
                              &SizeImpl<N>::col_widths,
                              &SizeImpl<N>::row_widths,
                              DefaultTiles<N>::cols,
                              DefaultTiles<N>::rows,
                              &SizeImpl<N>::known_power,
                              &SizeImpl<N>::loss_grad,
                              Blocked<N>::ok ? N / Blocked<N>::BC : N / TileW<N>::cols,
                              &SizeImpl<N>::adam_step,
                              blocked_cols_code<N>(),
                              blocked_rows_code<N>(),
                              Blocked<N>::ok ? (size_t)N * Plan<N>::TPT * sizeof(SpBits<N>) : 0,
                              &SizeImpl<N>::block_amplitudes,
                              ClusterCfg<N>::ok ? 900 : 0};
    return &t;
  }
};

}  // namespace spe

#define SPE_DEFINE_SIZE(NN) \
  namespace spe {           \
  const SizeOps* size_ops_##NN() { return SizeImpl<NN>::table(); } \
  }
