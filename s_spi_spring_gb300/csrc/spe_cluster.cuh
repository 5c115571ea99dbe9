// The iteration of a few small individuals: one thread-block cluster per
// individual, everything on chip from the first transform to the last.
//
// The two-pass kernels need two launches per iteration, and at 64^2 .. 256^2
// with few individuals a pass is a handful of CTAs whose time is latency: the
// launch, the round trip of the scratch through L2, one tile's chain of
// transforms.  Here CL CTAs hold N / CL rows each; the iterate stays in
// registers, the amplitudes and the support in shared memory, and the
// transposes between the row and the column transforms are stores into the
// other CTAs' shared memory, two cluster barriers per iteration.  Bit-identical
// to the pass kernels (the same plans, twiddles and point operations).
//
// Measured on GB300, ten RAAR iterations (passes before -> here): 128^2 x 1 76 ->
// 59 us, x 32 124 -> 84, x 48 148 -> 101 (x 64, past the rule's limit, 158 in
// passes: no more clusters fit at once); 64^2 x 1 59 -> 40, x 200 122 -> 73, x
// 1000 471 -> 305; 32^2 x 100 73 -> 41, x 1000 201 -> 115.  At 256^2 eight CTAs
// are too few for one individual (176 us against 90 in passes).  What is left
// is latency: two warps a scheduler, each transform's chain of exchanges and
// the two cluster barriers, 5 us an iteration at 128^2.
#pragma once
#include "spe_pipe.cuh"

namespace spe {

template <int N>
struct ClusterCfg {
  static constexpr bool ok = N == 32 || N == 64 || N == 128;
  // CTAs of a cluster (8: the portable size); a CTA's rows are whole warps'
  // worth of columns in the transposes
  static constexpr int CL = N == 32 ? 2 : N == 64 ? 4 : 8;
  // individuals up to which this is the faster form (above)
  static constexpr int MOST = N == 128 ? 48 : 1 << 30;
  static constexpr int MINB = N == 128 ? 3 : 6;  // resident CTAs: 85 registers a thread
  static constexpr int R = N / CL;  // rows, and columns, of a CTA
  static constexpr int TPT = Plan<N>::TPT;
  static constexpr int E = Elems<N>::value;
  static constexpr int NT = R * TPT;
  using LayR = LayPad<N, R>;
  using LayC = LayCol<N, R>;
  static constexpr int TWB = align128(TwiddleTable<N>::size() * 8);
  static constexpr int ROWS = align128(LayR::SIZE * 8);  // rows arriving from the column phase; its exchanges
  static constexpr int COLS = align128(LayC::SIZE * 8);  // columns arriving from the row phase; its exchanges
  static constexpr int AMP = R * N * 4, SUP = R * N * 4;
  static constexpr size_t SMEM = (size_t)TWB + ROWS + COLS + AMP + SUP;
};

__device__ __forceinline__ unsigned cluster_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// shared-memory address `local` of this CTA in CTA `rank` of the cluster
__device__ __forceinline__ unsigned cluster_addr(unsigned local, unsigned rank) {
  unsigned a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(local), "r"(rank));
  return a;
}
__device__ __forceinline__ void cluster_store(unsigned addr, float2 v) {
  asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(addr), "f"(v.x), "f"(v.y) : "memory");
}
// every thread of the cluster; what they stored before is visible after
__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

template <int N, int UPD>
__global__ void __launch_bounds__(ClusterCfg<N>::NT, ClusterCfg<N>::MINB)
    k_cluster_iterate(float2* __restrict__ rho, const int* __restrict__ S, const float* __restrict__ A, int ipp,
                      int first, int iters, float scale, float beta, Gate g, const float2* __restrict__ twg) {
  using C = ClusterCfg<N>;
  using LR = typename C::LayR;
  using LC = typename C::LayC;
  constexpr int NT = C::NT, E = C::E, R = C::R, TPT = C::TPT;
  static_assert(TPT <= 32 && NT % 32 == 0 && NT <= 1024 && R % 16 == 0 && C::SMEM <= 227 * 1024, "cluster shape");
  extern __shared__ __align__(128) unsigned char sm[];
  float2* tw = reinterpret_cast<float2*>(sm);
  float2* rows = reinterpret_cast<float2*>(sm + C::TWB);
  float2* cols = reinterpret_cast<float2*>(sm + C::TWB + C::ROWS);
  float* sA = reinterpret_cast<float*>(sm + C::TWB + C::ROWS + C::COLS);
  int* sS = reinterpret_cast<int*>(sA + R * N);
  load_twiddles<N>(tw, twg, NT);
  const int t = threadIdx.x;
  const int rank = (int)cluster_rank(), p = first + blockIdx.x / C::CL;
  const int l0 = rank * R;                  // the CTA's first row and column
  // row phase: row rc, positions x = elem_pos(e, rj), a row within a warp (its
  // exchanges meet at the warp); column phase: column cc, positions y =
  // elem_pos(e, cj), consecutive threads on consecutive columns
  const int rc = t / TPT, rj = t % TPT, cc = t % R, cj = t / R;
  const size_t rbase = (size_t)p * N * N + (size_t)(l0 + rc) * N;
  const float* Ap = A + (ipp > 0 ? (size_t)(p / ipp) * N * N : 0);
  const unsigned rows_s = (unsigned)__cvta_generic_to_shared(rows), cols_s = (unsigned)__cvta_generic_to_shared(cols);
  // the thread's own elements only: no barrier between these stores and reads
  float2 prev[E], v[E];
#pragma unroll
  for (int e = 0; e < E; ++e) prev[e] = rho[rbase + elem_pos<N>(e, rj)];
#pragma unroll
  for (int e = 0; e < E; ++e) {
    sS[e * NT + t] = S[rbase + elem_pos<N>(e, rj)];
    sA[e * NT + t] = __ldg(Ap + (size_t)elem_pos<N>(e, cj) * N + l0 + cc);
    v[e] = prev[e];
  }
  // FFT- is conj FFT+ conj, to the bit: one copy of each phase's transform
  // serves both directions (four copies did not fit the instruction cache, and
  // with two warps a scheduler its misses showed)
  auto conj = [&]() {
#pragma unroll
    for (int e = 0; e < E; ++e) v[e].y = -v[e].y;
  };
  // rows -> columns -> FFT+ (y) -> P_M -> FFT- (y) -> rows.  What arrives is
  // read into registers before its buffer serves the exchanges.
  auto column_phase = [&]() {
    // element x of row l0 + rc to CTA x / R
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const int x = elem_pos<N>(e, rj);
      cluster_store(cluster_addr(cols_s + 8u * (unsigned)LC::idx(l0 + rc, x % R), x / R), v[e]);
    }
    cluster_barrier();
#pragma unroll
    for (int e = 0; e < E; ++e) v[e] = cols[LC::idx(elem_pos<N>(e, cj), cc)];
    __syncthreads();
#pragma unroll 1
    for (int h = 0; h < 2; ++h) {
      fft_reg<N, LC, +1>(v, cols, tw, cc, cj);
      if (h == 0) {
#pragma unroll
        for (int e = 0; e < E; ++e) v[e] = project(v[e], sA[e * NT + t]);
      }
      conj();
    }
    // element y of column l0 + cc to CTA y / R
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const int y = elem_pos<N>(e, cj);
      cluster_store(cluster_addr(rows_s + 8u * (unsigned)LR::idx(l0 + cc, y % R), y / R), v[e]);
    }
    cluster_barrier();
#pragma unroll
    for (int e = 0; e < E; ++e) v[e] = rows[LR::idx(elem_pos<N>(e, rj), rc)];
    __syncwarp();
  };
  // no store reaches a CTA of the cluster before it has started
  cluster_barrier();
  // transform number 2 i of the rows: FFT+ of the iterate; 2 i + 1: FFT- of the
  // projected one, and its update (the last: the result)
#pragma unroll 1
  for (int h = 0;; ++h) {
    if (h & 1) conj();
    fft_pass_reg<N, TPT, +1, LR, 0, 1, SyncWarp>(v, rows, tw, rc, rj);
    if (!(h & 1)) {
      column_phase();  // (its last barrier follows the last store into another CTA)
      continue;
    }
    conj();
    if (h == 2 * iters + 1) break;
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const float2 rp = __fmul2_rn(v[e], make_float2(scale, scale));
      prev[e] = update<UPD>(rp, UPD == UPD_ER ? make_float2(0.f, 0.f) : prev[e], sS[e * NT + t], beta, g);
      v[e] = prev[e];
    }
  }
#pragma unroll
  for (int e = 0; e < E; ++e) rho[rbase + elem_pos<N>(e, rj)] = make_float2(v[e].x * scale, v[e].y * scale);
}

}  // namespace spe
