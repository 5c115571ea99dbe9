// Internal declarations shared by the engine's translation units.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include <random>
#include <vector>

namespace spe {

// Stages of the far-field loss gradient (SizeOps::loss_grad): all of it; up to
// the column pass, and the row pass, through a whole row-major T; the same two
// through T and the flags as they are (Ctx::flags, bad).
enum { GRAD_ALL = 0, GRAD_COLS = 1, GRAD_ROWS = 2, GRAD_FORWARD = 3, GRAD_BACKWARD = 4 };

// Host pattern encoding (spe_host.cpp).
int prepare_pattern(const float* in, int n, int cx, int cy, bool use_bounds, float* out);

// Random draws of one crossover child (Solver::Crossover, src/solver.cpp:750-801).
struct ChildDraw {
  int p1, p2, p3;    // parent indices (p1 through the error order)
  int cft;           // Fourier-space crossover
  int ssx, ssy;      // cell sizes
  int csx, csy;      // crossmap cells
  int ox, oy;        // offsets
  float rot;         // rotation angle
  int cmap;          // offset of the child's crossmap in the crossmap pool
};
// Draws all children in the reference's order from generator g.  Returns
// non-zero if a cell size would fall below one pixel.
int draw_children(std::mt19937& g, int count, const int* order, float suppdim, int n, float crossbalance,
                  float crossexp, float crossftin, std::vector<ChildDraw>& out, std::vector<int>& cmaps);

// Random draws of one starting individual (Solver::Initialize_rec,
// src/solver.cpp:880-906): disc items of radius sigma at (cx, cy) inside the
// support box, with a phase each; the modulus exponent and the scaling.
struct InitItem {
  float sigma, cx, cy, phase;
};
struct InitDraw {
  int first_item, nitems;
  float exponent, scaling;
};
void draw_init(std::mt19937& g, int count, int support_size, const float itemsize[2], const int nitems[2],
               const float exponent[2], const float scaling[2], float phase, std::vector<InitDraw>& inds,
               std::vector<InitItem>& items);

// Everything a size-specialised sequence needs about one call.
struct Ctx {
  int n;
  int first, count;
  cudaStream_t st;
  float2* rho;          // population density
  int* S;               // population support
  float2* T;            // scratch, one complex array per individual
  float2* T2;           // second scratch (evaluate / alignment)
  float* M;             // magnitudes (shrink-wrap)
  const float* A;       // amplitudes, n*n
  const float2* tw;     // exp(+2 pi i m / n), m < n
  double* partials;     // per-CTA reduction slots
  double* red;          // per-individual reduced values, count * 4 * slots
  int grid_div;         // persistent kernels use 1/grid_div of the resident CTAs (<= 1: all)
  cudaEvent_t mark;     // if set, recorded after the first column pass of an iteration call
  int ipp;              // individuals per pattern (slot p uses pattern p / ipp of A); 0: A is one pattern
  const void* tma;      // tensor maps of the TMA row pass (row_maps), or null
  int* err;             // device flag set by a bounded wait that gave up, or null
  // operands of the blocked-scratch kernels (spe_blocked.cuh), or null: the
  // amplitudes in register order, the packed support and its per-row-tile flags
  const float* At;
  const float* band;  // weights of the correlation ops (SizeOps::band_table)
  void* sp;
  unsigned char* odd;
  // marks of the loss passes: row tiles with support, and per individual
  // whether the column-transformed gradient is not finite (bad null: not marked,
  // for a caller that updates nothing outside the support)
  unsigned char* flags;
  unsigned* bad;
};

// One gathered, shifted copy of an individual (reference shift kernel,
// gpu_context.cu:1329-1357, as a gather: destination pixel d reads the source
// pixel that the reference's scatter writes to d), optionally gated by
// apply_support_er with the shifted support (gpu_context.cu:519-537).
struct ShiftItem {
  int src;       // source density slot (in the source pool)
  int dst;       // destination density slot
  int ssrc;      // source support slot or -1
  int sdst;      // destination support slot or -1
  int sx, sy;    // shift
  float pc, ps;  // cosine and sine of the added phase
  int flip;      // point reflection (twin image)
  int polar;     // 0: plain copy (no shift, flip or phase)
  int gate;      // apply the phase/support gate with the (shifted) support
  int gsrc;      // gate with support slot gsrc of the source support pool when no ssrc (-1: none)
};

// One child of the crossover (reference cross_density / cross_density_real /
// cross_support, gpu_context.cu:1699-1883)
struct CrossChild {
  int cft;           // Fourier-space crossover
  int csx, csy;      // crossmap cells
  int ssx, ssy;      // cell sizes
  int ox, oy;        // offsets
  float rot;         // rotation angle
  int cmap;          // offset of the crossmap in the crossmap pool
  int w;             // work index
  int p1;            // slot of parent 1 (its support is S1)
  int self, dst;     // slots of the child's own parent and of the child
};

// Operands of the crossover's kernels.  Work arrays of child w: W[per w + k],
// k = 0 self', 1 p1, 2 p2', 3 p3', 4 avg' (per = 5; 4 where the average is not
// used); Ws[3 w + k], k = 0 S', 1 S2', 2 S3'; C[w] the child.
struct CrossArgs {
  const float2* rho;   // source pool
  const int* S;
  float2* rho_out;     // the population that the children join
  int* S_out;
  const ShiftItem* items;    // per w + k
  const CrossChild* children;  // in work order
  float2* W;
  int* Ws;
  float2* C;
  unsigned char* bits;  // crossed pixels in column-pass order, one byte or 16-bit word per thread
  const int* cmaps;
  int cmap_total;
  const float* avg_mod;
  int per, count;       // count children from work index 0
  float crossdiff, use_average;
  int crosssym, update_support;
};

// One Adam step (SizeOps::adam_step).  On sides with blocked passes a run of
// steps may leave out what it knows: prepared (Ctx::T holds the forward row
// pass: the step before had `next`), fresh (the moments are 0 and not read),
// inside (the moments outside the support are 0 and stay 0), next (leave the
// updated densities' forward row pass in Ctx::T).
struct AdamStep {
  float b1, b2, step_size, inv_sqrt_bc2, eps;
  int prepared, fresh, inside, next;
};

// Tensor maps of the TMA row pass (spe_tma_maps.cu): row_maps_bytes() of
// storage holding one set of maps (T, rho, S) per row-tile width 1, 2, 4, 8.
// build_row_maps fills them for population arrays of `cap` individuals of
// side n; false when the side has no TMA row pass or the driver lacks
// cuTensorMapEncodeTiled.
size_t row_maps_bytes();
// the self-test kernel of the bounded waits (spe_tma.cuh): sets *err after
// its wait gives up
cudaError_t launch_wait_selftest(int* err, cudaStream_t st);
bool build_row_maps(void* out, int n, int cap, const float2* T, const float2* rho, const int* S);

// One reduction over per-CTA partials (k_reduce): component k of every tile's
// partial, kind 0 sum, 1 maximum, 2 argmax of (value, index)
struct RedJob {
  const double* part;
  int tpi, k, kind, slot;
};
struct RedJobs {
  RedJob job[8];
};

// Phase gate (see phase_out in spe_kernels.cuh): float thresholds of
// arg > hi / arg < -lo and the cos / sin of each threshold.
struct Gate {
  float hi, lo;
  float chi, shi;
  float clo, slo;
};

// Size-specialised operation table (one per compiled pattern size).
struct SizeOps {
  int n;
  int tiles_rows;  // CTAs per individual of a row pass
  int tiles_cols;  // CTAs per individual of a column pass
  int tw_size;     // twiddle table entries
  void (*fill_tw)(float2*, int n);  // tw_size entries for side n
  // upd: 0 HIO, 1 RAAR, 2 ER; wc / wr: tile widths of the column / row
  // pass of the iteration kernels (<= 0: defaults)
  cudaError_t (*iterate)(const Ctx&, int upd, int iterations, float beta, Gate g, int wc, int wr);
  // blurred modulus into M, per-CTA max into partials
  cudaError_t (*blur_magnitude)(const Ctx&, float sigma_ft);
  // error terms: stage 1 -> p1 (modulesum), stage 2 -> p2 (err, norm, max),
  // stage 3 -> p3 (err_r, norm_r); leaves |rho|'s row transforms in Ctx::T2
  cudaError_t (*error_terms)(const Ctx&, Gate g, double* p1, double* p2, double* p3);
  // the two peaks of the symmetry metric (get_symmetry), after error_terms and
  // from what it left in Ctx::T2, with the weights Ctx::band: column-pass partials (the sum whose square is the
  // first peak) and row-pass partials (value, index of the second)
  cudaError_t (*symmetry)(const Ctx&, double* psum, double* ppeak);
  // generic transforms over Ctx::count items starting at the given arrays
  // in-place 2D transform; sign +1: FFT+ unnormalised, -1: FFT- then /N^2
  cudaError_t (*fft2)(const Ctx&, float2* data, int sign);
  // M = |FFT+(src)| (tmp: scratch items)
  cudaError_t (*ft_magnitude)(const Ctx&, const float2* src, float2* tmp, float* M);
  // dst = FFT+(|src|) (in the passes' own order), the complex sums of src in
  // row-pass partials
  cudaError_t (*abs_spectrum_items)(const Ctx&, const float2* src, float2* dst, double* psum);
  // peaks (value, index) of |FFT-(cross power of D[xi[p]], Dref[ri[p]])|^2
  // with the weights Ctx::band: conj(D) Dref in part1, D Dref in part2.  D and
  // Dref come from abs_spectrum_items; scratch1, scratch2: count items each
  cudaError_t (*corr_peaks)(const Ctx&, const float2* D, const float2* Dref, const int* xi, const int* ri,
                            int norm_d, int norm_ref, float2* scratch1, float2* scratch2, double* part1,
                            double* part2);
  // Fourier-space children from gathered parents to population slots
  // (CrossArgs; the amplitudes of Ctx), or null where the side has no blocked
  // passes
  cudaError_t (*cross_fourier)(const Ctx&, const CrossArgs&, Gate g);
  // band-pass weights of the correlation ops for `npatterns` patterns
  cudaError_t (*band_table)(const float* A, float* band, int n, int npatterns, float minr, float maxr,
                            cudaStream_t st);
  // tile widths compiled for this size
  int (*col_widths)(int* out);
  int (*row_widths)(int* out);
  int default_cols, default_rows;  // 0 for sides without a compiled plan
  // partials of the column pass: sum over A >= 0 of |FFT+(rho)|^2 and A^2
  cudaError_t (*known_power)(const Ctx&, double* partials);
  // far-field loss (0 amplitude, 1 Poisson) of items [first, first+count) of
  // Ctx::rho / Ctx::S into column-pass partials; with grad, the adjoint
  // gradient times scale[item] (scale may be null).  stage GRAD_COLS stops
  // after the column pass (the column-transformed gradient left in Ctx::T);
  // GRAD_ROWS runs only the last pass, from Ctx::T into grad (which may be
  // Ctx::T: every row is read whole before it is written)
  cudaError_t (*loss_grad)(const Ctx&, int loss, float eps, double* partials, float2* grad, const float* scale,
                           int stage);
  int loss_tiles;  // loss partials per item
  // loss at the current densities into partials, then one Adam step in
  // place with moments m, v (see OpRowsGradAdam)
  cudaError_t (*adam_step)(const Ctx&, int loss, float eps, double* partials, float2* m, float2* v,
                           const AdamStep& a);
  // blocked-scratch kernels of the iteration (0 / null: none at this side):
  // the tile codes of the column and the row pass, the bytes of packed
  // support per individual, and the amplitudes' reordering
  int blocked_cols, blocked_rows;
  size_t sp_bytes;
  cudaError_t (*block_amplitudes)(const float* A, float* At, int npatterns, cudaStream_t st);
  // tile code of the default where that is a cluster per individual, else 0
  int cluster;
};

const SizeOps* size_ops(int n);
// sides without a compiled plan (spe_size_any.cu): the table of side n, or
// null when n has a prime factor above the accepted bound or its lines do
// not fit in shared memory
const SizeOps* size_ops_any(int n);

}  // namespace spe
