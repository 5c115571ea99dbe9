// Layouts of the population operations' workspace: one allocation, carved into
// 256-byte aligned pieces.
#pragma once
#include <cuda_runtime.h>

#include <cstddef>

#include "spe_internal.h"

namespace spe_detail {

// Pieces of `cap` bytes at `p`; with p null it only counts (`used`: what the
// pieces take so far).  After the last take `fits` tells whether all lie inside.
struct Carve {
  char* p;
  size_t cap;
  size_t used = 0;
  template <class T>
  T* take(size_t n) {
    used = (used + 255) & ~size_t(255);
    T* r = p ? reinterpret_cast<T*>(p + used) : nullptr;
    used += n * sizeof(T);
    return r;
  }
  bool fits() const { return used <= cap; }
};

// spe_crossover for P individuals of npix pixels (nred doubles of row-pass
// partials each): `pairs` alignments and `per` gathered parents a child, ncmaps
// crossmap cells.
// The same list of takes measures the workspace and carves it.
struct CrossWork {
  float2* D;        // spectra of the members and the average
  float2* scratch;  // correlations
  float2* W;        // parents of the children (before: scratch of the second product)
  float2* C;        // children
  int* Ws;          // shifted supports, three a child
  double *part, *part2, *psum, *peaks, *sums;
  int *xi, *ri;
  spe::ShiftItem* items;
  spe::CrossChild* children;
  unsigned char* bits;
  int* cmaps;
  CrossWork(Carve& cv, size_t P, size_t npix, size_t nred, int pairs, int per, size_t ncmaps) {
    const size_t n = P * pairs;
    D = cv.take<float2>((P + 1) * npix);
    scratch = cv.take<float2>(n * npix);
    W = cv.take<float2>(P * per * npix);
    C = cv.take<float2>(P * npix);
    Ws = cv.take<int>(3 * P * npix);
    part = cv.take<double>(n * nred);
    part2 = cv.take<double>(n * nred);
    psum = cv.take<double>((P + 1) * nred);
    peaks = cv.take<double>(n * 4);
    sums = cv.take<double>((P + 1) * 2);
    xi = cv.take<int>(n);
    ri = cv.take<int>(n);
    items = cv.take<spe::ShiftItem>(P * per);
    children = cv.take<spe::CrossChild>(P);
    bits = cv.take<unsigned char>(P * npix / 4);
    cmaps = cv.take<int>(ncmaps + 1);
  }
  static size_t bytes(size_t P, size_t npix, size_t nred, int pairs, int per, size_t ncmaps) {
    Carve cv{nullptr, 0};
    CrossWork(cv, P, npix, nred, pairs, per, ncmaps);
    return cv.used;
  }
};

}  // namespace spe_detail
