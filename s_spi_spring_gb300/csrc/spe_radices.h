// Radices of the run-time transforms (spe_size_any.cu).  Host code.
#pragma once
#include <algorithm>
#include <map>
#include <utility>

namespace spe {

constexpr int kMaxRadices = 24;

// Shared-memory wavefronts per 32 elements of a pass of radix R after passes of
// product NS (any_pass_r): a half-warp's 8-byte accesses take one for every
// address that its fullest of 16 banks holds.  The inputs are consecutive; the
// outputs lie R or NS apart and the twiddles n / (NS R) r, which with powers of 2
// is up to 8 or 16 to a bank.  Counted on two warps of a tile of 8 lines.
inline double pass_wavefronts(int n, int NS, int R) {
  const int LS = n | 1, m = n / R, step = n / (NS * R), warps = (8 * m + 31) / 32;
  const int samples = warps < 2 ? 1 : 2;
  int total = 0;
  for (int s = 0; s < samples; ++s)
    for (int h = 0; h < 2; ++h) {
      const int i0 = s * (warps / samples) * 32 + h * 16, lanes = std::min(16, 8 * m - i0);
      // the wavefronts of one access: address(line, butterfly of the line)
      auto access = [&](auto&& address) {
        int at[16], most = 0, full[16] = {};
        for (int l = 0; l < lanes; ++l) {
          at[l] = address((i0 + l) / m, (i0 + l) % m);
          bool seen = false;
          for (int k = 0; k < l; ++k) seen |= at[k] == at[l];
          if (!seen) most = std::max(most, ++full[at[l] % 16]);
        }
        return most;
      };
      total += lanes > 0 ? R : 0;
      for (int r = 0; r < R; ++r) {
        total += access([&](int c, int b) { return c * LS + b / NS * (NS * R) + b % NS + r * NS; });
        if (NS > 1 && r > 0) total += access([&](int, int b) { return b % NS * step * r; });
      }
    }
  return (double)total * warps / samples / (8.0 * n / 32.0);
}

// The radices 2 .. 10, in order, of `smooth` (a factor of n with primes up to 7)
// whose passes take the fewest wavefronts, with four for a pass's barrier and
// half a one for each element that a thread waits for (a single individual at
// 144: 91 us in 9 x 8 x 2, 82 in 6 x 4 x 6).  The times follow the count: 8
// iterations of 6 M pixels at 896 take 1306 us with 38 wavefronts, 1338 with 41,
// 1368 with 45, 1522 with 54.  The fewest radices alone do not give it: 8 x 7 x 4
// x 4 at 896 and 8 x 6 x 5 x 4 at 960 take 1522 and 1577 us, radices 8, 4 and the
// primes 1311 and 1379, 4 x 8 x 4 x 7 and 5 x 8 x 8 x 3 1251 and 1255.
inline int choose_radices(int n, int smooth, int* rad) {
  std::map<int, std::pair<double, int>> best;  // product so far -> (wavefronts, last radix)
  best[1] = {0.0, 0};
  for (auto it = best.begin(); it != best.end(); ++it)
    for (int R = 2; R <= 10; ++R) {
      const int NS = it->first;
      if (smooth % ((long long)NS * R) != 0) continue;
      const double w = it->second.first + pass_wavefronts(n, NS, R) + 4.0 + 0.5 * R;
      auto& to = best[NS * R];  // (above NS in the map's order: visited later)
      if (to.second == 0 || w < to.first) to = {w, R};
    }
  int k = 0;
  for (int NS = smooth; NS > 1; NS /= best[NS].second) {
    if (k == kMaxRadices) return 0;
    rad[k++] = best[NS].second;
  }
  std::reverse(rad, rad + k);
  return k;
}

}  // namespace spe
