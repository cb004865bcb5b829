// gpe_line_plan.h -- host side of the run-time-length sweeps: radices, digit strides,
// butterfly tables and tile shapes of one grid side (plain C++, no CUDA types).
#pragma once
#include <algorithm>
#include <cstddef>
#include <vector>

namespace gpe {

constexpr int LINE_PMAX = 8;      // phases
constexpr int LINE_T = 256;       // most threads per block

// Transform of one line length: shared by every tile shape (plan constants).
struct LineGeo {
  int n, P;
  int r[LINE_PMAX];               // radices
  int nb[LINE_PMAX];              // butterflies per line, n / r
  int nl[LINE_PMAX];              // columns of the phase's twiddle table: product of the later radices
  int S[LINE_PMAX];               // shared-memory stride of each digit
  unsigned mg_nb[LINE_PMAX];      // ceil(2^32 / nb) (0: nb = 1)
  int span;                       // shared elements of one line
  int np[LINE_PMAX];              // product of the earlier radices (the prefixes of a butterfly)
  int rmax;                       // largest radix
  int direct;                     // prime radices 7, 11, 13 by the direct sum (as the Stockham passes)
  const void* bf[LINE_PMAX];      // p > 0: int2 {first position, prefix << 16 | column} of butterfly q
  const void* tw[LINE_PMAX];      // p < P - 1: W^(k column) as [k - 1][column], after the phase
  const void* twi[LINE_PMAX];     // p > 0: W^(a prefix) as [a - 1][prefix], before the phase
  const void* w;                  // W_n^j, then their rounding residuals (direct prime radices)
};

// Tiles of one launch.
struct LineShape {
  int L;                          // lines per tile
  unsigned mg_L;                  // ceil(2^32 / L) (0: L = 1)
  int pitch;                      // z tiles: shared elements from one line to the next
  int tpr;                        // y/x tiles per row
  int T;                          // threads
  int tiles;                      // of the launch
  int tile0;                      // its first one
};

inline unsigned line_magic(int d) { return d == 1 ? 0u : (unsigned)((0x100000000ull + d - 1) / d); }

// FP32 operations per element of a radix-r butterfly (split constants), rounded.
inline int line_radix_ops(int r) {
  static const int ops[17] = {0, 0, 2, 6, 4, 8, 8, 14, 8, 12, 12, 22, 11, 26, 19, 15, 12};
  return ops[r];
}

// Radices of n: the product of 2 to 4 factors of at most 16 with the least work, counting
// a butterfly's operations and, per phase, about 12 for its pass through shared memory and
// its twiddles; half the largest radix on top keeps them balanced (registers, and as many
// butterflies as threads in every phase).  Larger radices first: phase 0 keeps that many
// loads from HBM in flight.  False when there is none (a prime, or a factor above 13).
inline bool line_radices(int n, std::vector<int>& best) {
  best.clear();
  int best_cost = 1 << 30;
  std::vector<int> cur;
  auto search = [&](auto&& self, int m, int most, int cost) -> void {
    if (m == 1) {
      if (cur.size() >= 2 && cost + cur[0] <= best_cost) { best_cost = cost + cur[0]; best = cur; }
      return;
    }
    if (cur.size() == 4) return;
    for (int r = std::min(most, m); r >= 2; --r)
      if (m % r == 0) {
        cur.push_back(r);
        self(self, m / r, r, cost + 2 * (line_radix_ops(r) + 12));
        cur.pop_back();
      }
  };
  search(search, n, 16, 0);
  return !best.empty();
}

// Geometry of n with the given radices (two or more).
inline bool line_geometry(int n, const std::vector<int>& r, LineGeo& g) {
  if (n < 4 || n > 1024 || r.size() < 2 || r.size() > (size_t)LINE_PMAX) return false;
  g = LineGeo();
  g.n = n;
  g.P = (int)r.size();
  int later = n;
  for (int p = 0; p < g.P; ++p) {
    later /= r[p];
    g.r[p] = r[p];
    g.rmax = std::max(g.rmax, r[p]);
    g.nb[p] = n / r[p];
    g.nl[p] = later;
    g.np[p] = n / (r[p] * later);
    g.S[p] = later;
    g.mg_nb[p] = line_magic(g.nb[p]);
  }
  // lanes of a z tile's last phase are S[0] apart: odd, so that they fall in different banks
  if (g.S[0] % 2 == 0) g.S[0] += 1;
  g.span = 1;
  for (int p = 0; p < g.P; ++p) g.span += (g.r[p] - 1) * g.S[p];
  return true;
}

// {first position, prefix << 16 | column} of the butterflies of phase p > 0: q runs over the
// output digits found so far (prefix = k0 + r0 k1 + .., all there is in the last phase, where
// q is therefore the lowest frequency of the butterfly) and the input digits still to come.
inline void line_butterflies(const LineGeo& g, int p, std::vector<int>& out) {
  out.resize(2 * (size_t)g.nb[p]);
  for (int q = 0; q < g.nb[p]; ++q) {
    int prefix = q / g.nl[p];
    const int col = q % g.nl[p], key = prefix << 16 | col;
    int base = col;               // (digits after p are stored contiguously)
    for (int i = 0; i < p; ++i) { base += (prefix % g.r[i]) * g.S[i]; prefix /= g.r[i]; }
    out[2 * q] = base;
    out[2 * q + 1] = key;
  }
}

// Threads of a block with L lines: between 16 and 6 elements per thread (at most LINE_T
// threads), the multiple of 32 that leaves the fewest lanes idle over the phases' rounds
// of butterflies, the larger of equals.
inline int line_threads(const LineGeo& g, int L) {
  const int E = L * g.n;
  const int lo = std::min(LINE_T, (E / 16 + 31) / 32 * 32), hi = std::min(LINE_T, (E / 6 + 31) / 32 * 32);
  long best = 0;
  int T = std::max(32, lo);
  for (int t = T; t <= std::max(T, hi); t += 32) {
    long cost = 0;
    for (int p = 0; p < g.P; ++p) {
      const long total = (long)L * g.nb[p], rounds = (total + t - 1) / t;
      cost += rounds * t * (line_radix_ops(g.r[p]) + 12) * g.r[p];
    }
    if (!best || cost <= best) { best = cost; T = t; }
  }
  return T;
}

// At least a block per SM where the grid has them.  (Two per SM were smaller blocks with more
// partial sums to finish: 35^3 complex64 imaginary time 37.8 -> 33.1 us per step, 60^3 48.9
// -> 40.4; half a block per SM 38.8 and 37.9, larger sides the same.)
constexpr int LINE_TILES_MIN = 148;

// z tiles: about 32 KB of consecutive lines, fewer while that leaves SMs without a block.
inline LineShape line_shape_z(const LineGeo& g, int csize) {
  LineShape s = LineShape();
  const int n = g.n;
  s.L = std::max(1, std::min(32, 32768 / (n * csize)));
  while (s.L > 1 && (n * n + s.L - 1) / s.L < LINE_TILES_MIN) s.L = (s.L + 1) / 2;
  s.tiles = (n * n + s.L - 1) / s.L;
  s.tpr = 1;
  s.mg_L = line_magic(s.L);
  // phase 0 writes runs of nb[0] positions per line: consecutive lanes keep consecutive
  // banks across a line's end when pitch = nb[0] modulo the banks
  const int banks = 128 / csize;
  s.pitch = g.span;
  while ((s.pitch - g.nb[0]) % banks) ++s.pitch;
  s.T = line_threads(g, s.L);
  return s;
}

// y/x tiles: 128-byte rows (balanced over a row of the cube), half of that where the tile
// would pass 72 KB; down to 32-byte sectors while SMs are left without a block.
inline LineShape line_shape_p(const LineGeo& g, int csize) {
  LineShape s = LineShape();
  const int n = g.n, least = 32 / csize;
  int most = 128 / csize;
  while (most > least && (long)g.span * most * csize > 72 * 1024) most /= 2;
  while (most > least && (long)n * ((n + most - 1) / most) < LINE_TILES_MIN) most /= 2;
  int tpr = (n + most - 1) / most;
  s.L = (n + tpr - 1) / tpr;
  s.L = std::min(n, (s.L + least - 1) / least * least);
  s.tpr = (n + s.L - 1) / s.L;
  s.tiles = n * s.tpr;
  s.mg_L = line_magic(s.L);
  s.T = line_threads(g, s.L);
  return s;
}

constexpr size_t LINE_HIST = 16 * 1024;   // shared memory for copies of the shell histogram

// dynamic shared memory: tile, per-line tables, reduction scratch, `bins` doubles of histograms
inline size_t line_smem(const LineGeo& g, const LineShape& s, int csize, bool z, int bins) {
  return (size_t)(z ? s.L * s.pitch : g.span * s.L) * csize + ((size_t)s.L * 24 + 15) / 16 * 16 + 32 * 4 * 16 +
         (size_t)bins * sizeof(double);
}

}  // namespace gpe
