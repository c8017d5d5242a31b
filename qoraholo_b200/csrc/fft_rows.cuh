// Tiles of rows on the two-factor line transforms (fft_two.cuh): `lines` rows per CTA, R2 threads each.
#pragma once

#include "fft_two.cuh"

namespace qhk {
namespace twofft {

// Slots of a tile of rows: consecutive threads are consecutive j of a line (first pass) or consecutive k1
// (second pass), so B = 1 and A is odd; lines are C apart, with C congruent to the number of threads per
// line modulo the 16 two-bank slots where a half-warp spans several lines.
__host__ __device__ __forceinline__ int row_line_pitch(const Factors& f) {
  const int need = f.r1 * (f.r2 | 1);
  const int want = f.r2 < 16 ? f.r2 : f.r1;
  return need + ((want - need) % 16 + 16) % 16;
}

// A thread's butterflies. The threads of the last warp beyond lines * R2 have none.
struct RowTile {
  int line, j;      // first pass: line and butterfly
  int line2, j2;    // second pass
  bool first, second;
};
__device__ __forceinline__ RowTile row_tile(const Factors& f, int lines) {
  RowTile r;
  const int t = static_cast<int>(threadIdx.x);
  r.line = t / f.r2;
  r.j = t - r.line * f.r2;
  r.first = r.line < lines;
  r.line2 = t / f.r1;
  r.j2 = t - r.line2 * f.r1;
  r.second = r.line2 < lines;
  return r;
}

// The launch of `total_lines` lines: about 256 threads per CTA, within 64 KB of shared memory; `staged`: a
// natural-order copy of every line (n + 1 values) beside the exchange.
struct RowLaunch {
  int lines, threads;
  std::size_t smem;
  unsigned grid;
};
inline RowLaunch row_launch(const Factors& f, std::size_t total_lines, bool staged) {
  const std::size_t line = (row_line_pitch(f) + (staged ? f.n() + 1 : 0)) * sizeof(float2);
  RowLaunch r;
  r.lines = 256 / f.r2;
  while (r.lines > 1 && r.lines * line > 64 * 1024) --r.lines;
  r.threads = (r.lines * f.r2 + 31) / 32 * 32;
  r.smem = r.lines * line;
  r.grid = static_cast<unsigned>((total_lines + r.lines - 1) / r.lines);
  return r;
}

}  // namespace twofft
}  // namespace qhk
