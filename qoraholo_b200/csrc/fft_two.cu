// FFT passes on the two-factor line transforms (fft_two.cuh): axis passes (tiles of columns) and row
// passes (real rows as half-length lines) for every length that is a product of two radices, at most
// 16 and at most 32. The first DFT of a line takes its values straight from global memory and the last one
// stores straight to it, so a transform costs one exchange through shared memory, where the staged engine
// (fft_engine.cuh) goes through it once per radix pass and twice more for the load and the store.
//
// What bounds these passes is HBM (or L2) latency and bandwidth: a tile's loads are all issued at once
// (16 to 32 per thread) and several CTAs share an SM, so one CTA's loads overlap another's transforms.
// Measured on B200 against the staged passes: half spectrum of 384^3, y passes 89 and 95 us (5.1 and 4.8 TB/s) from
// 171, z pass with the restore 196 us from 319; of 8 x 96^3, y 13 us from 33, z 19 us from 61; complex rows of
// 97 x 384^2 52 us from 97. 64, 128 and 256, with a compile-time form on the register engine (fft_reg.cu), stay
// there: 256^3 z with the restore 47 us against 54 here, y 26 against 25.
#include "debug.cuh"
#include "fft_rows.cuh"
#include "fft_two.hpp"

namespace qhk {

namespace {

using twofft::Factors;
using twofft::row_launch;
using twofft::row_line_pitch;
using twofft::row_tile;
using twofft::RowLaunch;
using twofft::RowTile;

// CTAs per SM to leave registers for, at 256 threads each (axis tiles are 16 columns of at most 16 threads or 8
// columns of at most 32, row tiles 256 threads): three of 80 registers where the radices fit them (the restore of
// 8 x 96^3 too: 19.1 us, in two CTAs 22.3), two of 128 for larger radices. The restore of second factors up to 24
// runs in three CTAs of 192 threads (384^3: 196 us, in two of 256 223).
constexpr int min_blocks(int max) { return max == twofft::kSmall ? 3 : 2; }

constexpr bool restores(int mode) {
  return mode == static_cast<int>(AxisMode::restore_half) || mode == static_cast<int>(AxisMode::restore_mask);
}
constexpr int axis_threads(int mode, int max) { return restores(mode) && max == twofft::kMid ? 192 : 256; }

// ---- axis passes ------------------------------------------------------------------------------------

// COLS = 1 << logc consecutive columns of one outer slice per CTA; COLS * R2 threads (R2 >= R1).
template <bool Fwd, int Mode, int Max>
__global__ void __launch_bounds__(axis_threads(Mode, Max), axis_threads(Mode, Max) == 192 ? 3 : min_blocks(Max))
    k_axis_two(float2* __restrict__ data, std::size_t so, std::size_t sp, int ni, Factors f, int logc,
               const float2* __restrict__ tw, float scale, const float2* __restrict__ aux_a,
               const std::uint8_t* __restrict__ aux_h, std::size_t sb) {
  extern __shared__ float2 xs[];
  constexpr int kFrom = static_cast<int>(AxisMode::from_data);
  constexpr int kHalf = static_cast<int>(AxisMode::restore_half);
  const int cols = 1 << logc;
  const int A = (f.r2 | 1) << logc, B = cols;
  if (!QHK_CHECK((static_cast<std::size_t>(f.r1) * A + (restores(Mode) ? f.n() * cols : 0)) * sizeof(float2) <=
                     debug::dynamic_smem_bytes() &&
                 static_cast<int>(blockDim.x) == f.r2 * cols)) {
    return;  // block-uniform
  }
  const int t = static_cast<int>(threadIdx.x);
  const int c = t & (cols - 1);
  const int j = t >> logc;  // butterfly of the first pass; j < R1 also has one of the second
  const int col = (static_cast<int>(blockIdx.x) << logc) + c;
  const bool live = col < ni;
  const std::size_t base =
      static_cast<std::size_t>(blockIdx.z) * sb + static_cast<std::size_t>(blockIdx.y) * so + (live ? col : 0);
  twofft::with_first<Max>(f.r1, [&]<int R>() {
    float2 v[R];
    const float2* p = (Mode == kFrom ? aux_a : data) + base + static_cast<std::size_t>(j) * sp;
    const std::size_t step = static_cast<std::size_t>(f.r2) * sp;
#pragma unroll
    for (int q = 0; q < R; ++q, p += step) v[q] = live ? *p : make_float2(0.0f, 0.0f);
    if constexpr (Mode == kFrom) {
#pragma unroll
      for (int q = 0; q < R; ++q) v[q] = cscale(v[q], scale);
    }
    twofft::first_pass<R, Fwd>(v, j, tw, xs + j * B + c, A);
  });
  const bool second = j < f.r1;
  if constexpr (restores(Mode)) {
    twofft::with_radix<Max>(f.r2, [&]<int R>() {
      // The restore's data a streams into shared memory (cp.async, read back by the same thread) while
      // the first pass finishes; the hit counts wait packed four to a register.
      float2* as = xs + f.r1 * A + t;
      const int pitch = f.r1 << logc;
      unsigned hp[(R + 3) / 4] = {};
      if (second && live) {
        std::size_t g = base + static_cast<std::size_t>(j) * sp;
        const std::size_t step = static_cast<std::size_t>(f.r1) * sp;
#pragma unroll
        for (int q = 0; q < R; ++q, g += step) {
          asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(static_cast<unsigned>(
                           __cvta_generic_to_shared(as + q * pitch))),
                       "l"(aux_a + g)
                       : "memory");
          hp[q / 4] |= static_cast<unsigned>(aux_h[g]) << (8 * (q % 4));
        }
      }
      asm volatile("cp.async.commit_group;\n" ::: "memory");
      __syncthreads();
      asm volatile("cp.async.wait_all;\n" ::: "memory");
      if (second) {
        float2 u[R];
        float2* x = xs + j * A + c;
        twofft::second_pass<R, true>(u, x, B);
#pragma unroll
        for (int q = 0; q < R; ++q) {
          const float2 a = live ? as[q * pitch] : make_float2(0.0f, 0.0f);
          const unsigned h = (hp[q / 4] >> (8 * (q % 4))) & 0xffu;
          if constexpr (Mode == kHalf) {
            const float w = 1.0f - 0.5f * static_cast<float>(h);
            u[q] = make_float2((a.x + w * u[q].x) * scale, (a.y + w * u[q].y) * scale);
          } else {
            if (h) u[q] = a;
          }
        }
        twofft::first_pass<R, false>(u, j, tw, x, B);  // the inverse, factors exchanged, into the same slots
      }
    });
    __syncthreads();
    if (!live) return;
    twofft::with_first<Max>(f.r1, [&]<int R>() {
      float2 v[R];
      twofft::second_pass<R, false>(v, xs + j * B + c, A);
      float2* p = data + base + static_cast<std::size_t>(j) * sp;
      const std::size_t step = static_cast<std::size_t>(f.r2) * sp;
#pragma unroll
      for (int q = 0; q < R; ++q, p += step) *p = v[q];
    });
  } else {
    __syncthreads();
    if (!second || !live) return;
    twofft::with_radix<Max>(f.r2, [&]<int R>() {
      float2 u[R];
      twofft::second_pass<R, Fwd>(u, xs + j * A + c, B);
      float2* p = data + base + static_cast<std::size_t>(j) * sp;
      const std::size_t step = static_cast<std::size_t>(f.r1) * sp;
      const float s = Mode == static_cast<int>(AxisMode::plain) ? scale : 1.0f;
#pragma unroll
      for (int q = 0; q < R; ++q, p += step) *p = s != 1.0f ? cscale(u[q], s) : u[q];
    });
  }
}

template <bool Fwd, int Mode, int Max>
void launch_axis_two(const Factors& f, int cols, float2* data, int n_outer, std::size_t so, std::size_t sp, int ni,
                     float scale, const AxisAux& aux, int batch, std::size_t sb, cudaStream_t s) {
  const std::size_t slots = static_cast<std::size_t>(f.r1) * (f.r2 | 1) * cols;
  const std::size_t smem = (slots + (restores(Mode) ? static_cast<std::size_t>(f.n()) * cols : 0)) * sizeof(float2);
  auto kernel = k_axis_two<Fwd, Mode, Max>;
  ensure_smem(kernel);
  const dim3 grid((ni + cols - 1) / cols, n_outer, batch);
  kernel<<<grid, f.r2 * cols, smem, s>>>(data, so, sp, ni, f, __builtin_ctz(static_cast<unsigned>(cols)),
                                         fft_len(f.n()).tw, scale, aux.a, aux.hits, sb);
  check_launch("fft axis pass");
}

template <int Max>
void axis_two_mode(const Factors& f, int cols, float2* data, int n_outer, std::size_t so, std::size_t sp, int ni,
                   bool forward, AxisMode mode, float scale, const AxisAux& aux, int batch, std::size_t sb,
                   cudaStream_t s) {
  switch (mode) {
    case AxisMode::plain:
      if (forward) {
        launch_axis_two<true, 0, Max>(f, cols, data, n_outer, so, sp, ni, scale, aux, batch, sb, s);
      } else {
        launch_axis_two<false, 0, Max>(f, cols, data, n_outer, so, sp, ni, scale, aux, batch, sb, s);
      }
      break;
    case AxisMode::restore_half:
      launch_axis_two<true, 1, Max>(f, cols, data, n_outer, so, sp, ni, scale, aux, batch, sb, s);
      break;
    case AxisMode::restore_mask:
      launch_axis_two<true, 2, Max>(f, cols, data, n_outer, so, sp, ni, scale, aux, batch, sb, s);
      break;
    case AxisMode::from_data:
      launch_axis_two<false, 3, Max>(f, cols, data, n_outer, so, sp, ni, scale, aux, batch, sb, s);
      break;
  }
}

// ---- real rows <-> half spectra -----------------------------------------------------------------------
// A row of nx = 2 M real values as M complex values (the pairs 2m, 2m + 1) through a length-M transform, with
// the split and merge formulas of the staged rows (fft3d.cu). A tile is `lines` rows, f.r2 threads each.

// Value m of the length-M line whose inverse transform gives the pairs of a row, from its half spectrum.
__device__ __forceinline__ float2 merge_value(const float2* __restrict__ e_row, int m, int M,
                                              const float2* __restrict__ twn) {
  float2 a = e_row[m], b = e_row[M - m];
  if (m == 0) a.y = b.y = 0.0f;  // a real signal has real bins 0 and M; their imaginary parts drop out
  const float2 sv = make_float2(a.x + b.x, a.y - b.y);  // a + conj(b)
  const float2 d = make_float2(a.x - b.x, a.y + b.y);   // a - conj(b)
  const float2 t = cmulc(d, __ldg(twn + m));             // d e^{2 pi i m / nx}
  return make_float2(sv.x - t.y, sv.y + t.x);            // sv + i t
}

// Lines in `zs` (natural order, M + 1 apart) to their rows' half spectra, one warp per row at a time.
__device__ __forceinline__ void split_rows(const float2* zs, int M, std::size_t row0, int lines, std::size_t rows,
                                           const float2* __restrict__ twn, float2* __restrict__ e) {
  const int warps = static_cast<int>(blockDim.x + 31) >> 5;
  for (int l = static_cast<int>(threadIdx.x) >> 5; l < lines && row0 + l < rows; l += warps) {
    const float2* z = zs + l * (M + 1);
    float2* out = e + (row0 + l) * (M + 1);
    for (int k = static_cast<int>(threadIdx.x) & 31; k <= M; k += 32) {
      const float2 zk = z[k == M ? 0 : k], zm = z[k == 0 ? 0 : M - k];
      const float2 ev = make_float2(0.5f * (zk.x + zm.x), 0.5f * (zk.y - zm.y));
      const float2 od = make_float2(0.5f * (zk.y + zm.y), -0.5f * (zk.x - zm.x));  // (zk - conj zm) / 2i
      out[k] = cadd(ev, cmul(__ldg(twn + k), od));
    }
  }
}

// Second pass of a forward transform into natural order, and the split.
template <int Max>
__device__ __forceinline__ void finish_r2c(const Factors& f, const RowTile& r, const float2* xs, int C, float2* zs,
                                           std::size_t row0, int lines, std::size_t rows,
                                           const float2* __restrict__ twn, float2* __restrict__ e) {
  const int M = f.n(), A = f.r2 | 1;
  __syncthreads();
  if (r.second) {
    twofft::with_radix<Max>(f.r2, [&]<int R>() {
      float2 u[R];
      twofft::second_pass<R, true>(u, xs + r.line2 * C + r.j2 * A, 1);
#pragma unroll
      for (int q = 0; q < R; ++q) zs[r.line2 * (M + 1) + r.j2 + f.r1 * q] = u[q];
    });
  }
  __syncthreads();
  split_rows(zs, M, row0, lines, rows, twn, e);
}

template <bool Clamp, int Max>
__global__ void __launch_bounds__(256, min_blocks(Max))
    k_rows_r2c_two(const float* __restrict__ x, float2* __restrict__ e, std::size_t rows, Factors f, int lines,
                   const float2* __restrict__ tw, const float2* __restrict__ twn) {
  extern __shared__ float2 xs[];
  const int M = f.n(), A = f.r2 | 1, C = row_line_pitch(f);
  if (!QHK_CHECK(static_cast<std::size_t>(lines) * (C + M + 1) * sizeof(float2) <= debug::dynamic_smem_bytes())) return;
  const std::size_t row0 = static_cast<std::size_t>(blockIdx.x) * lines;
  const RowTile r = row_tile(f, lines);
  if (r.first) {
    const bool live = row0 + r.line < rows;
    twofft::with_first<Max>(f.r1, [&]<int R>() {
      float2 v[R];
      const float2* p = reinterpret_cast<const float2*>(x) + (live ? row0 + r.line : 0) * M + r.j;
#pragma unroll
      for (int q = 0; q < R; ++q, p += f.r2) {
        v[q] = live ? *p : make_float2(0.0f, 0.0f);
        if (Clamp) v[q] = make_float2(fmaxf(v[q].x, 0.0f), fmaxf(v[q].y, 0.0f));
      }
      twofft::first_pass<R, true>(v, r.j, tw, xs + r.line * C + r.j, A);
    });
  }
  finish_r2c<Max>(f, r, xs, C, xs + lines * C, row0, lines, rows, twn, e);
}

template <int Mode, int Max>
__global__ void __launch_bounds__(256, min_blocks(Max))
    k_rows_c2r_two(const float2* __restrict__ e, float* __restrict__ x, std::size_t rows, Factors f, int lines,
                   const float2* __restrict__ tw, const float2* __restrict__ twn, float nm2, float inv_k02) {
  extern __shared__ float2 xs[];
  const int M = f.n(), A = f.r2 | 1, C = row_line_pitch(f);
  if (!QHK_CHECK(static_cast<std::size_t>(lines) * C * sizeof(float2) <= debug::dynamic_smem_bytes())) return;
  const std::size_t row0 = static_cast<std::size_t>(blockIdx.x) * lines;
  const RowTile r = row_tile(f, lines);
  if (r.first) {
    const float2* er = e + (row0 + r.line < rows ? row0 + r.line : 0) * (M + 1);
    twofft::with_first<Max>(f.r1, [&]<int R>() {
      float2 v[R];
#pragma unroll
      for (int q = 0; q < R; ++q) v[q] = merge_value(er, r.j + q * f.r2, M, twn);
      twofft::first_pass<R, false>(v, r.j, tw, xs + r.line * C + r.j, A);
    });
  }
  __syncthreads();
  if (r.second && row0 + r.line2 < rows) {
    twofft::with_radix<Max>(f.r2, [&]<int R>() {
      float2 u[R];
      twofft::second_pass<R, false>(u, xs + r.line2 * C + r.j2 * A, 1);
      float2* p = reinterpret_cast<float2*>(x) + (row0 + r.line2) * M + r.j2;
#pragma unroll
      for (int q = 0; q < R; ++q, p += f.r1) {
        float2 z = u[q];
        if (Mode == static_cast<int>(C2rMode::index)) {
          z = make_float2(index_from_potential(z.x, 0.0f, nm2, inv_k02), index_from_potential(z.y, 0.0f, nm2, inv_k02));
        }
        *p = z;
      }
    });
  }
}

// C2R, max(x, 0), R2C in place (one Gerchberg-Papoulis step boundary): the constraint falls between the
// second pass of the inverse and the first of the forward transform, on values one thread holds.
template <int Max>
__global__ void __launch_bounds__(256, min_blocks(Max))
    k_rows_c2r_r2c_two(float2* __restrict__ e, std::size_t rows, Factors f, int lines, const float2* __restrict__ tw,
                       const float2* __restrict__ twn) {
  extern __shared__ float2 xs[];
  const int M = f.n(), A = f.r2 | 1, C = row_line_pitch(f);
  if (!QHK_CHECK(static_cast<std::size_t>(lines) * (C + M + 1) * sizeof(float2) <= debug::dynamic_smem_bytes())) return;
  float2* zs = xs + lines * C;
  const std::size_t row0 = static_cast<std::size_t>(blockIdx.x) * lines;
  const RowTile r = row_tile(f, lines);
  if (r.first) {
    const float2* er = e + (row0 + r.line < rows ? row0 + r.line : 0) * (M + 1);
    twofft::with_first<Max>(f.r1, [&]<int R>() {
      float2 v[R];
#pragma unroll
      for (int q = 0; q < R; ++q) v[q] = merge_value(er, r.j + q * f.r2, M, twn);
      twofft::first_pass<R, false>(v, r.j, tw, xs + r.line * C + r.j, A);
    });
  }
  __syncthreads();
  if (r.second) {
    twofft::with_radix<Max>(f.r2, [&]<int R>() {
      float2 u[R];
      float2* s = xs + r.line2 * C + r.j2 * A;
      twofft::second_pass<R, false>(u, s, 1);
#pragma unroll
      for (int q = 0; q < R; ++q) u[q] = make_float2(fmaxf(u[q].x, 0.0f), fmaxf(u[q].y, 0.0f));
      twofft::first_pass<R, true>(u, r.j2, tw, s, 1);
    });
  }
  __syncthreads();
  if (r.first) {
    twofft::with_first<Max>(f.r1, [&]<int R>() {
      float2 v[R];
      twofft::second_pass<R, true>(v, xs + r.line * C + r.j, A);
#pragma unroll
      for (int q = 0; q < R; ++q) zs[r.line * (M + 1) + r.j + f.r2 * q] = v[q];
    });
  }
  __syncthreads();
  split_rows(zs, M, row0, lines, rows, twn, e);
}

// The end of one FISTA-TV iteration and the start of the next on rows (fft3d.cu k_rows_tv_final_r2c: the
// final primal, the momentum point, xprev, and the R2C of the momentum point), with the same operations;
// the momentum point is formed with row-contiguous loads into shared memory, one warp per row at a time. 256^3:
// 92 us (470 MB, 5.1 TB/s) from 108; 150 x 180^2: 36 us from 48.
template <int Max>
__global__ void __launch_bounds__(256, min_blocks(Max))
    k_rows_tv_final_r2c_two(const float* __restrict__ b, const float* __restrict__ pz, const float* __restrict__ py,
                            const float* __restrict__ px, int nz, int ny, float lambda, float momentum,
                            float* __restrict__ xprev, float2* __restrict__ e, std::size_t rows, Factors f, int lines,
                            const float2* __restrict__ tw, const float2* __restrict__ twn) {
  extern __shared__ float2 xs[];
  const int M = f.n(), n = 2 * M, A = f.r2 | 1, C = row_line_pitch(f);
  if (!QHK_CHECK(static_cast<std::size_t>(lines) * (C + M + 1) * sizeof(float2) <= debug::dynamic_smem_bytes())) return;
  float2* zs = xs + lines * C;  // the pairs of the momentum point's rows (M + 1 apart), then the spectrum
  const std::size_t row0 = static_cast<std::size_t>(blockIdx.x) * lines;
  const std::size_t nxy = static_cast<std::size_t>(n) * ny;
  {
    const int warps = static_cast<int>(blockDim.x + 31) >> 5;
    const int nr = static_cast<int>(min(static_cast<std::size_t>(lines), rows - min(row0, rows)));
    for (int w = static_cast<int>(threadIdx.x) >> 5; w < lines; w += warps) {
      float2* yrow = zs + w * (M + 1);
      if (w >= nr) {
        for (int m = static_cast<int>(threadIdx.x) & 31; m < M; m += 32) yrow[m] = make_float2(0.0f, 0.0f);
        continue;
      }
      const std::size_t r = row0 + w;
      const int z = static_cast<int>(r / ny), y = static_cast<int>(r - static_cast<std::size_t>(z) * ny);
#pragma unroll 2
      for (int m = static_cast<int>(threadIdx.x) & 31; m < M; m += 32) {
        const std::size_t i0 = r * n + 2 * m;
        const float2 bv = *reinterpret_cast<const float2*>(b + i0);
        const float2 cz = *reinterpret_cast<const float2*>(pz + i0);
        const float2 cy = *reinterpret_cast<const float2*>(py + i0);
        const float2 cx = *reinterpret_cast<const float2*>(px + i0);
        const float2 pv = *reinterpret_cast<const float2*>(xprev + i0);
        float2 bz = make_float2(0.0f, 0.0f), by = make_float2(0.0f, 0.0f);
        if (z > 0) bz = *reinterpret_cast<const float2*>(pz + i0 - nxy);
        if (y > 0) by = *reinterpret_cast<const float2*>(py + i0 - n);
        const float left = m > 0 ? px[i0 - 1] : 0.0f;
        const float bb[2] = {bv.x, bv.y}, czz[2] = {cz.x, cz.y}, cyy[2] = {cy.x, cy.y}, cxx[2] = {cx.x, cx.y};
        const float bzz[2] = {bz.x, bz.y}, byy[2] = {by.x, by.y}, pvv[2] = {pv.x, pv.y};
        float xv[2], yv[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const int xi = 2 * m + i;
          float sdiv = 0.0f;
          if (z < nz - 1) sdiv = __fadd_rn(sdiv, czz[i]);
          if (z > 0) sdiv = __fsub_rn(sdiv, bzz[i]);
          if (y < ny - 1) sdiv = __fadd_rn(sdiv, cyy[i]);
          if (y > 0) sdiv = __fsub_rn(sdiv, byy[i]);
          if (xi < n - 1) sdiv = __fadd_rn(sdiv, cxx[i]);
          if (xi > 0) sdiv = __fsub_rn(sdiv, i == 0 ? left : cxx[0]);
          xv[i] = tv_primal(bb[i], lambda, sdiv);
          yv[i] = __fadd_rn(xv[i], __fmul_rn(momentum, __fsub_rn(xv[i], pvv[i])));
        }
        *reinterpret_cast<float2*>(xprev + i0) = make_float2(xv[0], xv[1]);
        yrow[m] = make_float2(yv[0], yv[1]);
      }
    }
  }
  __syncthreads();
  const RowTile r = row_tile(f, lines);
  if (r.first) {
    twofft::with_first<Max>(f.r1, [&]<int R>() {
      float2 v[R];
      const float2* p = zs + r.line * (M + 1) + r.j;
#pragma unroll
      for (int q = 0; q < R; ++q, p += f.r2) v[q] = *p;
      twofft::first_pass<R, true>(v, r.j, tw, xs + r.line * C + r.j, A);
    });
  }
  finish_r2c<Max>(f, r, xs, C, zs, row0, lines, rows, twn, e);
}

// ---- complex rows -------------------------------------------------------------------------------------

template <bool Fwd, int Mode, int Max>
__global__ void __launch_bounds__(256, min_blocks(Max))
    k_rows_c2c_two(float2* __restrict__ data, std::size_t rows, Factors f, int lines, const float2* __restrict__ tw,
                   float scale, float* __restrict__ index, float nm2, float inv_k02) {
  extern __shared__ float2 xs[];
  const int n = f.n(), A = f.r2 | 1, C = row_line_pitch(f);
  if (!QHK_CHECK(static_cast<std::size_t>(lines) * C * sizeof(float2) <= debug::dynamic_smem_bytes())) return;
  constexpr bool first_fwd = Mode == static_cast<int>(RowMode::plain) && Fwd;
  const std::size_t line0 = static_cast<std::size_t>(blockIdx.x) * lines;
  const RowTile r = row_tile(f, lines);
  const std::size_t row = line0 + r.line, row2 = line0 + r.line2;
  if (r.first) {
    const bool live = row < rows;
    twofft::with_first<Max>(f.r1, [&]<int R>() {
      float2 v[R];
      const float2* p = data + (live ? row : 0) * n + r.j;
#pragma unroll
      for (int q = 0; q < R; ++q, p += f.r2) v[q] = live ? *p : make_float2(0.0f, 0.0f);
      twofft::first_pass<R, first_fwd>(v, r.j, tw, xs + r.line * C + r.j, A);
    });
  }
  __syncthreads();
  if (r.second && row2 < rows) {
    twofft::with_radix<Max>(f.r2, [&]<int R>() {
      float2 u[R];
      float2* s = xs + r.line2 * C + r.j2 * A;
      twofft::second_pass<R, first_fwd>(u, s, 1);
      if constexpr (Mode == static_cast<int>(RowMode::inv_clamp_fwd)) {
#pragma unroll
        for (int q = 0; q < R; ++q) u[q] = make_float2(fmaxf(u[q].x * scale, 0.0f), 0.0f);
        twofft::first_pass<R, true>(u, r.j2, tw, s, 1);
      } else {
        const std::size_t g = row2 * n + r.j2;
#pragma unroll
        for (int q = 0; q < R; ++q) {
          if constexpr (Mode == static_cast<int>(RowMode::inv_index)) {
            index[g + q * f.r1] = index_from_potential(u[q].x * scale, u[q].y * scale, nm2, inv_k02);
          } else {
            data[g + q * f.r1] = scale != 1.0f ? cscale(u[q], scale) : u[q];
          }
        }
      }
    });
  }
  if constexpr (Mode == static_cast<int>(RowMode::inv_clamp_fwd)) {
    __syncthreads();
    if (r.first && row < rows) {
      twofft::with_first<Max>(f.r1, [&]<int R>() {
        float2 v[R];
        twofft::second_pass<R, true>(v, xs + r.line * C + r.j, A);
        float2* p = data + row * n + r.j;
#pragma unroll
        for (int q = 0; q < R; ++q, p += f.r2) *p = v[q];
      });
    }
  }
}

// Calls g.template operator()<Max>(factors) when the engine covers length n.
template <class G>
bool with_factors(int n, G&& g) {
  Factors f;
  if (!fft_reg_engine_enabled() || !twofft::factors(n, &f)) return false;
  twofft::with_class(f, [&]<int Max>() { g.template operator()<Max>(f); });
  return true;
}

}  // namespace

bool axis_two_covers(int n) {
  Factors f;
  return fft_reg_engine_enabled() && twofft::factors(n, &f);
}

std::vector<int> axis_two_columns(int n) {
  Factors f;
  if (!twofft::factors(n, &f) || f.r2 > 16) return {8};
  return {16, 8};
}

bool axis_pass_two(int cols, float2* data, int n_outer, std::size_t so, int n, std::size_t sp, int ni, bool forward,
                   AxisMode mode, float scale, const AxisAux& aux, cudaStream_t s, int batch, std::size_t sb) {
  return with_factors(n, [&]<int Max>(const Factors& f) {
    if (f.r2 > 16) cols = 8;
    axis_two_mode<Max>(f, cols, data, n_outer, so, sp, ni, forward, mode, scale, aux, batch, sb, s);
  });
}

bool rows_r2c_two(const float* x, float2* e, std::size_t rows, int nx, bool clamp, cudaStream_t s) {
  return with_factors(nx / 2, [&]<int Max>(const Factors& f) {
    const RowLaunch r = row_launch(f, rows, true);
    auto kernel = clamp ? k_rows_r2c_two<true, Max> : k_rows_r2c_two<false, Max>;
    ensure_smem(kernel);
    kernel<<<r.grid, r.threads, r.smem, s>>>(x, e, rows, f, r.lines, fft_len(nx / 2).tw, fft_len(nx).tw);
    check_launch("rows r2c");
  });
}

bool rows_c2r_two(const float2* e, float* x, std::size_t rows, int nx, C2rMode mode, float nm2, float inv_k02,
                  cudaStream_t s) {
  return with_factors(nx / 2, [&]<int Max>(const Factors& f) {
    const RowLaunch r = row_launch(f, rows, false);
    auto kernel = mode == C2rMode::index ? k_rows_c2r_two<1, Max> : k_rows_c2r_two<0, Max>;
    ensure_smem(kernel);
    kernel<<<r.grid, r.threads, r.smem, s>>>(e, x, rows, f, r.lines, fft_len(nx / 2).tw, fft_len(nx).tw, nm2, inv_k02);
    check_launch("rows c2r");
  });
}

bool rows_c2r_r2c_two(float2* e, std::size_t rows, int nx, cudaStream_t s) {
  return with_factors(nx / 2, [&]<int Max>(const Factors& f) {
    const RowLaunch r = row_launch(f, rows, true);
    ensure_smem(k_rows_c2r_r2c_two<Max>);
    k_rows_c2r_r2c_two<Max><<<r.grid, r.threads, r.smem, s>>>(e, rows, f, r.lines, fft_len(nx / 2).tw, fft_len(nx).tw);
    check_launch("rows c2r r2c");
  });
}

bool rows_tv_final_r2c_two(const float* b, const float* const p[3], int nz, int ny, int nx, float lambda,
                           float momentum, float* xprev, float2* e, cudaStream_t s) {
  return with_factors(nx / 2, [&]<int Max>(const Factors& f) {
    const std::size_t rows = static_cast<std::size_t>(nz) * ny;
    const RowLaunch r = row_launch(f, rows, true);
    ensure_smem(k_rows_tv_final_r2c_two<Max>);
    k_rows_tv_final_r2c_two<Max><<<r.grid, r.threads, r.smem, s>>>(b, p[0], p[1], p[2], nz, ny, lambda, momentum,
                                                                   xprev, e, rows, f, r.lines, fft_len(nx / 2).tw,
                                                                   fft_len(nx).tw);
    check_launch("rows tv final r2c");
  });
}

bool rows_c2c_two(float2* data, std::size_t rows, int nx, bool forward, RowMode mode, float scale, float* index,
                  float nm2, float inv_k02, cudaStream_t s) {
  return with_factors(nx, [&]<int Max>(const Factors& f) {
    const RowLaunch r = row_launch(f, rows, false);
    auto kernel = mode == RowMode::inv_clamp_fwd ? k_rows_c2c_two<false, 1, Max>
                  : mode == RowMode::inv_index   ? k_rows_c2c_two<false, 2, Max>
                  : forward                      ? k_rows_c2c_two<true, 0, Max>
                                                 : k_rows_c2c_two<false, 0, Max>;
    ensure_smem(kernel);
    kernel<<<r.grid, r.threads, r.smem, s>>>(data, rows, f, r.lines, fft_len(nx).tw, scale, index, nm2, inv_k02);
    check_launch("rows c2c");
  });
}

}  // namespace qhk
