// Host interface of the passes on the two-factor line transforms (fft_two.cu, fft_plane.cu). Each returns
// false when it does not cover the length (or the plane does not fit), and has then done nothing.
#pragma once

#include <vector>

#include "qhk_internal.hpp"

namespace qhk {

// An axis pass (qhk_internal.hpp axis_pass) with `cols` columns per CTA, one of axis_two_columns(n) (the
// first is the default), for lengths that are a product of two of the engine's radices.
bool axis_two_covers(int n);
std::vector<int> axis_two_columns(int n);
bool axis_pass_two(int cols, float2* data, int n_outer, std::size_t so, int n, std::size_t sp, int ni, bool forward,
                   AxisMode mode, float scale, const AxisAux& aux, cudaStream_t s, int batch, std::size_t sb);

// The row passes of qhk_internal.hpp, for even nx that axis_two_covers.
bool rows_r2c_two(const float* x, float2* e, std::size_t rows, int nx, bool clamp, cudaStream_t s);
bool rows_c2r_two(const float2* e, float* x, std::size_t rows, int nx, C2rMode mode, float nm2, float inv_k02,
                  cudaStream_t s);
bool rows_c2r_r2c_two(float2* e, std::size_t rows, int nx, cudaStream_t s);
bool rows_tv_final_r2c_two(const float* b, const float* const p[3], int nz, int ny, int nx, float lambda,
                           float momentum, float* xprev, float2* e, cudaStream_t s);
bool rows_c2c_two(float2* data, std::size_t rows, int nx, bool forward, RowMode mode, float scale, float* index,
                  float nm2, float inv_k02, cudaStream_t s);

// One Gerchberg-Papoulis step between two z passes, in place on `planes` half-spectrum planes (n, n / 2 + 1):
// inverse y transform, C2R, max(x, 0), R2C, forward y transform, a plane on chip throughout.
bool plane_gp_covers(int n);
bool plane_gp(float2* e, std::size_t planes, int n, cudaStream_t s);

}  // namespace qhk
