// One Gerchberg-Papoulis step between two z passes with each plane of the half spectrum on chip: inverse y
// transform, C2R along x, max(x, 0), R2C, forward y transform, in one launch and one pass over memory,
// where separate y and row passes make three. Bounded by the seven phases' latency and shared-memory traffic
// (six round trips of the plane) at the one to four CTAs that an SM's shared memory and registers hold.
// Measured on B200 per step, against the three passes: 64^3 7 us from 9 (and two launches fewer), 128^3 14 us
// from 19; 8 x 96^3 35 us, where the three staged passes took 146.
//
// A CTA takes a plane (n, n / 2 + 1) of complex64 whose n rows lie in shared memory at an odd pitch. Every
// phase works in place, on slots that one thread alone reads and writes between two barriers:
//   1  y, radix R1: from global memory, position j + R2 q of column kx, to row k1 R2 + j
//   2  y, radix R2: rows j2 R2 + (0 .. R2 - 1), after which row a R2 + b holds y = a + R1 b
//   3  x, radix X1 (even), pairs of rows (i, i + n / 2) as one complex line of length n (their real rows are
//      its real and imaginary parts): butterflies j and X2 - j together, since positions k and
//      n - k come from the same two bins; value (k1, j) of the line goes to column j + X2 (k1 mod X1 / 2) of
//      the first row (k1 < X1 / 2) or the second, which are bins that this pair of butterflies read
//   4  x, radix X2 inverse, the constraint, radix X2 forward (factors exchanged), on one line's slots k1
//   5  x, radix X1 and the split into the two rows' bins, butterflies j and X2 - j, as 3 backwards
//   6  y, radix R2 forward, as 2
//   7  y, radix R1, to global memory, as 1 backwards
// Threads run over kx in the y phases and over row pairs in the x phases: with the odd pitch no phase has
// bank conflicts, and the global accesses are contiguous rows of n / 2 + 1 values.
#include "debug.cuh"
#include "fft_two.cuh"
#include "fft_two.hpp"

namespace qhk {

namespace {

using twofft::Factors;

__host__ __device__ __forceinline__ int plane_pitch(int n) { return (n / 2 + 1) | 1; }

// The thread count that bounds the registers: 96 a thread for the small radices, which five CTAs of 128 threads
// leave an SM (8 x 96^3: 35 us per step, 39 with the 118 that the compiler would take), 128 for the others.
constexpr int plane_bound(int max) { return max == twofft::kSmall ? 640 : 512; }

template <int Max>
__global__ void __launch_bounds__(plane_bound(Max), 1)
    k_plane_gp(float2* __restrict__ e, int n, Factors fy, Factors fx, const float2* __restrict__ tw) {
  extern __shared__ float2 sm[];
  const int h = n / 2 + 1, P = plane_pitch(n), H = n / 2;
  if (!QHK_CHECK(static_cast<std::size_t>(n) * P * sizeof(float2) <= debug::dynamic_smem_bytes())) return;
  float2* plane = e + static_cast<std::size_t>(blockIdx.x) * n * h;
  const int tid = static_cast<int>(threadIdx.x), nth = static_cast<int>(blockDim.x);

  // 1: column kx, butterfly j.
  twofft::with_first<Max>(fy.r1, [&]<int R>() {
    for (int i = tid; i < h * fy.r2; i += nth) {
      const int j = i / h, kx = i - j * h;
      float2 v[R];
      const float2* p = plane + j * h + kx;
      const int step = fy.r2 * h;
#pragma unroll
      for (int q = 0; q < R; ++q) v[q] = p[q * step];
      twofft::first_pass<R, false>(v, j, tw, sm + j * P + kx, fy.r2 * P);
    }
  });
  __syncthreads();
  // 2
  twofft::with_radix<Max>(fy.r2, [&]<int R>() {
    for (int i = tid; i < h * fy.r1; i += nth) {
      const int j = i / h, kx = i - j * h;
      float2 u[R];
      float2* p = sm + j * R * P + kx;
      twofft::second_pass<R, false>(u, p, P);
#pragma unroll
      for (int q = 0; q < R; ++q) p[q * P] = u[q];
    }
  });
  __syncthreads();
  // 3
  const int units = (fx.r2 + 1) / 2;  // butterflies j < X2 / 2 with X2 - j; unit 0: 0 and (X2 even) X2 / 2
  twofft::with_first<Max>(fx.r1, [&]<int R>() {
    if constexpr (R % 2 == 0 && R <= 14) {  // larger planes do not fit
      const int X2 = fx.r2;
      for (int i = tid; i < H * units; i += nth) {
        const int j = i / H;
        float2* a = sm + (i - j * H) * P;
        float2* b = a + H * P;
        const int w0 = j == 0 ? X2 / 2 : X2 - j;  // the other butterfly
        const bool has_w = j != 0 || X2 % 2 == 0;
        float2 v[R], w[R];
        if (j == 0) {
          // Butterfly 0 holds positions X2 q, closed under k -> n - k, butterfly X2 / 2 likewise; bins 0 and
          // n / 2 are real.
          v[0] = make_float2(a[0].x, b[0].x);
          v[R / 2] = make_float2(a[H].x, b[H].x);
#pragma unroll
          for (int q = 1; q < R / 2; ++q) {
            const float2 x = a[X2 * q], y = b[X2 * q];
            v[q] = make_float2(x.x - y.y, x.y + y.x);
            v[R - q] = make_float2(x.x + y.y, y.x - x.y);
          }
#pragma unroll
          for (int q = 0; q < R / 2; ++q) {
            const int k = has_w ? w0 + X2 * q : 0;
            const float2 x = a[k], y = b[k];
            w[q] = make_float2(x.x - y.y, x.y + y.x);
            w[R - 1 - q] = make_float2(x.x + y.y, y.x - x.y);
          }
        } else {
#pragma unroll
          for (int q = 0; q < R / 2; ++q) {
            const float2 x = a[j + X2 * q], y = b[j + X2 * q];
            v[q] = make_float2(x.x - y.y, x.y + y.x);
            w[R - 1 - q] = make_float2(x.x + y.y, y.x - x.y);
            const float2 x2 = a[w0 + X2 * q], y2 = b[w0 + X2 * q];
            w[q] = make_float2(x2.x - y2.y, x2.y + y2.x);
            v[R - 1 - q] = make_float2(x2.x + y2.y, y2.x - x2.y);
          }
        }
        twofft::dft<R, false>(v);
#pragma unroll
        for (int k1 = 0; k1 < R; ++k1) {
          const float2 z = k1 ? cmulc(v[k1], __ldg(tw + j * k1)) : v[0];
          (k1 < R / 2 ? a : b)[j + X2 * (k1 % (R / 2))] = z;
        }
        if (has_w) {
          twofft::dft<R, false>(w);
#pragma unroll
          for (int k1 = 0; k1 < R; ++k1) {
            const float2 z = k1 ? cmulc(w[k1], __ldg(tw + w0 * k1)) : w[0];
            (k1 < R / 2 ? a : b)[w0 + X2 * (k1 % (R / 2))] = z;
          }
        }
      }
    }
  });
  __syncthreads();
  // 4
  twofft::with_radix<Max>(fx.r2, [&]<int R>() {
    const int half = fx.r1 / 2;
    for (int i = tid; i < H * fx.r1; i += nth) {
      const int j = i / H;  // k1
      const int row = i - j * H;
      float2* s = sm + (j < half ? row : row + H) * P + R * (j < half ? j : j - half);
      float2 u[R];
      twofft::second_pass<R, false>(u, s, 1);
#pragma unroll
      for (int q = 0; q < R; ++q) u[q] = make_float2(fmaxf(u[q].x, 0.0f), fmaxf(u[q].y, 0.0f));
      twofft::first_pass<R, true>(u, j, tw, s, 1);
    }
  });
  __syncthreads();
  // 5
  twofft::with_first<Max>(fx.r1, [&]<int R>() {
    if constexpr (R % 2 == 0 && R <= 14) {  // larger planes do not fit
      const int X2 = fx.r2;
      const auto split = [](float2 zk, float2 zm, float2* a, float2* b) {
        *a = make_float2(0.5f * (zk.x + zm.x), 0.5f * (zk.y - zm.y));
        *b = make_float2(0.5f * (zk.y + zm.y), -0.5f * (zk.x - zm.x));
      };
      for (int i = tid; i < H * units; i += nth) {
        const int j = i / H;
        float2* a = sm + (i - j * H) * P;
        float2* b = a + H * P;
        const int w0 = j == 0 ? X2 / 2 : X2 - j;
        const bool has_w = j != 0 || X2 % 2 == 0;
        float2 v[R], w[R];
#pragma unroll
        for (int k1 = 0; k1 < R; ++k1) {
          v[k1] = (k1 < R / 2 ? a : b)[j + X2 * (k1 % (R / 2))];
          w[k1] = (k1 < R / 2 ? a : b)[(has_w ? w0 : 0) + X2 * (k1 % (R / 2))];
        }
        twofft::dft<R, true>(v);
        twofft::dft<R, true>(w);
        if (j == 0) {
          split(v[0], v[0], a, b);
          split(v[R / 2], v[R / 2], a + H, b + H);
#pragma unroll
          for (int q = 1; q < R / 2; ++q) split(v[q], v[R - q], a + X2 * q, b + X2 * q);
          if (has_w) {
#pragma unroll
            for (int q = 0; q < R / 2; ++q) split(w[q], w[R - 1 - q], a + w0 + X2 * q, b + w0 + X2 * q);
          }
        } else {
#pragma unroll
          for (int q = 0; q < R / 2; ++q) {
            split(v[q], w[R - 1 - q], a + j + X2 * q, b + j + X2 * q);
            split(w[q], v[R - 1 - q], a + w0 + X2 * q, b + w0 + X2 * q);
          }
        }
      }
    }
  });
  __syncthreads();
  // 6
  twofft::with_radix<Max>(fy.r2, [&]<int R>() {
    for (int i = tid; i < h * fy.r1; i += nth) {
      const int j = i / h, kx = i - j * h;
      float2 u[R];
      float2* p = sm + j * R * P + kx;
#pragma unroll
      for (int q = 0; q < R; ++q) u[q] = p[q * P];
      twofft::first_pass<R, true>(u, j, tw, p, P);
    }
  });
  __syncthreads();
  // 7
  twofft::with_first<Max>(fy.r1, [&]<int R>() {
    for (int i = tid; i < h * fy.r2; i += nth) {
      const int j = i / h, kx = i - j * h;
      float2 v[R];
      twofft::second_pass<R, true>(v, sm + j * P + kx, fy.r2 * P);
      float2* p = plane + j * h + kx;
      const int step = fy.r2 * h;
#pragma unroll
      for (int q = 0; q < R; ++q) p[q * step] = v[q];
    }
  });
}

std::size_t plane_smem(int n) { return static_cast<std::size_t>(n) * plane_pitch(n) * sizeof(float2); }

// The factors of the x transform, of the y transform's class: the first one even and at most 14 (the y
// transform's own where they are).
bool x_factors(const Factors& fy, Factors* x) {
  int max = 0;
  twofft::with_class(fy, [&]<int Max>() { max = Max; });
  for (int r1 = 14; r1 >= 2; r1 -= 2) {
    const int r2 = fy.n() / r1;
    if (r1 * r2 == fy.n() && twofft::radix(r2) && twofft::in_class(r1, max) && twofft::in_class(r2, max)) {
      *x = Factors{r1, r2};
      if (r1 <= r2) return true;
    }
  }
  return x->r1 != 0;
}

bool plane_factors(int n, Factors* fy, Factors* fx) {
  return n % 2 == 0 && plane_smem(n) <= 227 * 1024 && twofft::factors(n, fy) && x_factors(*fy, fx);
}

}  // namespace

bool plane_gp_covers(int n) {
  Factors fy, fx;
  return fft_reg_engine_enabled() && plane_factors(n, &fy, &fx);
}

bool plane_gp(float2* e, std::size_t planes, int n, cudaStream_t s) {
  Factors fy, fx;
  if (!fft_reg_engine_enabled() || !plane_factors(n, &fy, &fx)) return false;
  // 128 registers a thread allow 512 threads per SM: in one CTA where the planes do not fill the GPU twice or
  // only one fits the shared memory, else in two or four, whose loads overlap each other's transforms.
  const int resident = static_cast<int>((227 * 1024) / (plane_smem(n) + 1024));
  const int threads = planes <= static_cast<std::size_t>(sm_count()) || resident < 2 ? 512 : resident < 4 ? 256 : 128;
  const float2* tw = fft_len(n).tw;
  twofft::with_class(fy, [&]<int Max>() {
    ensure_smem(k_plane_gp<Max>);
    k_plane_gp<Max><<<static_cast<unsigned>(planes), threads, plane_smem(n), s>>>(e, n, fy, fx, tw);
  });
  check_launch("gp plane pass");
  return true;
}

}  // namespace qhk
