// Two-factor line transforms: a line of N = R1 R2 points as one in-register DFT per factor with a single
// exchange through shared memory between them, for every N whose factors are radices this header has.
//
// With n = j + R2 q (j < R2, q < R1) and k = k1 + R1 k2 (k1 < R1, k2 < R2):
//
//   X[k1 + R1 k2] = sum_j W_R2^{j k2} W_N^{j k1} sum_q W_R1^{q k1} x[j + R2 q]
//
// first pass: butterfly j (one thread) takes x[j + R2 q], a length-R1 DFT, times W_N^{j k1}, into slot
// (k1, j) of the line's exchange buffer; second pass: butterfly j2 = k1 takes the R2 values (j2, j), a
// length-R2 DFT, whose outputs are the positions j2 + R1 k2. Two properties the callers build on:
//   * the second pass reads and may write back exactly its own slots, so a transform followed by a
//     pointwise step and the opposite transform needs no second buffer: the opposite transform runs with
//     the factors exchanged, its first pass (radix R2, positions j2 + R1 q) on the values the thread
//     already holds, into the same slots, and its last pass (radix R1) on the slots of the very first;
//   * the last pass of that pair leaves butterfly j the positions j + R2 q it loaded first.
// The factors are run-time values: `with_radix` switches to the code of a radix, in which everything is
// unrolled and the roots of unity are immediates. Forward sign e^{-2 pi i / N}, unnormalised.
#pragma once

#include <cuda_runtime.h>

#include "fft_engine.cuh"

namespace qhk {
namespace twofft {

// cos and sin of 2 pi k / R by the Taylor series on the first octant (compile time).
constexpr double turn_cos(int k, int R);
constexpr double turn_sin(int k, int R) {
  k %= R;
  if (k < 0) k += R;
  if (2 * k > R) return -turn_sin(R - k, R);  // sin(2 pi - a) = -sin a
  if (4 * k > R) {                             // sin(pi - a) = sin a, with pi = R / 2 turns of 1 / R
    return turn_sin(R - 2 * k, 2 * R);
  }
  if (8 * k > R) return turn_cos(R - 4 * k, 4 * R);  // sin a = cos(pi / 2 - a)
  const double x = 6.283185307179586476925286766559 * k / R;
  double term = x, sum = x;
  for (int i = 1; i < 12; ++i) {
    term *= -x * x / ((2 * i) * (2 * i + 1));
    sum += term;
  }
  return sum;
}
constexpr double turn_cos(int k, int R) {
  k %= R;
  if (k < 0) k += R;
  if (2 * k > R) return turn_cos(R - k, R);
  if (4 * k > R) return -turn_cos(R - 2 * k, 2 * R);
  if (8 * k > R) return turn_sin(R - 4 * k, 4 * R);
  const double x = 6.283185307179586476925286766559 * k / R;
  double term = 1.0, sum = 1.0;
  for (int i = 1; i < 12; ++i) {
    term *= -x * x / ((2 * i - 1) * (2 * i));
    sum += term;
  }
  return sum;
}

// e^{-2 pi i k / R}, k < R.
template <int R>
struct Roots {
  float c[R], s[R];
  constexpr Roots() : c{}, s{} {
    for (int k = 0; k < R; ++k) {
      c[k] = static_cast<float>(turn_cos(k, R));
      s[k] = static_cast<float>(-turn_sin(k, R));
    }
  }
};

// v W_R^m (its conjugate for the inverse), R and m constant after unrolling.
template <int R, bool Fwd>
__device__ __forceinline__ float2 times_root(float2 v, int m) {
  constexpr Roots<R> w{};
  const int q = m % R;
  if (q == 0) return v;
  if (2 * q == R) return make_float2(-v.x, -v.y);
  if (4 * q == R) return Fwd ? make_float2(v.y, -v.x) : make_float2(-v.y, v.x);
  if (4 * q == 3 * R) return Fwd ? make_float2(-v.y, v.x) : make_float2(v.y, -v.x);
  const float c = w.c[q], s = Fwd ? w.s[q] : -w.s[q];
  return make_float2(v.x * c - v.y * s, v.x * s + v.y * c);
}

template <int R, bool Fwd>
__device__ __forceinline__ void dft(float2* v);

// Length N1 N2 as N2-point DFTs over n2 (n = n1 + N1 n2), twiddles, N1-point DFTs over n1.
template <int N1, int N2, bool Fwd>
__device__ __forceinline__ void dft_split(float2* v) {
  float2 a[N1][N2];
#pragma unroll
  for (int n1 = 0; n1 < N1; ++n1) {
#pragma unroll
    for (int n2 = 0; n2 < N2; ++n2) a[n1][n2] = v[n1 + N1 * n2];
    dft<N2, Fwd>(a[n1]);
  }
#pragma unroll
  for (int k1 = 0; k1 < N2; ++k1) {
    float2 b[N1];
#pragma unroll
    for (int n1 = 0; n1 < N1; ++n1) b[n1] = times_root<N1 * N2, Fwd>(a[n1][k1], n1 * k1);
    dft<N1, Fwd>(b);
#pragma unroll
    for (int k2 = 0; k2 < N1; ++k2) v[k1 + N2 * k2] = b[k2];
  }
}

// An odd prime P: the sums and differences of the pairs (k, P - k) against the cosines and sines.
template <int P, bool Fwd>
__device__ __forceinline__ void dft_prime(float2* v) {
  constexpr Roots<P> w{};
  constexpr int H = P / 2;
  float2 a[H], b[H], o[P];
  o[0] = v[0];
#pragma unroll
  for (int k = 0; k < H; ++k) {
    a[k] = cadd(v[k + 1], v[P - 1 - k]);
    b[k] = csub(v[k + 1], v[P - 1 - k]);
    o[0] = cadd(o[0], a[k]);
  }
#pragma unroll
  for (int m = 1; m <= H; ++m) {
    float2 e = v[0], d = make_float2(0.0f, 0.0f);
#pragma unroll
    for (int k = 0; k < H; ++k) {
      const float c = w.c[(m * (k + 1)) % P], s = -w.s[(m * (k + 1)) % P];  // cos, sin of 2 pi m (k + 1) / P
      e = make_float2(e.x + c * a[k].x, e.y + c * a[k].y);
      d = make_float2(d.x + s * b[k].x, d.y + s * b[k].y);
    }
    const float2 r = fftdev::rot<Fwd>(d);  // -i d forward, +i d inverse
    o[m] = cadd(e, r);
    o[P - m] = csub(e, r);
  }
#pragma unroll
  for (int k = 0; k < P; ++k) v[k] = o[k];
}

template <int R, bool Fwd>
__device__ __forceinline__ void dft(float2* v) {
  if constexpr (R == 1) {
  } else if constexpr (R == 2 || R == 3 || R == 4 || R == 5 || R == 8) {
    fftdev::dft<R, Fwd>(v);
  } else if constexpr (R % 16 == 0) {
    dft_split<R / 8 < 4 ? 4 : R / 8, R / 8 < 4 ? R / 4 : 8, Fwd>(v);  // 16 = 4 4, 32 = 4 8
  } else if constexpr (R % 8 == 0) {
    dft_split<R / 8, 8, Fwd>(v);
  } else if constexpr (R % 4 == 0) {
    dft_split<R / 4, 4, Fwd>(v);
  } else if constexpr (R % 2 == 0) {
    dft_split<2, R / 2, Fwd>(v);
  } else if constexpr (R % 3 == 0 && R > 3) {
    dft_split<3, R / 3, Fwd>(v);
  } else if constexpr (R % 5 == 0 && R > 5) {
    dft_split<5, R / 5, Fwd>(v);
  } else {
    dft_prime<R, Fwd>(v);
  }
}

// The radices: up to 16 for the first factor, larger ones up to 32 for the second. Kernels are instantiated
// per class, which sets their registers: radices 2^a 3^b 5^c up to 16, 24 or 32 for the second factor, or
// (kAny) all of them, those with factors 7, 11 and 13 too, whose DFTs hold twice the values.
constexpr int kSmall = 16, kMid = 24, kLarge = 32, kAny = 64;
constexpr bool radix(int r) {
  return (r >= 2 && r <= 16) || r == 18 || r == 20 || r == 21 || r == 22 || r == 24 || r == 25 || r == 26 || r == 28 ||
         r == 30 || r == 32;
}
constexpr bool smooth_radix(int r) { return r % 7 != 0 && r % 11 != 0 && r % 13 != 0; }
constexpr bool in_class(int r, int max) { return max == kAny || (r <= max && smooth_radix(r)); }

// Calls f.template operator()<R>() for the radix R == r of the class; the first factor's radices only.
template <int Max, class F>
__device__ __forceinline__ void with_first(int r, F&& f) {
  switch (r) {
#define QHK_RADIX(R)                                                \
  case R:                                                           \
    if constexpr (in_class(R, Max)) f.template operator()<R>();     \
    return;
#define QHK_FIRST                                                                                                 \
  QHK_RADIX(2) QHK_RADIX(3) QHK_RADIX(4) QHK_RADIX(5) QHK_RADIX(6) QHK_RADIX(7) QHK_RADIX(8) QHK_RADIX(9)         \
  QHK_RADIX(10) QHK_RADIX(11) QHK_RADIX(12) QHK_RADIX(13) QHK_RADIX(14) QHK_RADIX(15) QHK_RADIX(16)
    QHK_FIRST
    default: return;
  }
}
// The same for either factor.
template <int Max, class F>
__device__ __forceinline__ void with_radix(int r, F&& f) {
  switch (r) {
    QHK_FIRST
    QHK_RADIX(18) QHK_RADIX(20) QHK_RADIX(21) QHK_RADIX(22) QHK_RADIX(24) QHK_RADIX(25) QHK_RADIX(26)
    QHK_RADIX(28) QHK_RADIX(30) QHK_RADIX(32)
#undef QHK_FIRST
#undef QHK_RADIX
    default: return;
  }
}

// The factors of a line length. Kernels that give a line r2 threads (rows, axis passes, field columns, BPM slices)
// need r1 <= r2, which `factors` (r1 up to 16, for with_first) and the field columns' own choice (r1 up to 32, for
// with_radix) see to. The planes of fft_plane.cu stride their threads over the butterflies and need no order: their x
// factors may have r1 > r2 (182 = 14 x 13).
struct Factors {
  int r1 = 0, r2 = 0;
  __host__ __device__ int n() const { return r1 * r2; }
};

// Calls g.template operator()<Max>() with the kernel class of the factors.
template <class G>
void with_class(const Factors& f, G&& g) {
  if (!smooth_radix(f.r1) || !smooth_radix(f.r2)) {
    g.template operator()<kAny>();
  } else if (f.r2 <= kSmall) {
    g.template operator()<kSmall>();
  } else if (f.r2 <= kMid) {
    g.template operator()<kMid>();
  } else {
    g.template operator()<kLarge>();
  }
}

// The most even pair of radices with product n; false when there is none.
inline bool factors(int n, Factors* f) {
  for (int r1 = 16; r1 >= 2; --r1) {
    const int r2 = n / r1;
    if (r1 * r2 == n && r2 >= r1 && radix(r2)) {
      *f = Factors{r1, r2};
      return true;
    }
  }
  return false;
}

// Slots of a tile of lines: value (k1, j) of a line at k1 * A + j * B + line * C.
struct Slots {
  int A, B, C;
};

// First pass on the values v[q] = x[j + R2 q] already loaded: DFT, twiddle, into the slots (k1, j).
template <int R, bool Fwd>
__device__ __forceinline__ void first_pass(float2 (&v)[R], int j, const float2* __restrict__ tw, float2* xs, int A) {
  dft<R, Fwd>(v);
  xs[0] = v[0];
#pragma unroll
  for (int k1 = 1; k1 < R; ++k1) {
    const float2 w = __ldg(tw + j * k1);
    xs[k1 * A] = Fwd ? cmul(v[k1], w) : cmulc(v[k1], w);
  }
}

// Second pass: the slots (j2, j), j < R, at xs[j * B], into u (outputs k = j2 + R1 q in u[q]).
template <int R, bool Fwd>
__device__ __forceinline__ void second_pass(float2 (&u)[R], const float2* xs, int B) {
#pragma unroll
  for (int j = 0; j < R; ++j) u[j] = xs[j * B];
  dft<R, Fwd>(u);
}

}  // namespace twofft
}  // namespace qhk
