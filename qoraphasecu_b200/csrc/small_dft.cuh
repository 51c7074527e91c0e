// In-register DFTs of 2..16, 18, 20, 21, 24 and 25 points, for the mixed-radix
// passes: the
// power-of-two and radix-3/5 butterflies of butterfly.cuh, the primes 7, 11
// and 13 by their symmetric form, and the composites from those.
//
// Forward uses W = exp(-2 pi i / R); INV flips the sign of every imaginary
// unit. Inputs and outputs are in natural order.
#pragma once

#include <type_traits>
#include <utility>

#include "butterfly.cuh"

namespace qpb {

// sin and cos of 2 pi k / n, evaluated by the compiler in FP64 (Taylor series
// on [-pi, pi], 20 terms: below 1e-15 from the exact value) so that they
// become the immediate constants of the butterflies.
constexpr double turn_sine(int k, int n) {
  constexpr double kPi = 3.14159265358979323846;
  k = ((k % n) + n) % n;
  if (2 * k > n) k -= n;
  const double x = 2.0 * kPi * k / n;
  double term = x, sum = x;
  for (int i = 1; i < 20; ++i) {
    term *= -x * x / ((2 * i) * (2 * i + 1));
    sum += term;
  }
  return sum;
}
constexpr double turn_cosine(int k, int n) {
  constexpr double kPi = 3.14159265358979323846;
  k = ((k % n) + n) % n;
  if (2 * k > n) k -= n;
  const double x = 2.0 * kPi * k / n;
  double term = 1.0, sum = 1.0;
  for (int i = 1; i < 20; ++i) {
    term *= -x * x / ((2 * i - 1) * (2 * i));
    sum += term;
  }
  return sum;
}

// f(0), f(1), .. f(N - 1) with compile-time indices.
template <int N, class F>
__device__ __forceinline__ void unrolled(F&& f) {
  [&]<int... I>(std::integer_sequence<int, I...>) {
    (f(std::integral_constant<int, I>{}), ...);
  }(std::make_integer_sequence<int, N>{});
}

// An odd prime R: with a_i = v_i + v_{R-i} and b_i = v_i - v_{R-i},
// X_m and X_{R-m} are r -+ i s, r = v_0 + sum a_i cos(2 pi i m / R) and
// s = sum b_i sin(2 pi i m / R).
template <int R, bool INV>
__device__ __forceinline__ void dft_odd_prime(float2* v) {
  constexpr int H = (R - 1) / 2;
  float2 a[H], b[H];
  float2 sum = v[0];
#pragma unroll
  for (int i = 0; i < H; ++i) {
    a[i] = cadd(v[i + 1], v[R - 1 - i]);
    b[i] = csub(v[i + 1], v[R - 1 - i]);
    sum = cadd(sum, a[i]);
  }
  const float2 v0 = v[0];
  v[0] = sum;
  unrolled<H>([&](auto mi) {
    constexpr int m = mi + 1;
    float2 r = v0;
    float2 s = {0.0f, 0.0f};
    unrolled<H>([&](auto ii) {
      constexpr int i = ii;
      constexpr float c = static_cast<float>(turn_cosine((i + 1) * m, R));
      constexpr float d = static_cast<float>(turn_sine((i + 1) * m, R));
      r = cfma(c, a[i], r);
      s = i == 0 ? cscale(b[i], d) : cfma(d, b[i], s);
    });
    v[m] = cadd_w4<INV>(r, s);
    v[R - m] = csub_w4<INV>(r, s);
  });
}

template <int R, bool INV>
__device__ __forceinline__ void small_dft(float2* v);

// R = A B with coprime A and B (Good and Thomas): input index (B n1 + A n2)
// mod R, output index by the Chinese remainder theorem; no twiddles.
template <int A, int B, bool INV>
__device__ __forceinline__ void dft_coprime(float2* v) {
  constexpr int R = A * B;
  constexpr auto inverse = [](int x, int m) {
    for (int y = 1; y < m; ++y) {
      if (x * y % m == 1) return y;
    }
    return 0;
  };
  constexpr int kA = B * inverse(B % A, A);  // 1 mod A, 0 mod B
  constexpr int kB = A * inverse(A % B, B);  // 0 mod A, 1 mod B
  float2 t[A][B];
#pragma unroll
  for (int n1 = 0; n1 < A; ++n1) {
#pragma unroll
    for (int n2 = 0; n2 < B; ++n2) t[n1][n2] = v[(B * n1 + A * n2) % R];
    small_dft<B, INV>(t[n1]);
  }
#pragma unroll
  for (int k2 = 0; k2 < B; ++k2) {
    float2 u[A];
#pragma unroll
    for (int n1 = 0; n1 < A; ++n1) u[n1] = t[n1][k2];
    small_dft<A, INV>(u);
#pragma unroll
    for (int k1 = 0; k1 < A; ++k1) v[(kA * k1 + kB * k2) % R] = u[k1];
  }
}

// R = P P: P-point DFTs, twiddles W_R^{n1 k2}, P-point DFTs.
template <int P, bool INV>
__device__ __forceinline__ void dft_square(float2* v) {
  constexpr int R = P * P;
  float2 t[P][P];
#pragma unroll
  for (int n1 = 0; n1 < P; ++n1) {
#pragma unroll
    for (int n2 = 0; n2 < P; ++n2) t[n1][n2] = v[n1 + P * n2];
    small_dft<P, INV>(t[n1]);
  }
  unrolled<P - 1>([&](auto i) {
    unrolled<P - 1>([&](auto k) {
      constexpr int e = (i + 1) * (k + 1);
      constexpr float c = static_cast<float>(turn_cosine(e, R));
      constexpr float s = static_cast<float>(turn_sine(e, R));
      t[i + 1][k + 1] = cmul_constant<INV>(t[i + 1][k + 1], c, s);
    });
  });
#pragma unroll
  for (int k2 = 0; k2 < P; ++k2) {
    float2 u[P];
#pragma unroll
    for (int n1 = 0; n1 < P; ++n1) u[n1] = t[n1][k2];
    small_dft<P, INV>(u);
#pragma unroll
    for (int k1 = 0; k1 < P; ++k1) v[k2 + P * k1] = u[k1];
  }
}

// Points small_dft takes.
constexpr bool small_dft_length(int r) {
  return (r >= 2 && r <= 16) || r == 18 || r == 20 || r == 21 || r == 24 || r == 25;
}

template <int R, bool INV>
__device__ __forceinline__ void small_dft(float2* v) {
  static_assert(small_dft_length(R));
  if constexpr (R == 2) {
    bfly2<INV>(v[0], v[1]);
  } else if constexpr (R == 3) {
    bfly3<INV>(v[0], v[1], v[2]);
  } else if constexpr (R == 4) {
    bfly4<INV>(v[0], v[1], v[2], v[3]);
  } else if constexpr (R == 5) {
    bfly5<INV>(v[0], v[1], v[2], v[3], v[4]);
  } else if constexpr (R == 8) {
    bfly8<INV>(v);
  } else if constexpr (R == 9) {
    dft_square<3, INV>(v);
  } else if constexpr (R == 16) {
    bfly16<INV>(v);
  } else if constexpr (R == 6) {
    dft_coprime<2, 3, INV>(v);
  } else if constexpr (R == 10) {
    dft_coprime<2, 5, INV>(v);
  } else if constexpr (R == 12) {
    dft_coprime<4, 3, INV>(v);
  } else if constexpr (R == 14) {
    dft_coprime<2, 7, INV>(v);
  } else if constexpr (R == 15) {
    dft_coprime<3, 5, INV>(v);
  } else if constexpr (R == 18) {
    dft_coprime<2, 9, INV>(v);
  } else if constexpr (R == 20) {
    dft_coprime<4, 5, INV>(v);
  } else if constexpr (R == 21) {
    dft_coprime<3, 7, INV>(v);
  } else if constexpr (R == 24) {
    dft_coprime<3, 8, INV>(v);
  } else if constexpr (R == 25) {
    dft_square<5, INV>(v);
  } else {
    dft_odd_prime<R, INV>(v);
  }
}

}  // namespace qpb
