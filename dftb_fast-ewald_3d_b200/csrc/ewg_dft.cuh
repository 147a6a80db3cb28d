// ewg_dft.cuh -- small DFTs held in registers, N = 2 .. 24, natural order in and
// out, no twiddle table: composite lengths split into coprime factors by the
// prime-factor algorithm (Good 1958, Thomas 1963; no twiddles), 9 and 16 by
// Cooley-Tukey with constant roots.
#pragma once

#include "ewg_fft.cuh"

namespace ewg {

// cos and sin of 2 pi e / N for the Cooley-Tukey splits (N = 9: e in {1, 2, 4};
// N = 16: e in {1, 2, 3, 4, 6, 9}).
__host__ __device__ constexpr double root_cos(int n, int e) {
  return n == 9 ? (e == 1 ? 0.76604444311897803520
                          : (e == 2 ? 0.17364817766693034885 : -0.93969262078590838405))
                : (e == 1   ? 0.92387953251128675613
                   : e == 2 ? 0.70710678118654752440
                   : e == 3 ? 0.38268343236508977173
                   : e == 4 ? 0.0
                   : e == 6 ? -0.70710678118654752440
                            : -0.92387953251128675613);
}
__host__ __device__ constexpr double root_sin(int n, int e) {
  return n == 9 ? (e == 1 ? 0.64278760968653932632
                          : (e == 2 ? 0.98480775301220805937 : 0.34202014332566873304))
                : (e == 1   ? 0.38268343236508977173
                   : e == 2 ? 0.70710678118654752440
                   : e == 3 ? 0.92387953251128675613
                   : e == 4 ? 1.0
                   : e == 6 ? 0.70710678118654752440
                            : -0.38268343236508977173);
}

// First coprime factor of a composite register length (the other is N / first).
__host__ __device__ constexpr int pfa_first(int n) {
  return n == 12 || n == 20 ? 4 : n == 24 ? 8 : n == 15 || n == 21 ? 3 : 2;
}
// x with a x = 1 mod b.
__host__ __device__ constexpr int inv_mod(int a, int b) {
  int x = 1;
  while (a * x % b != 1 % b) ++x;
  return x;
}

template <typename R, int SIGN, int N>
__device__ __forceinline__ void dft_reg(cx<R>* u) {
  if constexpr (N == 2 || N == 3 || N == 4 || N == 5 || N == 7 || N == 8) {
    dft_fixed<R, SIGN, N>(u, nullptr, N);
  } else if constexpr (N == 9 || N == 16) {
    constexpr int P = N == 9 ? 3 : 4;
    cx<R> t[N];
#pragma unroll
    for (int n2 = 0; n2 < P; ++n2) {
      cx<R> v[P];
#pragma unroll
      for (int n1 = 0; n1 < P; ++n1) v[n1] = u[P * n1 + n2];
      dft_reg<R, SIGN, P>(v);
#pragma unroll
      for (int k1 = 0; k1 < P; ++k1) {
        const int e = n2 * k1;
        if (e == 0)
          t[k1 * P + n2] = v[k1];
        else if (N == 16 && e == 4)
          t[k1 * P + n2] = mul_si<R, SIGN>(v[k1]);
        else
          t[k1 * P + n2] = mul(v[k1], mk(R(root_cos(N, e)), R(SIGN * root_sin(N, e))));
      }
    }
#pragma unroll
    for (int k1 = 0; k1 < P; ++k1) {
      dft_reg<R, SIGN, P>(t + k1 * P);
#pragma unroll
      for (int k2 = 0; k2 < P; ++k2) u[k1 + P * k2] = t[k1 * P + k2];
    }
  } else {
    constexpr int A = pfa_first(N), B = N / A;
    constexpr int eA = B * inv_mod(B, A), eB = A * inv_mod(A, B);
    static_assert(A * B == N, "coprime split");
    cx<R> t[N];
#pragma unroll
    for (int n2 = 0; n2 < B; ++n2) {
      cx<R> v[A];
#pragma unroll
      for (int n1 = 0; n1 < A; ++n1) v[n1] = u[(B * n1 + A * n2) % N];
      dft_reg<R, SIGN, A>(v);
#pragma unroll
      for (int k1 = 0; k1 < A; ++k1) t[k1 * B + n2] = v[k1];
    }
#pragma unroll
    for (int k1 = 0; k1 < A; ++k1) {
      dft_reg<R, SIGN, B>(t + k1 * B);
#pragma unroll
      for (int k2 = 0; k2 < B; ++k2) u[(eA * k1 + eB * k2) % N] = t[k1 * B + k2];
    }
  }
}

}  // namespace ewg
