// Forward R-point DFT butterflies of the composite radices 6, 9, 10, 12, 14
// and 15, built in registers from the generated prime and power-of-two
// codelets. Coprime factors use the Good-Thomas index maps (no twiddles):
// inputs n = (N2 n1 + N1 n2) mod N, outputs k = (e1 k1 + e2 k2) mod N with
// e1 = 1 mod N1, 0 mod N2 and e2 = 0 mod N1, 1 mod N2. 9 = 3 x 3 needs the
// four W9 products between its two layers.
#pragma once
#include "codelets.cuh"

namespace fftz {

__host__ __device__ constexpr int pfa_inv(int a, int m) {  // a^-1 mod m
  for (int x = 1; x < m; x++)
    if ((a * x) % m == 1) return x;
  return 0;
}

template <int N1, int N2> struct DftPfa {
  template <typename T, typename T2>
  static __device__ __forceinline__ void apply(T2 (&v)[N1 * N2]) {
    constexpr int N = N1 * N2;
    constexpr int E1 = N2 * pfa_inv(N2 % N1, N1), E2 = N1 * pfa_inv(N1 % N2, N2);
    T2 a[N1][N2];
#pragma unroll
    for (int n1 = 0; n1 < N1; n1++) {
#pragma unroll
      for (int n2 = 0; n2 < N2; n2++) a[n1][n2] = v[(N2 * n1 + N1 * n2) % N];
      Dft<N2>::template apply<T, T2>(a[n1]);
    }
#pragma unroll
    for (int k2 = 0; k2 < N2; k2++) {
      T2 c[N1];
#pragma unroll
      for (int n1 = 0; n1 < N1; n1++) c[n1] = a[n1][k2];
      Dft<N1>::template apply<T, T2>(c);
#pragma unroll
      for (int k1 = 0; k1 < N1; k1++) v[(E1 * k1 + E2 * k2) % N] = c[k1];
    }
  }
};

template <> struct Dft<1> {  // one-point lines
  template <typename T, typename T2>
  static __device__ __forceinline__ void apply(T2 (&)[1]) {}
};
template <> struct Dft<6> : DftPfa<2, 3> {};
template <> struct Dft<10> : DftPfa<2, 5> {};
template <> struct Dft<12> : DftPfa<4, 3> {};
template <> struct Dft<14> : DftPfa<2, 7> {};
template <> struct Dft<15> : DftPfa<3, 5> {};

template <> struct Dft<9> {
  template <typename T, typename T2>
  static __device__ __forceinline__ void apply(T2 (&v)[9]) {
    // W9^1, W9^2, W9^4 = e^{-2 pi i {40, 80, 160} deg / 360}
    const T c1 = T(0.766044443118978035), s1 = T(0.642787609686539326);
    const T c2 = T(0.173648177666930349), s2 = T(0.984807753012208059);
    const T c4 = T(-0.939692620785908384), s4 = T(0.342020143325668733);
    T2 a[3][3];
#pragma unroll
    for (int n2 = 0; n2 < 3; n2++) {
#pragma unroll
      for (int n1 = 0; n1 < 3; n1++) a[n2][n1] = v[3 * n1 + n2];
      Dft<3>::template apply<T, T2>(a[n2]);
    }
    auto rot = [](T2 x, T c, T s) {  // x * (c - i s)
      T2 r;
      r.x = x.x * c + x.y * s;
      r.y = x.y * c - x.x * s;
      return r;
    };
    a[1][1] = rot(a[1][1], c1, s1);
    a[1][2] = rot(a[1][2], c2, s2);
    a[2][1] = rot(a[2][1], c2, s2);
    a[2][2] = rot(a[2][2], c4, s4);
#pragma unroll
    for (int k1 = 0; k1 < 3; k1++) {
      T2 c[3] = {a[0][k1], a[1][k1], a[2][k1]};
      Dft<3>::template apply<T, T2>(c);
#pragma unroll
      for (int k2 = 0; k2 < 3; k2++) v[k1 + 3 * k2] = c[k2];
    }
  }
};

}  // namespace fftz
