// Products with the 1-D reference-element stiffness Kh by even/odd halves
// (shared by the operator apply and the on-chip CG).
//
// Kh is centrosymmetric (Kh[a][b] = Kh[N-a][N-b]): with e_b = v_b + v_{N-b}
// and d_b = v_b - v_{N-b},
//   (Kh v)_a     = sum_b Ce[a][b] e_b + sum_b Co[a][b] d_b
//   (Kh v)_{N-a} = sum_b Ce[a][b] e_b - sum_b Co[a][b] d_b,
// about half the multiplications of the full product.
#pragma once
#include "common.cuh"

namespace seg {

template <int N>
struct Eo {
  static constexpr int H = (N + 1) / 2;       // node pairs
  static constexpr int M = (N + 1) & 1;       // 1: a middle node
  static constexpr int E = H + M;
  static constexpr int NC = E * E + H * H;    // coefficients: Ce [E][E], then Co [H][H]
};

// The coefficients of scale * Kh, each pair of mirrored entries averaged (in
// double: the products' error is the same with long double coefficients at
// every order).
template <int N, class A>
inline void eo_coefs(const double* Kh, double scale, A* cf) {
  constexpr int H = Eo<N>::H, E = Eo<N>::E, n = N + 1;
  auto sym = [&](int a, int b) {
    return 0.5 * (Kh[a * n + b] + Kh[(N - a) * n + (N - b)]);
  };
  for (int a = 0; a < E; a++)
    for (int b = 0; b < E; b++)
      cf[a * E + b] = (A)(scale * (b < H ? 0.5 * (sym(a, b) + sym(a, N - b)) : sym(a, b)));
  for (int a = 0; a < H; a++)
    for (int b = 0; b < H; b++)
      cf[E * E + a * H + b] = (A)(scale * (0.5 * (sym(a, b) - sym(a, N - b))));
}

// o = Kh v; with ENERGY returns v . o (else 0).
template <int N, bool ENERGY, class A>
__device__ __forceinline__ A eo_product(const A* cf, const A (&v)[N + 1], A (&o)[N + 1]) {
  constexpr int H = Eo<N>::H, E = Eo<N>::E;
  A e[E], d[H], s[E];
#pragma unroll
  for (int b = 0; b < H; b++) {
    e[b] = v[b] + v[N - b];
    d[b] = v[b] - v[N - b];
  }
  if constexpr (Eo<N>::M == 1) e[H] = v[H];
#pragma unroll
  for (int a = 0; a < E; a++) {
    s[a] = A(0);
#pragma unroll
    for (int b = 0; b < E; b++) s[a] = fma(cf[a * E + b], e[b], s[a]);
  }
  A en = A(0), od = A(0);
#pragma unroll
  for (int a = 0; a < H; a++) {
    A t = A(0);
#pragma unroll
    for (int b = 0; b < H; b++) t = fma(cf[E * E + a * H + b], d[b], t);
    o[a] = s[a] + t;
    o[N - a] = s[a] - t;
    // v_a o_a + v_{N-a} o_{N-a} = s e_a + t d_a
    if constexpr (ENERGY) {
      en = fma(s[a], e[a], en);
      od = fma(t, d[a], od);
    }
  }
  if constexpr (Eo<N>::M == 1) {
    o[H] = s[H];
    if constexpr (ENERGY) en = fma(s[H], e[H], en);
  }
  return en + od;
}

}  // namespace seg
