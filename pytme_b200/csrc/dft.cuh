// Complex arithmetic and the small DFTs in registers that every own transform is built from:
// the columns of colfft.cuh, the line FFTs of linefft.cuh, the Stockham passes of
// mixed-precision plans and the scan's four-step z pass.
#pragma once

#include <cuda_runtime.h>
#include <cstdint>

namespace tmb {
namespace fft {

__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
  return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ float2 cconj(float2 a) { return make_float2(a.x, -a.y); }
__device__ __forceinline__ float2 cscale(float2 a, float s) { return make_float2(a.x * s, a.y * s); }

// multiply by -i (forward, DIR=-1) or +i (inverse, DIR=+1)
template <int DIR>
__device__ __forceinline__ float2 rot90(float2 a) {
  return DIR < 0 ? make_float2(a.y, -a.x) : make_float2(-a.y, a.x);
}

// ---- small DFTs in registers; DIR = -1 computes sum_j v_j exp(-2 pi i jk/R)
template <int DIR>
__device__ __forceinline__ void dft2(float2* v) {
  float2 a = v[0], b = v[1];
  v[0] = cadd(a, b);
  v[1] = csub(a, b);
}

template <int DIR>
__device__ __forceinline__ void dft3(float2* v) {
  const float c = -0.5f;
  const float s = (DIR < 0 ? -1.f : 1.f) * 0.86602540378443864676f;
  float2 t1 = cadd(v[1], v[2]);
  float2 t2 = csub(v[1], v[2]);
  float2 m = make_float2(v[0].x + c * t1.x, v[0].y + c * t1.y);
  float2 r = make_float2(-s * t2.y, s * t2.x);  // i * s * t2
  v[0] = cadd(v[0], t1);
  v[1] = cadd(m, r);
  v[2] = csub(m, r);
}

template <int DIR>
__device__ __forceinline__ void dft4(float2* v) {
  float2 a0 = cadd(v[0], v[2]);
  float2 a1 = csub(v[0], v[2]);
  float2 a2 = cadd(v[1], v[3]);
  float2 a3 = rot90<DIR>(csub(v[1], v[3]));
  v[0] = cadd(a0, a2);
  v[2] = csub(a0, a2);
  v[1] = cadd(a1, a3);
  v[3] = csub(a1, a3);
}

template <int DIR>
__device__ __forceinline__ void dft5(float2* v) {
  // Winograd-style 5-point DFT with constants from cos/sin(2 pi / 5), cos/sin(4 pi / 5).
  const float c1 = 0.30901699437494742410f;   // cos(2pi/5)
  const float c2 = -0.80901699437494742410f;  // cos(4pi/5)
  const float sg = DIR < 0 ? -1.f : 1.f;
  const float s1 = sg * 0.95105651629515357212f;  // sin(2pi/5)
  const float s2 = sg * 0.58778525229247312917f;  // sin(4pi/5)
  float2 a1 = cadd(v[1], v[4]), b1 = csub(v[1], v[4]);
  float2 a2 = cadd(v[2], v[3]), b2 = csub(v[2], v[3]);
  float2 x0 = v[0];
  float2 m1 = make_float2(x0.x + c1 * a1.x + c2 * a2.x, x0.y + c1 * a1.y + c2 * a2.y);
  float2 m2 = make_float2(x0.x + c2 * a1.x + c1 * a2.x, x0.y + c2 * a1.y + c1 * a2.y);
  // i * (s1 b1 + s2 b2), i * (s2 b1 - s1 b2)
  float2 n1 = make_float2(-(s1 * b1.y + s2 * b2.y), s1 * b1.x + s2 * b2.x);
  float2 n2 = make_float2(-(s2 * b1.y - s1 * b2.y), s2 * b1.x - s1 * b2.x);
  v[0] = make_float2(x0.x + a1.x + a2.x, x0.y + a1.y + a2.y);
  v[1] = cadd(m1, n1);
  v[4] = csub(m1, n1);
  v[2] = cadd(m2, n2);
  v[3] = csub(m2, n2);
}

template <int DIR>
__device__ __forceinline__ void dft8(float2* v) {
  const float h = 0.70710678118654752440f;
  float2 e[4] = {v[0], v[2], v[4], v[6]};
  float2 o[4] = {v[1], v[3], v[5], v[7]};
  dft4<DIR>(e);
  dft4<DIR>(o);
  // o[k] *= exp(DIR * 2 pi i k / 8)
  o[1] = DIR < 0 ? make_float2(h * (o[1].x + o[1].y), h * (o[1].y - o[1].x))
                 : make_float2(h * (o[1].x - o[1].y), h * (o[1].y + o[1].x));
  o[2] = rot90<DIR>(o[2]);
  o[3] = DIR < 0 ? make_float2(h * (o[3].y - o[3].x), -h * (o[3].x + o[3].y))
                 : make_float2(-h * (o[3].x + o[3].y), h * (o[3].x - o[3].y));
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    v[k] = cadd(e[k], o[k]);
    v[k + 4] = csub(e[k], o[k]);
  }
}

// ---- small DFTs of compile-time size in registers (DIR -1 forward, +1 inverse)
// 16 = 4 x 4 and 9 = 3 x 3 Cooley-Tukey with their constant twiddles; 7, 11, 13 by the
// symmetry of an odd prime; 6, 10, 12, 14, 15, 20 = Good-Thomas prime-factor forms (coprime
// factors, no twiddles).
template <int DIR>
__device__ __forceinline__ void dft16(float2* v) {
  const float c1 = 0.92387953251128675613f, s1 = 0.38268343236508977173f;
  const float h = 0.70710678118654752440f;
  const float sg = DIR < 0 ? -1.f : 1.f;
  // w16^j for j = 0..9 (exp(DIR * 2 pi i j / 16))
  const float2 w[10] = {make_float2(1.f, 0.f), make_float2(c1, sg * s1), make_float2(h, sg * h),
                        make_float2(s1, sg * c1), make_float2(0.f, sg * 1.f),
                        make_float2(-s1, sg * c1), make_float2(-h, sg * h),
                        make_float2(-c1, sg * s1), make_float2(-1.f, 0.f),
                        make_float2(-c1, -sg * s1)};
  float2 a[4][4];
#pragma unroll
  for (int n1 = 0; n1 < 4; ++n1) {
#pragma unroll
    for (int n2 = 0; n2 < 4; ++n2) a[n1][n2] = v[4 * n2 + n1];
    dft4<DIR>(a[n1]);
#pragma unroll
    for (int k2 = 1; k2 < 4; ++k2) {
      const int e = n1 * k2;
      if (e) a[n1][k2] = cmul(a[n1][k2], w[e]);
    }
  }
#pragma unroll
  for (int k2 = 0; k2 < 4; ++k2) {
    float2 b[4] = {a[0][k2], a[1][k2], a[2][k2], a[3][k2]};
    dft4<DIR>(b);
#pragma unroll
    for (int k1 = 0; k1 < 4; ++k1) v[k2 + 4 * k1] = b[k1];
  }
}

// 9 = 3 x 3 Cooley-Tukey with its constant twiddles w9^1, w9^2, w9^4.
template <int DIR>
__device__ __forceinline__ void dft9(float2* v) {
  const float sg = DIR < 0 ? -1.f : 1.f;
  const float2 w1 = make_float2(0.76604444311897803520f, sg * 0.64278760968653932632f);
  const float2 w2 = make_float2(0.17364817766693034885f, sg * 0.98480775301220805937f);
  const float2 w4 = make_float2(-0.93969262078590838405f, sg * 0.34202014332566873304f);
  float2 a[3][3];
#pragma unroll
  for (int n1 = 0; n1 < 3; ++n1) {
#pragma unroll
    for (int n2 = 0; n2 < 3; ++n2) a[n1][n2] = v[3 * n2 + n1];
    dft3<DIR>(a[n1]);
  }
  a[1][1] = cmul(a[1][1], w1);
  a[1][2] = cmul(a[1][2], w2);
  a[2][1] = cmul(a[2][1], w2);
  a[2][2] = cmul(a[2][2], w4);
#pragma unroll
  for (int k2 = 0; k2 < 3; ++k2) {
    float2 b[3] = {a[0][k2], a[1][k2], a[2][k2]};
    dft3<DIR>(b);
#pragma unroll
    for (int k1 = 0; k1 < 3; ++k1) v[k2 + 3 * k1] = b[k1];
  }
}

// Odd prime P by its symmetry: with a_k = v[k] + v[P-k], b_k = v[k] - v[P-k],
// X[j], X[P-j] = v[0] + sum_k cos(2 pi jk/P) a_k  +- DIR i sum_k sin(2 pi jk/P) b_k.
template <int P, int DIR>
__device__ __forceinline__ void dft_odd_prime(float2* v) {
  static_assert(P == 7 || P == 11 || P == 13, "unsupported prime");
  constexpr int H = (P - 1) / 2;
  // cos and sin of 2 pi j / P
  const float c7[4] = {1.f, 0.62348980185873353053f, -0.22252093395631440429f,
                       -0.90096886790241912624f};
  const float s7[4] = {0.f, 0.78183148246802980871f, 0.97492791218182360702f,
                       0.43388373911755812048f};
  const float c11[6] = {1.f, 0.84125353283118116886f, 0.41541501300188642553f,
                        -0.14231483827328514044f, -0.65486073394528506406f,
                        -0.95949297361449738989f};
  const float s11[6] = {0.f, 0.54064081745559758211f, 0.90963199535451837141f,
                        0.98982144188093273237f, 0.75574957435425828378f,
                        0.28173255684142969771f};
  const float c13[7] = {1.f, 0.88545602565320989590f, 0.56806474673115580251f,
                        0.12053668025532305335f, -0.35460488704253562597f,
                        -0.74851074817110109863f, -0.97094181742605202716f};
  const float s13[7] = {0.f, 0.46472317204376854566f, 0.82298386589365639458f,
                        0.99270887409805399280f, 0.93501624268541482344f,
                        0.66312265824079520238f, 0.23931566428755776715f};
  float2 a[H + 1], b[H + 1];
  float2 sum = v[0];
#pragma unroll
  for (int k = 1; k <= H; ++k) {
    a[k] = cadd(v[k], v[P - k]);
    b[k] = csub(v[k], v[P - k]);
    sum = cadd(sum, a[k]);
  }
  const float2 v0 = v[0];
#pragma unroll
  for (int j = 1; j <= H; ++j) {
    float2 m = v0, n = make_float2(0.f, 0.f);
#pragma unroll
    for (int k = 1; k <= H; ++k) {
      const int e = (j * k) % P;
      const int f = e <= H ? e : P - e;
      const float c = P == 7 ? c7[f & 3] : P == 11 ? c11[f % 6] : c13[f];
      const float s = (DIR < 0 ? -1.f : 1.f) * (e <= H ? 1.f : -1.f) *
                      (P == 7 ? s7[f & 3] : P == 11 ? s11[f % 6] : s13[f]);
      m.x += c * a[k].x;
      m.y += c * a[k].y;
      n.x -= s * b[k].y;  // i s b
      n.y += s * b[k].x;
    }
    v[j] = cadd(m, n);
    v[P - j] = csub(m, n);
  }
  v[0] = sum;
}

constexpr int modinv(int a, int m) {
  for (int x = 1; x < m; ++x)
    if ((a * x) % m == 1) return x;
  return 1;
}

template <int R, int DIR>
__device__ __forceinline__ void dft_prime_or_pow2(float2* v) {
  if constexpr (R == 2) dft2<DIR>(v);
  else if constexpr (R == 3) dft3<DIR>(v);
  else if constexpr (R == 4) dft4<DIR>(v);
  else if constexpr (R == 5) dft5<DIR>(v);
  else if constexpr (R == 7 || R == 11 || R == 13) dft_odd_prime<R, DIR>(v);
  else if constexpr (R == 8) dft8<DIR>(v);
  else dft16<DIR>(v);
}

template <int N1, int N2, int DIR>
__device__ __forceinline__ void dft_pfa(float2* v) {
  constexpr int N = N1 * N2;
  constexpr int K1 = N2 * modinv(N2 % N1, N1);
  constexpr int K2 = N1 * modinv(N1 % N2, N2);
  float2 a[N2][N1];
#pragma unroll
  for (int n2 = 0; n2 < N2; ++n2) {
#pragma unroll
    for (int n1 = 0; n1 < N1; ++n1) a[n2][n1] = v[(N2 * n1 + N1 * n2) % N];
    dft_prime_or_pow2<N1, DIR>(a[n2]);
  }
#pragma unroll
  for (int k1 = 0; k1 < N1; ++k1) {
    float2 b[N2];
#pragma unroll
    for (int n2 = 0; n2 < N2; ++n2) b[n2] = a[n2][k1];
    dft_prime_or_pow2<N2, DIR>(b);
#pragma unroll
    for (int k2 = 0; k2 < N2; ++k2) v[(K1 * k1 + K2 * k2) % N] = b[k2];
  }
}

template <int N, int DIR>
__device__ __forceinline__ void dft_small(float2* v) {
  if constexpr (N == 1) {
  } else if constexpr (N == 2 || N == 3 || N == 4 || N == 5 || N == 7 || N == 8 || N == 11 ||
                       N == 13 || N == 16) {
    dft_prime_or_pow2<N, DIR>(v);
  } else if constexpr (N == 9) dft9<DIR>(v);
  else if constexpr (N == 14) dft_pfa<2, 7, DIR>(v);
  else if constexpr (N == 6) dft_pfa<2, 3, DIR>(v);
  else if constexpr (N == 10) dft_pfa<2, 5, DIR>(v);
  else if constexpr (N == 12) dft_pfa<4, 3, DIR>(v);
  else if constexpr (N == 15) dft_pfa<3, 5, DIR>(v);
  else if constexpr (N == 20) dft_pfa<4, 5, DIR>(v);
  else static_assert(N == 0, "unsupported small DFT size");
}

}  // namespace fft
}  // namespace tmb
