// Register DFTs shared by the fused FFT kernels (fft_dc.cu, fft_rows.cu): lengths 1 to 16, forward
// (DIR > 0, e^{-2 pi i / R}) and inverse (DIR < 0), unnormalised, natural order in and out.
#pragma once

#include "llr_common.cuh"

namespace llr {
namespace {

// x * W where W = tw (forward) or conj(tw) (inverse)
template <int DIR>
__device__ __forceinline__ float2 twmul(float2 x, float2 tw) {
  return DIR > 0 ? cmul(x, tw) : cmul_bc(x, tw);
}

// -i * x (forward) / +i * x (inverse)
template <int DIR>
__device__ __forceinline__ float2 rot(float2 x) {
  return DIR > 0 ? make_float2(x.y, -x.x) : make_float2(-x.y, x.x);
}

template <int R, int DIR>
struct Dft;

template <int DIR>
struct Dft<1, DIR> {
  __device__ __forceinline__ static void run(float2* v, const float2*) {}
};

template <int DIR>
struct Dft<2, DIR> {
  __device__ __forceinline__ static void run(float2* v, const float2*) {
    const float2 a = v[0], b = v[1];
    v[0] = cadd(a, b);
    v[1] = csub(a, b);
  }
};

template <int DIR>
struct Dft<3, DIR> {
  __device__ __forceinline__ static void run(float2* v, const float2*) {
    const float s = 0.86602540378443864676f;   // sin(2 pi / 3)
    const float2 a = v[0], b = v[1], c = v[2];
    const float2 t1 = cadd(b, c);
    const float2 t2 = make_float2(a.x - 0.5f * t1.x, a.y - 0.5f * t1.y);
    const float2 t3 = cscale(csub(b, c), s);
    const float2 r = rot<DIR>(t3);   // -i s (b - c) forward
    v[0] = cadd(a, t1);
    v[1] = cadd(t2, r);
    v[2] = csub(t2, r);
  }
};

template <int DIR>
struct Dft<4, DIR> {
  __device__ __forceinline__ static void run(float2* v, const float2*) {
    const float2 a = v[0], b = v[1], c = v[2], d = v[3];
    const float2 s0 = cadd(a, c), s1 = csub(a, c), s2 = cadd(b, d), s3 = rot<DIR>(csub(b, d));
    v[0] = cadd(s0, s2);
    v[2] = csub(s0, s2);
    v[1] = cadd(s1, s3);
    v[3] = csub(s1, s3);
  }
};

// W_R^m = e^{-2 pi i m / R} for the register DFTs, evaluated at compile time from the Taylor
// series of cos and sin in double precision (|x| <= 2 pi, 30 terms).
constexpr double kTwoPi = 6.283185307179586476925286766559;
constexpr double taylor_cos(double x) {
  double t = 1.0, s = 1.0;
  for (int k = 1; k < 30; ++k) { t *= -x * x / ((2.0 * k - 1.0) * (2.0 * k)); s += t; }
  return s;
}
constexpr double taylor_sin(double x) {
  double t = x, s = x;
  for (int k = 1; k < 30; ++k) { t *= -x * x / ((2.0 * k) * (2.0 * k + 1.0)); s += t; }
  return s;
}
template <int R>
struct TwTab {
  float re[R], im[R];
  constexpr TwTab() : re(), im() {
    for (int m = 0; m < R; ++m) {
      re[m] = (float)taylor_cos(kTwoPi * m / R);
      im[m] = (float)-taylor_sin(kTwoPi * m / R);
    }
  }
};
template <int R>
__device__ constexpr TwTab<R> kTw = TwTab<R>();

// R = R1 * R2 Cooley-Tukey in registers: input natural order n = R2 n1 + n2, output natural
// order k = k1 + R1 k2; twiddles W_R^{n2 k1} are compile-time constants.
template <int R1, int R2, int DIR>
__device__ __forceinline__ void dft_ct(float2* v, const float2*, const float2* w1, const float2* w2) {
  constexpr int R = R1 * R2;
  float2 a[R];
#pragma unroll
  for (int n2 = 0; n2 < R2; ++n2) {
    float2 t[R1];
#pragma unroll
    for (int n1 = 0; n1 < R1; ++n1) t[n1] = v[R2 * n1 + n2];
    Dft<R1, DIR>::run(t, w1);
#pragma unroll
    for (int k1 = 0; k1 < R1; ++k1) {
      const int m = (n2 * k1) % R;
      a[k1 * R2 + n2] = m == 0 ? t[k1] : twmul<DIR>(t[k1], make_float2(kTw<R>.re[m], kTw<R>.im[m]));
    }
  }
#pragma unroll
  for (int k1 = 0; k1 < R1; ++k1) {
    float2 t[R2];
#pragma unroll
    for (int n2 = 0; n2 < R2; ++n2) t[n2] = a[k1 * R2 + n2];
    Dft<R2, DIR>::run(t, w2);
#pragma unroll
    for (int k2 = 0; k2 < R2; ++k2) v[k1 + R1 * k2] = t[k2];
  }
}

// Odd prime R: with s_n = x_n + x_{R-n} and d_n = x_n - x_{R-n}, X_k and X_{R-k} share
// x_0 + sum s_n cos(2 pi k n / R) and differ in the sign of i sum d_n sin(2 pi k n / R).
template <int R, int DIR>
__device__ __forceinline__ void dft_prime(float2* v) {
  constexpr int H = (R - 1) / 2;
  float2 s[H], d[H];
#pragma unroll
  for (int n = 1; n <= H; ++n) {
    s[n - 1] = cadd(v[n], v[R - n]);
    d[n - 1] = csub(v[n], v[R - n]);
  }
  const float2 x0 = v[0];
#pragma unroll
  for (int n = 0; n < H; ++n) v[0] = cadd(v[0], s[n]);
#pragma unroll
  for (int k = 1; k <= H; ++k) {
    float2 a = x0, b = make_float2(0.f, 0.f);
#pragma unroll
    for (int n = 1; n <= H; ++n) {
      const float c = kTw<R>.re[(k * n) % R], sn = -kTw<R>.im[(k * n) % R];
      a.x = fmaf(s[n - 1].x, c, a.x);
      a.y = fmaf(s[n - 1].y, c, a.y);
      b.x = fmaf(d[n - 1].x, sn, b.x);
      b.y = fmaf(d[n - 1].y, sn, b.y);
    }
    const float2 r = rot<DIR>(b);
    v[k] = cadd(a, r);
    v[R - k] = csub(a, r);
  }
}

template <int DIR>
struct Dft<5, DIR> {
  __device__ __forceinline__ static void run(float2* v, const float2*) { dft_prime<5, DIR>(v); }
};
template <int DIR>
struct Dft<7, DIR> {
  __device__ __forceinline__ static void run(float2* v, const float2*) { dft_prime<7, DIR>(v); }
};
template <int DIR>
struct Dft<11, DIR> {
  __device__ __forceinline__ static void run(float2* v, const float2*) { dft_prime<11, DIR>(v); }
};
template <int DIR>
struct Dft<13, DIR> {
  __device__ __forceinline__ static void run(float2* v, const float2*) { dft_prime<13, DIR>(v); }
};
template <int DIR>
struct Dft<9, DIR> {
  __device__ __forceinline__ static void run(float2* v, const float2* w) { dft_ct<3, 3, DIR>(v, w, nullptr, nullptr); }
};
template <int DIR>
struct Dft<10, DIR> {
  __device__ __forceinline__ static void run(float2* v, const float2* w) { dft_ct<5, 2, DIR>(v, w, nullptr, nullptr); }
};
template <int DIR>
struct Dft<14, DIR> {
  __device__ __forceinline__ static void run(float2* v, const float2* w) { dft_ct<7, 2, DIR>(v, w, nullptr, nullptr); }
};
template <int DIR>
struct Dft<15, DIR> {
  __device__ __forceinline__ static void run(float2* v, const float2* w) { dft_ct<5, 3, DIR>(v, w, nullptr, nullptr); }
};
template <int DIR>
struct Dft<6, DIR> {
  __device__ __forceinline__ static void run(float2* v, const float2* w) { dft_ct<3, 2, DIR>(v, w, nullptr, nullptr); }
};
template <int DIR>
struct Dft<8, DIR> {
  __device__ __forceinline__ static void run(float2* v, const float2* w) { dft_ct<4, 2, DIR>(v, w, nullptr, nullptr); }
};
template <int DIR>
struct Dft<12, DIR> {
  __device__ __forceinline__ static void run(float2* v, const float2* w) { dft_ct<4, 3, DIR>(v, w, nullptr, nullptr); }
};
template <int DIR>
struct Dft<16, DIR> {
  __device__ __forceinline__ static void run(float2* v, const float2* w) { dft_ct<4, 4, DIR>(v, w, nullptr, nullptr); }
};

// f(Radix<R>{}) for the run-time radix R in 1..16.
template <int R>
struct Radix {
  static constexpr int value = R;
};
template <class F>
__device__ __forceinline__ void with_radix(int R, F f) {
  switch (R) {
    case 1: f(Radix<1>{}); break;
    case 2: f(Radix<2>{}); break;
    case 3: f(Radix<3>{}); break;
    case 4: f(Radix<4>{}); break;
    case 5: f(Radix<5>{}); break;
    case 6: f(Radix<6>{}); break;
    case 7: f(Radix<7>{}); break;
    case 8: f(Radix<8>{}); break;
    case 9: f(Radix<9>{}); break;
    case 10: f(Radix<10>{}); break;
    case 11: f(Radix<11>{}); break;
    case 12: f(Radix<12>{}); break;
    case 13: f(Radix<13>{}); break;
    case 14: f(Radix<14>{}); break;
    case 15: f(Radix<15>{}); break;
    case 16: f(Radix<16>{}); break;
    default: break;
  }
}

}  // namespace

// n = n1 n2 with both at most 16, as balanced as possible (false: none).
inline bool radix_split(int n, int& n1, int& n2) {
  int best = -1;
  for (int a = 16; a >= 1; --a)
    if (n % a == 0 && n / a <= 16) {
      const int b = n / a, bal = a > b ? a - b : b - a;
      if (best < 0 || bal < best) { best = bal; n1 = a; n2 = b; }
    }
  return best >= 0;
}

}  // namespace llr
