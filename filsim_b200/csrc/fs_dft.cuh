// fs_dft.cuh -- small discrete Fourier transforms in registers, for double and
// for packed FP32 pairs.
//
// Dft<R, T>::run(re, im) is the forward R-point transform (kernel exp(-2 pi i jk / R),
// natural order in and out) of values held in registers. T is double (one line per
// thread) or F2 (two lines per thread: the two halves of each packed register pair
// belong to two lines, so a butterfly costs one instruction for both). The inverse
// transform is the same code with re and im exchanged.
#pragma once
#include "fs_f32x2.cuh"

// a packed pair of floats with arithmetic operators
struct F2 {
  f2p v;
  static __device__ __forceinline__ F2 c(double x) { return {f2_pack((float)x, (float)x)}; }
  // a b + d
  static __device__ __forceinline__ F2 fma(F2 a, F2 b, F2 d) { return {f2_fma(a.v, b.v, d.v)}; }
};
__device__ __forceinline__ F2 operator+(F2 a, F2 b) { return {f2_add(a.v, b.v)}; }
__device__ __forceinline__ F2 operator-(F2 a, F2 b) { return {f2_sub(a.v, b.v)}; }
__device__ __forceinline__ F2 operator*(F2 a, F2 b) { return {f2_mul(a.v, b.v)}; }
__device__ __forceinline__ F2 operator-(F2 a) { return {f2_neg(a.v)}; }

template <typename T>
struct Num;
template <>
struct Num<double> {
  static constexpr bool IS_DOUBLE = true;
  static __host__ __device__ __forceinline__ double c(double x) { return x; }
  static __host__ __device__ __forceinline__ double fma(double a, double b, double d) { return ::fma(a, b, d); }
};
template <>
struct Num<F2> {
  static constexpr bool IS_DOUBLE = false;
  static __device__ __forceinline__ F2 c(double x) { return F2::c(x); }
  static __device__ __forceinline__ F2 fma(F2 a, F2 b, F2 d) { return F2::fma(a, b, d); }
};

// cos and sin of 2 pi j / n at compile time, to the last place: the angle is reduced
// to t = pi a / b below pi / 4 with its rounding error r carried along, and the
// Maclaurin series (its first dropped term is below 1e-22) is summed by Horner's
// rule and corrected to first order in r.
constexpr double veltkamp_hi(double x) { return 134217729.0 * x - (134217729.0 * x - x); }
struct Angle {
  double t, r;
};
constexpr Angle pi_fraction(int a, int b) {  // |a|, b below 2^12, so that the partial products are exact
  const double p1 = 3.14159265160560607910156250, p2 = 1.98418714791870343106e-9, p3 = 1.14423774522196636802e-17;
  const double t = (p1 * a + (p2 * a + p3 * a)) / b, t1 = veltkamp_hi(t), t2 = t - t1;
  return {t, ((p1 * a - t1 * b) + (p2 * a - t2 * b) + p3 * a) / b};
}
constexpr double horner_cos(double t) {
  double s = 1.0;
  for (int k = 11; k >= 2; --k) s = 1.0 - s * t * t / ((2 * k - 1) * (2 * k));
  return 1.0 - s * t * t / 2;
}
constexpr double horner_sin(double t) {
  double s = 1.0;
  for (int k = 11; k >= 2; --k) s = 1.0 - s * t * t / ((2 * k) * (2 * k + 1));
  return t - s * t * t * t / 6;
}
constexpr double sin_pi(int a, int b) {
  const Angle g = pi_fraction(a, b);
  return horner_sin(g.t) + g.r * horner_cos(g.t);
}
constexpr double cos_pi(int a, int b) {
  const Angle g = pi_fraction(a, b);
  return horner_cos(g.t) - g.r * horner_sin(g.t);
}
constexpr double dft_sin(int j, int n) {
  j %= n;
  if (j < 0) j += n;
  if (2 * j > n) return -dft_sin(n - j, n);
  if (4 * j > n) return 8 * j > 3 * n ? sin_pi(n - 2 * j, n) : cos_pi(4 * j - n, 2 * n);
  return 8 * j > n ? cos_pi(n - 4 * j, 2 * n) : sin_pi(2 * j, n);
}
constexpr double dft_cos(int j, int n) {
  // cos(2 pi j / n) = sin(2 pi (4 j + n) / (4 n))
  return dft_sin(4 * j + n, 4 * n);
}
template <int J, int N>
struct Root {
  static constexpr double c = dft_cos(J, N), s = dft_sin(J, N);
};
#define DFT_FN static __host__ __device__ __forceinline__

// (re, im) times exp(-2 pi i J / N), J and N compile-time
template <int J, int N, typename T>
__host__ __device__ __forceinline__ void mul_root(T &re, T &im) {
  constexpr int j = J % N;
  if constexpr (j == 0) {
    return;
  } else if constexpr (4 * j == N) {  // -i
    const T t = re;
    re = im;
    im = Num<T>::c(0.0) - t;
  } else if constexpr (2 * j == N) {
    re = Num<T>::c(0.0) - re;
    im = Num<T>::c(0.0) - im;
  } else if constexpr (8 * j == N) {  // (1 - i) / sqrt 2
    const T s = Num<T>::c(Root<1, 8>::c), a = re + im, b = im - re;
    re = a * s;
    im = b * s;
  } else if constexpr (8 * j == 3 * N) {  // (-1 - i) / sqrt 2
    const T s = Num<T>::c(Root<1, 8>::c), ms = Num<T>::c(-Root<1, 8>::c), a = im - re, b = re + im;
    re = a * s;
    im = b * ms;
  } else {
    constexpr double wr = Root<j, N>::c, wi = -Root<j, N>::s;
    const T cr = Num<T>::c(wr), ci = Num<T>::c(wi), mi = Num<T>::c(-wi);
    const T a = Num<T>::fma(im, mi, re * cr), b = Num<T>::fma(re, ci, im * cr);
    re = a;
    im = b;
  }
}

template <int R, typename T>
struct Dft;

template <typename T>
struct Dft<1, T> {
  DFT_FN void run(T (&)[1], T (&)[1]) {}
};
template <typename T>
struct Dft<2, T> {
  DFT_FN void run(T (&re)[2], T (&im)[2]) {
    const T a = re[0], b = im[0];
    re[0] = a + re[1];
    im[0] = b + im[1];
    re[1] = a - re[1];
    im[1] = b - im[1];
  }
};
template <typename T>
struct Dft<3, T> {
  DFT_FN void run(T (&re)[3], T (&im)[3]) {
    const T h = Num<T>::c(-0.5), s = Num<T>::c(Root<1, 3>::s), ms = Num<T>::c(-Root<1, 3>::s);
    const T sr = re[1] + re[2], si = im[1] + im[2], dr = re[1] - re[2], di = im[1] - im[2];
    const T mr = Num<T>::fma(sr, h, re[0]), mi = Num<T>::fma(si, h, im[0]);
    re[0] = re[0] + sr;
    im[0] = im[0] + si;
    // mr + i mi -/+ i s (dr + i di)
    re[1] = Num<T>::fma(di, s, mr);
    im[1] = Num<T>::fma(dr, ms, mi);
    re[2] = Num<T>::fma(di, ms, mr);
    im[2] = Num<T>::fma(dr, s, mi);
  }
};
template <typename T>
struct Dft<4, T> {
  DFT_FN void run(T (&re)[4], T (&im)[4]) {
    const T ar = re[0] + re[2], ai = im[0] + im[2], br = re[0] - re[2], bi = im[0] - im[2];
    const T cr = re[1] + re[3], ci = im[1] + im[3], dr = re[1] - re[3], di = im[1] - im[3];
    re[0] = ar + cr;
    im[0] = ai + ci;
    re[1] = br + di;  // b - i d
    im[1] = bi - dr;
    re[2] = ar - cr;
    im[2] = ai - ci;
    re[3] = br - di;
    im[3] = bi + dr;
  }
};
// odd primes: symmetric and antisymmetric halves
template <int R, typename T>
struct DftOdd {
  DFT_FN void run(T (&re)[R], T (&im)[R]) {
    constexpr int H = R / 2;
    T sr[H], si[H], dr[H], di[H];
#pragma unroll
    for (int j = 0; j < H; ++j) {
      sr[j] = re[1 + j] + re[R - 1 - j];
      si[j] = im[1 + j] + im[R - 1 - j];
      dr[j] = re[1 + j] - re[R - 1 - j];
      di[j] = im[1 + j] - im[R - 1 - j];
    }
    const T r0 = re[0], i0 = im[0];
#pragma unroll
    for (int j = 0; j < H; ++j) {
      re[0] = re[0] + sr[j];
      im[0] = im[0] + si[j];
    }
    out<1>(re, im, r0, i0, sr, si, dr, di);
  }
  template <int K>
  DFT_FN void out(T (&re)[R], T (&im)[R], T r0, T i0, T (&sr)[R / 2], T (&si)[R / 2],
                                             T (&dr)[R / 2], T (&di)[R / 2]) {
    constexpr int H = R / 2;
    if constexpr (K <= H) {
      T ar = r0, ai = i0;  // sum of s_j cos
      acc_cos<K, 1>(ar, ai, sr, si);
      T br = dr[0] * Num<T>::c(Root<K, R>::s), bi = di[0] * Num<T>::c(Root<K, R>::s);
      acc_sin<K, 2>(br, bi, dr, di);
      re[K] = ar + bi;  // a - i b
      im[K] = ai - br;
      re[R - K] = ar - bi;
      im[R - K] = ai + br;
      out<K + 1>(re, im, r0, i0, sr, si, dr, di);
    }
  }
  template <int K, int J>
  DFT_FN void acc_cos(T &ar, T &ai, T (&sr)[R / 2], T (&si)[R / 2]) {
    if constexpr (J <= R / 2) {
      const T w = Num<T>::c(Root<J * K, R>::c);
      ar = Num<T>::fma(sr[J - 1], w, ar);
      ai = Num<T>::fma(si[J - 1], w, ai);
      acc_cos<K, J + 1>(ar, ai, sr, si);
    }
  }
  template <int K, int J>
  DFT_FN void acc_sin(T &br, T &bi, T (&dr)[R / 2], T (&di)[R / 2]) {
    if constexpr (J <= R / 2) {
      const T w = Num<T>::c(Root<J * K, R>::s);
      br = Num<T>::fma(dr[J - 1], w, br);
      bi = Num<T>::fma(di[J - 1], w, bi);
      acc_sin<K, J + 1>(br, bi, dr, di);
    }
  }
};
template <typename T>
struct Dft<5, T> : DftOdd<5, T> {};
template <typename T>
struct Dft<7, T> : DftOdd<7, T> {};

// R = A B: input n = B a + b, output k = ka + A kb
template <int A, int B, typename T>
struct DftAB {
  static constexpr int R = A * B;
  DFT_FN void run(T (&re)[R], T (&im)[R]) {
    T xr[B][A], xi[B][A];
    rows<0>(re, im, xr, xi);
    cols<0>(re, im, xr, xi);
  }
  template <int b>
  DFT_FN void rows(T (&re)[R], T (&im)[R], T (&xr)[B][A], T (&xi)[B][A]) {
    if constexpr (b < B) {
#pragma unroll
      for (int a = 0; a < A; ++a) {
        xr[b][a] = re[B * a + b];
        xi[b][a] = im[B * a + b];
      }
      Dft<A, T>::run(xr[b], xi[b]);
      twiddle<b, 1>(xr[b], xi[b]);
      rows<b + 1>(re, im, xr, xi);
    }
  }
  template <int b, int ka>
  DFT_FN void twiddle(T (&xr)[A], T (&xi)[A]) {
    if constexpr (ka < A) {
      mul_root<b * ka, R>(xr[ka], xi[ka]);
      twiddle<b, ka + 1>(xr, xi);
    }
  }
  template <int ka>
  DFT_FN void cols(T (&re)[R], T (&im)[R], T (&xr)[B][A], T (&xi)[B][A]) {
    if constexpr (ka < A) {
      T cr[B], ci[B];
#pragma unroll
      for (int b = 0; b < B; ++b) {
        cr[b] = xr[b][ka];
        ci[b] = xi[b][ka];
      }
      Dft<B, T>::run(cr, ci);
#pragma unroll
      for (int b = 0; b < B; ++b) {
        re[ka + A * b] = cr[b];
        im[ka + A * b] = ci[b];
      }
      cols<ka + 1>(re, im, xr, xi);
    }
  }
};
template <typename T>
struct Dft<6, T> : DftAB<2, 3, T> {};
template <typename T>
struct Dft<8, T> : DftAB<2, 4, T> {};
template <typename T>
struct Dft<9, T> : DftAB<3, 3, T> {};
template <typename T>
struct Dft<10, T> : DftAB<2, 5, T> {};
template <typename T>
struct Dft<12, T> : DftAB<3, 4, T> {};
template <typename T>
struct Dft<14, T> : DftAB<2, 7, T> {};
template <typename T>
struct Dft<15, T> : DftAB<3, 5, T> {};
template <typename T>
struct Dft<16, T> : DftAB<4, 4, T> {};
template <typename T>
struct Dft<18, T> : DftAB<2, 9, T> {};
template <typename T>
struct Dft<20, T> : DftAB<4, 5, T> {};
