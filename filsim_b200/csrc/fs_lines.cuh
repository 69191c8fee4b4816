// fs_lines.cuh -- the line transforms of the periodic Stokes solve, for double (fs_lines64.cu)
// and for packed FP32 pairs (fs_lines32.cu).
//
// A line of N = R1 R2 (R3) points is transformed by a few threads, each holding one
// radix-R group in registers at a time, with one exchange through shared memory
// between two radix steps (decimation in frequency):
//   n = t + M j (M = N / R1): R1-point transforms over j, times w_N^(t k1);
//   then the M-point transforms over t for each k1 the same way,
// so a thread ends with X[k1 + R1 (k2 + R2 k3)] over its last digit in natural order. Everything that moves through
// memory is a 16-byte value: one complex double, or the same complex number of two
// neighbouring FP32 lines as (re0, re1, im0, im1), so that FP32 butterflies are packed
// f32x2 instructions and both precisions share the code and the access patterns.
#pragma once
#include "fs_internal.cuh"
#include <type_traits>
#include "fs_dft.cuh"

typedef ulonglong2 V16;  // one transform value in memory: (re, im) of T

template <typename T>
struct Io;
template <>
struct Io<double> {
  static __device__ __forceinline__ void get(const V16 &v, double &re, double &im) {
    re = __longlong_as_double((long long)v.x);
    im = __longlong_as_double((long long)v.y);
  }
  static __device__ __forceinline__ V16 put(double re, double im) {
    return make_ulonglong2((unsigned long long)__double_as_longlong(re), (unsigned long long)__double_as_longlong(im));
  }
};
template <>
struct Io<F2> {
  static __device__ __forceinline__ void get(const V16 &v, F2 &re, F2 &im) {
    re.v = v.x;
    im.v = v.y;
  }
  static __device__ __forceinline__ V16 put(F2 re, F2 im) { return make_ulonglong2(re.v, im.v); }
};

// 16-byte copy from global to shared memory without a register or an L1 line: the loads
// of strided lines stay in flight whatever the split of the SM's memory leaves to L1
__device__ __forceinline__ void copy16(V16 *smem, const V16 *gmem) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((unsigned)__cvta_generic_to_shared(smem)), "l"(gmem)
               : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// (re, im) times the table value w = (cos, -sin) (FP32: each twice)
template <typename T>
__device__ __forceinline__ void mul_w(T &re, T &im, const V16 &w) {
  T wr, wi;
  Io<T>::get(w, wr, wi);
  const T a = Num<T>::fma(re, wr, -(im * wi));  // one rounding less than a difference of products
  im = Num<T>::fma(re, wi, im * wr);
  re = a;
}
template <typename T>
__device__ __forceinline__ void mul_tw(T &re, T &im, const V16 *__restrict__ w) {
  mul_w<T>(re, im, __ldg(w));
}

// Radices of a line. Y and z lines: at most 16 points in registers (18 and 20 for z lines of 432
// and 400 points, which like all z lines take two steps), the fewest exchanges, and as even a
// split as the factors allow (threads per line = N / smallest radix). X lines end with three
// components per thread: at most 8 points each there.
template <int N>
struct Radices;
template <int N>
struct RadicesX;
#define FS_RADICES(S, N, A, B, C)                 \
  template <>                                     \
  struct S<N> {                                   \
    static constexpr int R1 = A, R2 = B, R3 = C; \
  };
FS_RADICES(Radices, 16, 4, 4, 1)
FS_RADICES(Radices, 24, 4, 6, 1)
FS_RADICES(Radices, 32, 4, 8, 1)
FS_RADICES(Radices, 40, 5, 8, 1)
FS_RADICES(Radices, 48, 6, 8, 1)
FS_RADICES(Radices, 56, 7, 8, 1)
FS_RADICES(Radices, 64, 8, 8, 1)
FS_RADICES(Radices, 72, 8, 9, 1)
FS_RADICES(Radices, 80, 8, 10, 1)
FS_RADICES(Radices, 96, 8, 12, 1)
FS_RADICES(Radices, 112, 8, 14, 1)
FS_RADICES(Radices, 120, 10, 12, 1)
FS_RADICES(Radices, 128, 8, 16, 1)
FS_RADICES(Radices, 144, 12, 12, 1)
FS_RADICES(Radices, 160, 10, 16, 1)
FS_RADICES(Radices, 168, 12, 14, 1)
FS_RADICES(Radices, 192, 12, 16, 1)
FS_RADICES(Radices, 200, 10, 20, 1)
FS_RADICES(Radices, 216, 12, 18, 1)
FS_RADICES(Radices, 224, 14, 16, 1)
FS_RADICES(Radices, 240, 15, 16, 1)
FS_RADICES(Radices, 256, 16, 16, 1)
FS_RADICES(Radices, 288, 8, 6, 6)
FS_RADICES(Radices, 320, 8, 8, 5)
FS_RADICES(Radices, 336, 8, 6, 7)
FS_RADICES(Radices, 384, 8, 8, 6)
FS_RADICES(Radices, 400, 8, 10, 5)
FS_RADICES(Radices, 432, 8, 9, 6)
FS_RADICES(Radices, 448, 8, 8, 7)
FS_RADICES(Radices, 480, 8, 10, 6)
FS_RADICES(Radices, 512, 8, 8, 8)
FS_RADICES(RadicesX, 32, 4, 8, 1)
FS_RADICES(RadicesX, 48, 6, 8, 1)
FS_RADICES(RadicesX, 64, 8, 8, 1)
FS_RADICES(RadicesX, 80, 4, 4, 5)
FS_RADICES(RadicesX, 96, 4, 4, 6)
FS_RADICES(RadicesX, 112, 4, 4, 7)
FS_RADICES(RadicesX, 128, 4, 4, 8)
FS_RADICES(RadicesX, 144, 4, 6, 6)
FS_RADICES(RadicesX, 160, 8, 4, 5)
FS_RADICES(RadicesX, 192, 8, 4, 6)
FS_RADICES(RadicesX, 224, 8, 4, 7)
FS_RADICES(RadicesX, 240, 8, 6, 5)
FS_RADICES(RadicesX, 256, 8, 8, 4)
FS_RADICES(RadicesX, 288, 8, 6, 6)
FS_RADICES(RadicesX, 320, 8, 8, 5)
FS_RADICES(RadicesX, 336, 8, 6, 7)
FS_RADICES(RadicesX, 384, 8, 8, 6)
FS_RADICES(RadicesX, 400, 8, 10, 5)
FS_RADICES(RadicesX, 432, 8, 9, 6)
FS_RADICES(RadicesX, 448, 8, 8, 7)
FS_RADICES(RadicesX, 480, 8, 10, 6)
FS_RADICES(RadicesX, 512, 8, 8, 8)
#undef FS_RADICES

template <int N_, typename R>
struct LineOf {
  static constexpr int N = N_, R1 = R::R1, R2 = R::R2, R3 = R::R3;
  static constexpr int M = N / R1;                                  // threads of the first step
  static constexpr int T2 = R3 == 1 ? R1 : R1 * R3;                 // of the second
  static constexpr int RL = R3 == 1 ? R2 : R3;                      // radix of the last step
  static constexpr int TL = N / RL;                                 // threads of the last step
  static constexpr int TH = M > T2 ? (M > TL ? M : TL) : (T2 > TL ? T2 : TL);
  static constexpr int TW1 = (R1 - 1) * M;                          // first-step table [k1 - 1][t]
  static constexpr int TW2 = R3 == 1 ? 0 : (R2 - 1) * R3;           // second-step table [k2 - 1][t']
  static constexpr int TW = TW1 + TW2;
  static __host__ __device__ constexpr int last_index(int t, int j) { return t + TL * j; }  // index of register j
};
template <int N>
using Line = LineOf<N, Radices<N>>;
template <int N>
using LineX = LineOf<N, RadicesX<N>>;

// The steps of one line. Its exchange buffer holds value p at S[p CS]; between two steps
// every thread of the CTA passes a barrier. A step with fewer groups than threads leaves
// the rest idle. MS: distance of the k1 blocks in the buffer, M, or M + 1 where a row of
// CS values is half a row of banks (the last step reads across the blocks). Forward: line_first (a[j] = x[t + M j] in), line_mid if R3 > 1, line_last
// (z[j] = X[t + TL j] out). Backwards (k_lines_x_project) the same steps in reverse, with
// re and im exchanged for the inverse and each twiddle before its step. Mid and last steps
// touch only positions of their own group, so they may write where they read.
template <typename L, int CS, int MS, typename T>
__device__ __forceinline__ void line_first(T (&ar)[L::R1], T (&ai)[L::R1], V16 *S, int t, const V16 *__restrict__ tw) {
  Dft<L::R1, T>::run(ar, ai);
#pragma unroll
  for (int k = 0; k < L::R1; ++k) {
    if (k) mul_tw<T>(ar[k], ai[k], tw + (k - 1) * L::M + t);
    S[(k * MS + t) * CS] = Io<T>::put(ar[k], ai[k]);
  }
}
// t < T2: group (k1, u) = (t / R3, t % R3) of NC lines whose buffers are NS apart
template <typename L, int CS, int MS, int NC, int NS, bool ADJ, typename T>
__device__ __forceinline__ void line_mid(V16 *S, int t, const V16 *__restrict__ tw) {
  const int u = t % L::R3;
  const V16 *__restrict__ tw2 = tw + L::TW1 + u;
  V16 *P0 = S + ((t / L::R3) * MS + u) * CS;
  V16 w[L::R2];
  if constexpr (NC > 1) {  // read once for all lines
#pragma unroll
    for (int k = 1; k < L::R2; ++k) w[k] = __ldg(tw2 + (k - 1) * L::R3);
  }
#pragma unroll 1
  for (int c = 0; c < NC; ++c) {
    V16 *P = P0 + c * NS;
    T br[L::R2], bi[L::R2];
#pragma unroll
    for (int k = 0; k < L::R2; ++k) {
      ADJ ? Io<T>::get(P[k * L::R3 * CS], bi[k], br[k]) : Io<T>::get(P[k * L::R3 * CS], br[k], bi[k]);
      if (ADJ && k) mul_w<T>(br[k], bi[k], NC > 1 ? w[k] : __ldg(tw2 + (k - 1) * L::R3));
    }
    Dft<L::R2, T>::run(br, bi);
#pragma unroll
    for (int k = 0; k < L::R2; ++k) {
      if (!ADJ && k) mul_w<T>(br[k], bi[k], NC > 1 ? w[k] : __ldg(tw2 + (k - 1) * L::R3));
      P[k * L::R3 * CS] = ADJ ? Io<T>::put(bi[k], br[k]) : Io<T>::put(br[k], bi[k]);
    }
  }
}
// t < TL: group k1 + R1 k2 = t, values k1 MS + k2 R3 + j (R3 > 1) or k1 MS + j
template <typename L, int MS>
__device__ __forceinline__ int last_base(int t) {
  return (t % L::R1) * MS + (t / L::R1) * L::R3;
}
template <typename L, int CS, int MS, typename T>
__device__ __forceinline__ void line_last(T (&zr)[L::RL], T (&zi)[L::RL], const V16 *S, int t) {
  const V16 *P = S + last_base<L, MS>(t) * CS;
#pragma unroll
  for (int j = 0; j < L::RL; ++j) Io<T>::get(P[j * CS], zr[j], zi[j]);
  Dft<L::RL, T>::run(zr, zi);
}

// ---- y lines, in place --------------------------------------------------------------
// Bound by HBM and the L1 data path together (512 points: 8.75 16-byte L1 accesses a
// value). 512^3, FP64 1.24 ms a pass (5.2 TB/s, 0.80 of the copy bandwidth), FP32 0.68 ms
// (0.73); 256^3 0.158 and 0.085 ms (0.79, 0.74). cuFFT's strided passes: 1.32 ms and 0.134 ms.
// The half spectrum lies as [c][x][y][v]: nv values along z (FP64: kz = v; FP32: kz =
// 2 v, 2 v + 1), rows of nvp. A CTA takes COLS neighbouring columns (o, v), o = (c, x),
// numbered o nv + v, so no column is padding; its threads hold COLS consecutive
// 16-byte values of each row: 128-byte accesses at COLS = 8.
template <int N, typename T>
struct YShape {
  // long FP32 lines: half rows in CTAs of half the size (512 points: 0.73 -> 0.68 ms at 512^3;
  // FP64, whose rows carry half the columns, 1.24 -> 1.33)
  static constexpr int COLS = 8 * Line<N>::TH <= 256 || Num<T>::IS_DOUBLE ? 8 : 4;
  static constexpr int THREADS = COLS * Line<N>::TH;
  static constexpr int MS = COLS < 8 ? Line<N>::M | 1 : Line<N>::M;
  static constexpr size_t SMEM = sizeof(V16) * (size_t)COLS * Line<N>::R1 * MS;
  // at 64 registers from 256 threads on, at 128 below
  static constexpr int CTAS = THREADS > 512 ? 1 : THREADS >= 256 ? 1024 / THREADS : 512 / THREADS;
};
template <int N, typename T, bool INV>
__global__ void __launch_bounds__(YShape<N, T>::THREADS, YShape<N, T>::CTAS)
    k_lines_y(V16 *__restrict__ A, int ncol, int nv, int nvp, const V16 *__restrict__ tw) {
  FS_AFTER_PREVIOUS();
  typedef Line<N> L;
  constexpr int COLS = YShape<N, T>::COLS, MS = YShape<N, T>::MS;
  extern __shared__ V16 line_smem[];
  const int c = threadIdx.x % COLS, t = threadIdx.x / COLS;
  // columns past the last one repeat it and store nothing
  const bool on = blockIdx.x * COLS + c < ncol;
  const int e = on ? blockIdx.x * COLS + c : ncol - 1, o = e / nv, v = e - o * nv;
  V16 *base = A + (size_t)o * N * nvp + v;
  V16 *S = line_smem + c;
  if (t < L::M) {
    T ar[L::R1], ai[L::R1];
#pragma unroll
    for (int j = 0; j < L::R1; ++j)
      copy16(S + (j * MS + t) * COLS, base + (size_t)(t + L::M * j) * nvp);
    copy_commit();
    copy_wait<0>();  // a thread reads what it copied itself
#pragma unroll
    for (int j = 0; j < L::R1; ++j) {
      const V16 x = S[(j * MS + t) * COLS];
      INV ? Io<T>::get(x, ai[j], ar[j]) : Io<T>::get(x, ar[j], ai[j]);
    }
    line_first<L, COLS, MS, T>(ar, ai, S, t, tw);
  }
  __syncthreads();
  if constexpr (L::R3 > 1) {
    if (t < L::T2) line_mid<L, COLS, MS, 1, 0, false, T>(S, t, tw);
    __syncthreads();
  }
  if (t < L::TL) {
    T zr[L::RL], zi[L::RL];
    line_last<L, COLS, MS, T>(zr, zi, S, t);
    if (on) {
#pragma unroll
      for (int j = 0; j < L::RL; ++j)
        base[(size_t)L::last_index(t, j) * nvp] = INV ? Io<T>::put(zi[j], zr[j]) : Io<T>::put(zr[j], zi[j]);
    }
  }
}

// ---- x lines: forward, Stokes projection, inverse, in place ---------------------------
// A thread holds the same radix group of the three components, so the projection
// (flow_solve, FCMfunctions.cpp:668-722) needs no exchange: norm = 1 / (qx^2 + qy^2 +
// 1e-18 + qz^2), u = norm (f - q (q . f) norm) / (Nx Ny Nz), the k = 0 mode zeroed.
// Bound by the L1 data path (12 accesses a value) at the two CTAs of 256 threads that three
// components of 512 points leave room for: FP64 2.2 ms at 512^3, where two cuFFT passes and
// the projection took 3.8; 0.24 ms at 256^3 (0.41). Measured slower: one thread group per
// component with an exchange of q . f (3.96 ms), 2 or 8 columns per CTA (2.8, 2.1 to
// 0.30 ms), loads through registers (their L1 lines do not fit beside the buffers: 2.86 ms).
template <int N>
struct XShape {
  static constexpr int TH = LineX<N>::TH;
  static constexpr int COLS = TH <= 8 ? 16 : TH <= 40 ? 8 : 4;
  static constexpr int THREADS = COLS * TH;
  static constexpr int MS = COLS < 8 ? LineX<N>::M | 1 : LineX<N>::M;
  static constexpr int NS = COLS * LineX<N>::R1 * MS;  // one component's exchange buffer
  static constexpr size_t SMEM = sizeof(V16) * 3 * NS;
  static constexpr int CTAS = THREADS > 256 ? 2 : 512 / THREADS;  // at most 128 registers, 96 above 256 threads
};
template <typename T>
struct Wave;  // kz of one value and the reciprocal of the squared wavenumber
template <>
struct Wave<double> {
  static __device__ __forceinline__ double kz(int v, double ff) { return (double)v * ff; }
  static __device__ __forceinline__ double inv(double s) { return 1.0 / s; }
  static __device__ __forceinline__ void zero(int v, double &s) {
    if (v == 0) s = 0.0;
  }
};
template <>
struct Wave<F2> {
  static __device__ __forceinline__ F2 kz(int v, double ff) {
    return {f2_pack((float)(2 * v) * (float)ff, (float)(2 * v + 1) * (float)ff)};
  }
  static __device__ __forceinline__ F2 inv(F2 s) {
    const float2 f = f2_unpack(s.v);
    return {f2_pack(__frcp_rn(f.x), __frcp_rn(f.y))};
  }
  static __device__ __forceinline__ void zero(int v, F2 &s) {  // kz = 0 is the first of its pair
    if (v == 0) s.v = f2_pack(0.f, f2_unpack(s.v).y);
  }
};

struct XArgs {
  int ncol, ny, nv, nvp;
  size_t rstride, cstride;  // between x planes and between components
  double ffx, ffy, ffz;
  double inv_total, inv_total_lo;  // 1 / (Nx Ny Nz) to this precision, and what rounding it left out
};
template <int N, typename T>
__global__ void __launch_bounds__(XShape<N>::THREADS, XShape<N>::CTAS)
    k_lines_x_project(V16 *__restrict__ A, XArgs g, const V16 *__restrict__ tw) {
  FS_AFTER_PREVIOUS();
  typedef LineX<N> L;
  constexpr int COLS = XShape<N>::COLS, MS = XShape<N>::MS, NS = XShape<N>::NS;
  extern __shared__ V16 line_smem[];
  const int c = threadIdx.x % COLS, t = threadIdx.x / COLS;
  // columns past the last one repeat it and store nothing
  const bool on = blockIdx.x * COLS + c < g.ncol;
  const int e = on ? blockIdx.x * COLS + c : g.ncol - 1, y = e / g.nv, v = e - y * g.nv;
  V16 *base = A + (size_t)y * g.nvp + v;
  V16 *S = line_smem + c;
  if (t < L::M) {
#pragma unroll
    for (int a = 0; a < 3; ++a) {
#pragma unroll
      for (int j = 0; j < L::R1; ++j)
        copy16(S + a * NS + (j * MS + t) * COLS, base + a * g.cstride + (size_t)(t + L::M * j) * g.rstride);
      copy_commit();
    }
    V16 w[L::R1];
#pragma unroll
    for (int k = 1; k < L::R1; ++k) w[k] = __ldg(tw + (k - 1) * L::M + t);
#pragma unroll 1
    for (int a = 0; a < 3; ++a) {
      if (a == 0) copy_wait<2>();  // a thread reads what it copied itself
      else if (a == 1) copy_wait<1>();
      else copy_wait<0>();
      T ar[L::R1], ai[L::R1];
#pragma unroll
      for (int j = 0; j < L::R1; ++j) Io<T>::get(S[a * NS + (j * MS + t) * COLS], ar[j], ai[j]);
      Dft<L::R1, T>::run(ar, ai);
#pragma unroll
      for (int k = 0; k < L::R1; ++k) {
        if (k) mul_w<T>(ar[k], ai[k], w[k]);
        S[a * NS + (k * MS + t) * COLS] = Io<T>::put(ar[k], ai[k]);
      }
    }
  }
  __syncthreads();
  if constexpr (L::R3 > 1) {
    if (t < L::T2) line_mid<L, COLS, MS, 3, NS, false, T>(S, t, tw);
    __syncthreads();
  }
  if (t < L::TL) {
    T zr[3][L::RL], zi[3][L::RL];
#pragma unroll
    for (int a = 0; a < 3; ++a) line_last<L, COLS, MS, T>(zr[a], zi[a], S + a * NS, t);
    const T q2 = Num<T>::c((double)((y <= g.ny / 2) ? y : y - g.ny) * g.ffy), q3 = Wave<T>::kz(v, g.ffz);
#pragma unroll
    for (int j = 0; j < L::RL; ++j) {
      const int k = L::last_index(t, j);
      const T q1 = Num<T>::c((double)((k <= N / 2) ? k : k - N) * g.ffx);
      const T norm = Wave<T>::inv(Num<T>::fma(q3, q3, Num<T>::fma(q2, q2, q1 * q1) + Num<T>::c(1e-18)));
      // minus q . f / q^2, so that f - q (q . f) / q^2 is one rounding
      const T kfr = -(Num<T>::fma(q3, zr[2][j], Num<T>::fma(q2, zr[1][j], q1 * zr[0][j])) * norm);
      const T kfi = -(Num<T>::fma(q3, zi[2][j], Num<T>::fma(q2, zi[1][j], q1 * zi[0][j])) * norm);
      T sc = Num<T>::fma(norm, Num<T>::c(g.inv_total), norm * Num<T>::c(g.inv_total_lo));
      if (k == 0 && y == 0) Wave<T>::zero(v, sc);
      zr[0][j] = sc * Num<T>::fma(q1, kfr, zr[0][j]);
      zi[0][j] = sc * Num<T>::fma(q1, kfi, zi[0][j]);
      zr[1][j] = sc * Num<T>::fma(q2, kfr, zr[1][j]);
      zi[1][j] = sc * Num<T>::fma(q2, kfi, zi[1][j]);
      zr[2][j] = sc * Num<T>::fma(q3, kfr, zr[2][j]);
      zi[2][j] = sc * Num<T>::fma(q3, kfi, zi[2][j]);
    }
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      Dft<L::RL, T>::run(zi[a], zr[a]);
      V16 *P = S + a * NS + last_base<L, MS>(t) * COLS;
#pragma unroll
      for (int j = 0; j < L::RL; ++j) P[j * COLS] = Io<T>::put(zr[a][j], zi[a][j]);
    }
  }
  __syncthreads();
  if constexpr (L::R3 > 1) {
    if (t < L::T2) line_mid<L, COLS, MS, 3, NS, true, T>(S, t, tw);
    __syncthreads();
  }
  if (t < L::M) {  // the inverse: re and im exchanged
    V16 w[L::R1];
#pragma unroll
    for (int k = 1; k < L::R1; ++k) w[k] = __ldg(tw + (k - 1) * L::M + t);
#pragma unroll 1
    for (int a = 0; a < 3; ++a) {
      T ar[L::R1], ai[L::R1];
#pragma unroll
      for (int k = 0; k < L::R1; ++k) {
        Io<T>::get(S[a * NS + (k * MS + t) * COLS], ai[k], ar[k]);
        if (k) mul_w<T>(ar[k], ai[k], w[k]);
      }
      Dft<L::R1, T>::run(ar, ai);
      if (on) {
#pragma unroll
        for (int j = 0; j < L::R1; ++j)
          base[a * g.cstride + (size_t)(t + L::M * j) * g.rstride] = Io<T>::put(ai[j], ar[j]);
      }
    }
  }
}

// ---- z lines: real, 2 M points, as M complex points ------------------------------------
// Forward: Z the M-point transform of x[2n] + i x[2n+1]; with w = exp(-2 pi i k / 2M),
// X[k] = (Z_k + conj Z_(M-k)) / 2 - (i w / 2) (Z_k - conj Z_(M-k)), k = 0 .. M (Z_M = Z_0).
// Inverse: the imaginary parts of X_0 and X_M dropped, Z_k = (X_k + conj X_(M-k)) +
// i conj(w) (X_k - conj X_(M-k)), its unnormalised inverse gives x[2n] + i x[2n+1].
// A unit is one line (FP64) or two neighbouring lines (FP32); LU units per CTA. 512^3:
// FP64 1.17 and 1.20 ms (0.85, 0.82 of the copy bandwidth; cuFFT 1.53, 1.63), FP32 0.68, 0.69.
template <int M>
struct ZShape {
  typedef Line<M> L;
  static constexpr int LU = 128 / L::TH > 1 ? 128 / L::TH : 1;
  static constexpr int THREADS = LU * L::TH;
  // exchange rows padded to an odd length (conflict-free strided reads); natural order needs M + 2
  static constexpr int PM = L::M | 1;
  static constexpr int BUF = L::R1 * PM > M + 2 ? L::R1 * PM : M + 2;
  static constexpr int STRIDE = BUF | 1;  // values per unit
  static constexpr size_t SMEM = sizeof(V16) * (size_t)LU * STRIDE;
};
// the transform of one z unit: two steps through the padded exchange buffer
template <int M, typename T>
__device__ __forceinline__ void z_dif(T (&ar)[Line<M>::R1], T (&ai)[Line<M>::R1], T (&zr)[Line<M>::RL],
                                      T (&zi)[Line<M>::RL], V16 *S, int t, const V16 *__restrict__ tw) {
  typedef Line<M> L;
  static_assert(L::R3 == 1, "z lines take two steps");
  constexpr int PM = ZShape<M>::PM;
  if (t < L::M) {
    Dft<L::R1, T>::run(ar, ai);
#pragma unroll
    for (int k = 0; k < L::R1; ++k) {
      if (k) mul_tw<T>(ar[k], ai[k], tw + (k - 1) * L::M + t);
      S[k * PM + t] = Io<T>::put(ar[k], ai[k]);
    }
  }
  __syncthreads();
  if (t < L::TL) {
#pragma unroll
    for (int j = 0; j < L::RL; ++j) Io<T>::get(S[t * PM + j], zr[j], zi[j]);
    Dft<L::RL, T>::run(zr, zi);
  }
}

// X_k of a unit from Z in natural order
template <int M, typename T>
__device__ __forceinline__ void untangle(const V16 *S, int k, const V16 *__restrict__ tu, T &xr, T &xi) {
  T zr, zi, mr, mi;
  Io<T>::get(S[k == M ? 0 : k], zr, zi);
  Io<T>::get(S[k == 0 ? 0 : M - k], mr, mi);
  const T h = Num<T>::c(0.5);
  const T er = (zr + mr) * h, ei = (zi - mi) * h;  // (Z_k + conj Z_(M-k)) / 2
  T dr = (zi + mi) * h, di = (mr - zr) * h;        // -i (Z_k - conj Z_(M-k)) / 2
  mul_tw<T>(dr, di, tu + k);
  xr = er + dr;
  xi = ei + di;
}

template <int M, typename T>
__global__ void __launch_bounds__(ZShape<M>::THREADS) k_lines_z_fwd(const void *__restrict__ f_, V16 *__restrict__ A,
                                                                    int nunit, int nvp, const V16 *__restrict__ tw) {
  FS_AFTER_PREVIOUS();
  typedef Line<M> L;
  typedef ZShape<M> Z;
  constexpr bool F64 = Num<T>::IS_DOUBLE;
  extern __shared__ V16 line_smem[];
  const int l = threadIdx.x / L::TH, t = threadIdx.x - l * L::TH;
  const int u0 = blockIdx.x * Z::LU;
  const bool on = u0 + l < nunit;
  V16 *S = line_smem + l * Z::STRIDE;
  T ar[L::R1], ai[L::R1], zr[L::RL], zi[L::RL];
  if (t < L::M && on) {
    if constexpr (F64) {
      const double2 *p = (const double2 *)f_ + (size_t)(u0 + l) * M + t;
#pragma unroll
      for (int j = 0; j < L::R1; ++j) {
        const double2 x = __ldg(p + L::M * j);
        ar[j] = x.x;
        ai[j] = x.y;
      }
    } else {
      const float2 *p = (const float2 *)f_ + (size_t)(u0 + l) * 2 * M + t;
      float2 a[L::R1], b[L::R1];
#pragma unroll
      for (int j = 0; j < L::R1; ++j) {
        a[j] = __ldg(p + L::M * j);
        b[j] = __ldg(p + M + L::M * j);
      }
#pragma unroll
      for (int j = 0; j < L::R1; ++j) {
        ar[j].v = f2_pack(a[j].x, b[j].x);
        ai[j].v = f2_pack(a[j].y, b[j].y);
      }
    }
  }
  z_dif<M, T>(ar, ai, zr, zi, S, t, tw);
  __syncthreads();  // the exchange values are no longer read
  if (t < L::TL) {
#pragma unroll
    for (int j = 0; j < L::RL; ++j) S[L::last_index(t, j)] = Io<T>::put(zr[j], zi[j]);
  }
  __syncthreads();
  const V16 *tu = tw + L::TW;
  if constexpr (F64) {
    for (int i = threadIdx.x; i < Z::LU * (M + 1); i += Z::THREADS) {
      const int r = i / (M + 1), k = i - r * (M + 1);
      if (u0 + r >= nunit) continue;
      T xr, xi;
      untangle<M, T>(line_smem + r * Z::STRIDE, k, tu, xr, xi);
      A[(size_t)(u0 + r) * nvp + k] = Io<T>::put(xr, xi);
    }
  } else {
    constexpr int NV = M / 2 + 1;  // pairs kz = 2 v, 2 v + 1; the last pair's second value is padding
    for (int i = threadIdx.x; i < Z::LU * NV; i += Z::THREADS) {
      const int r = i / NV, v = i - r * NV;
      if (u0 + r >= nunit) continue;
      T r0, i0, r1, i1;
      untangle<M, T>(line_smem + r * Z::STRIDE, 2 * v, tu, r0, i0);
      if (2 * v < M)
        untangle<M, T>(line_smem + r * Z::STRIDE, 2 * v + 1, tu, r1, i1);
      else
        r1.v = i1.v = 0ull;
      const float2 a0 = f2_unpack(r0.v), b0 = f2_unpack(i0.v), a1 = f2_unpack(r1.v), b1 = f2_unpack(i1.v);
      V16 *out = A + (size_t)2 * (u0 + r) * nvp + v;
      out[0] = make_ulonglong2(f2_pack(a0.x, a1.x), f2_pack(b0.x, b1.x));
      out[nvp] = make_ulonglong2(f2_pack(a0.y, a1.y), f2_pack(b0.y, b1.y));
    }
  }
}

template <int M, typename T>
__global__ void __launch_bounds__(ZShape<M>::THREADS) k_lines_z_inv(const V16 *__restrict__ A, void *__restrict__ u_,
                                                                    int nunit, int nvp, const V16 *__restrict__ tw) {
  FS_AFTER_PREVIOUS();
  typedef Line<M> L;
  typedef ZShape<M> Z;
  constexpr bool F64 = Num<T>::IS_DOUBLE;
  extern __shared__ V16 line_smem[];
  const int l = threadIdx.x / L::TH, t = threadIdx.x - l * L::TH;
  const int u0 = blockIdx.x * Z::LU;
  const bool on = u0 + l < nunit;
  V16 *S = line_smem + l * Z::STRIDE;
  // the spectrum rows into shared memory, natural order, all of a thread's loads in flight
  constexpr int NV = F64 ? M + 1 : M / 2 + 1, ITS = (Z::LU * NV + Z::THREADS - 1) / Z::THREADS;
  {
    constexpr int ROWS = F64 ? 1 : 2;
    V16 x[ITS][ROWS];
#pragma unroll
    for (int n = 0; n < ITS; ++n) {
      const int i = threadIdx.x + n * Z::THREADS, r = i / NV, v = i - r * NV;
      if (r < Z::LU && u0 + r < nunit) {
#pragma unroll
        for (int h = 0; h < ROWS; ++h) x[n][h] = __ldg(A + ((size_t)ROWS * (u0 + r) + h) * nvp + v);
      }
    }
#pragma unroll
    for (int n = 0; n < ITS; ++n) {
      const int i = threadIdx.x + n * Z::THREADS, r = i / NV, v = i - r * NV;
      if (r < Z::LU) {
        V16 *o = line_smem + r * Z::STRIDE;
        if constexpr (F64) {
          if (v == 0 || v == M) x[n][0].y = 0ull;
          o[v] = x[n][0];
        } else {
          float2 ar = f2_unpack(x[n][0].x), ai = f2_unpack(x[n][0].y), br = f2_unpack(x[n][1].x),
                 bi = f2_unpack(x[n][1].y);
          if (v == 0 || 2 * v == M) ai.x = bi.x = 0.f;
          o[2 * v] = make_ulonglong2(f2_pack(ar.x, br.x), f2_pack(ai.x, bi.x));
          if (2 * v < M) o[2 * v + 1] = make_ulonglong2(f2_pack(ar.y, br.y), f2_pack(ai.y, bi.y));
        }
      }
    }
  }
  __syncthreads();
  T ar[L::R1], ai[L::R1], zr[L::RL], zi[L::RL];
  if (t < L::M) {
    const V16 *tu = tw + L::TW;
#pragma unroll
    for (int j = 0; j < L::R1; ++j) {
      const int k = t + L::M * j;
      T xr, xi, mr, mi;
      Io<T>::get(S[k], xr, xi);
      Io<T>::get(S[M - k], mr, mi);
      const T er = xr + mr, ei = xi - mi;  // X_k + conj X_(M-k)
      T dr = xr - mr, di = xi + mi;        // X_k - conj X_(M-k), times conj(w): exchanged parts times w
      mul_tw<T>(di, dr, tu + k);
      ar[j] = er - di;  // + i times it
      ai[j] = ei + dr;
    }
  }
  __syncthreads();  // X is no longer read
  z_dif<M, T>(ai, ar, zi, zr, S, t, tw);
  if (t < L::TL && on) {
    if constexpr (F64) {
      double2 *p = (double2 *)u_ + (size_t)(u0 + l) * M;
#pragma unroll
      for (int j = 0; j < L::RL; ++j) p[L::last_index(t, j)] = make_double2(zr[j], zi[j]);
    } else {
      float2 *p = (float2 *)u_ + (size_t)(u0 + l) * 2 * M;
#pragma unroll
      for (int j = 0; j < L::RL; ++j) {
        const float2 r = f2_unpack(zr[j].v), i = f2_unpack(zi[j].v);
        p[L::last_index(t, j)] = make_float2(r.x, i.x);
        p[M + L::last_index(t, j)] = make_float2(r.y, i.y);
      }
    }
  }
}

// ---- host side ----------------------------------------------------------------------------
// values along z per row, and the row length (even: rows start on 32-byte sectors)
template <typename T>
int lines_nv(int nz) { return Num<T>::IS_DOUBLE ? nz / 2 + 1 : nz / 4 + 1; }
template <typename T>
int lines_nvp(int nz) { return (lines_nv<T>(nz) + 1) & ~1; }

#define FS_LINE_LENGTHS(X)                                                                                   \
  X(32) X(48) X(64) X(80) X(96) X(112) X(128) X(144) X(160) X(192) X(224) X(240) X(256) X(288) X(320) X(336) \
  X(384) X(400) X(432) X(448) X(480) X(512)
// the list is line_length's rule: each length that it takes, and no other
#define FS_LINE_COUNT(N) +(line_length(N) ? 1 : 100)
static_assert(FS_LINE_LENGTHS(FS_LINE_COUNT) == line_lengths(), "lengths of the line transforms");
#undef FS_LINE_COUNT
#define FS_LINE_CASE(N) \
  case N: return f(std::integral_constant<int, N>());
// f with the length n as a constant
template <typename F>
fs_status with_length(int n, F f) {
  switch (n) { FS_LINE_LENGTHS(FS_LINE_CASE) }
  return FS_ERR_INVALID_ARG;
}
#undef FS_LINE_CASE
#define FS_LINES_SWITCH(n, fn, ...) \
  FS_TRY(with_length(n, [&](auto len) { return fn<decltype(len)::value, T>(__VA_ARGS__); }))

// table values of one line: first- and second-step twiddles, then (z lines) w^k, k <= N
struct TwRoot {
  int j, n;  // exp(-2 pi i j / n)
};
template <typename L>
void line_roots(std::vector<TwRoot> &out) {
  for (int k = 1; k < L::R1; ++k)
    for (int t = 0; t < L::M; ++t) out.push_back({k * t % L::N, L::N});
  if (L::R3 > 1)
    for (int k = 1; k < L::R2; ++k)
      for (int u = 0; u < L::R3; ++u) out.push_back({k * u % L::M, L::M});
}
template <int N, typename T>
fs_status x_roots(std::vector<TwRoot> &out) {
  line_roots<LineX<N>>(out);
  return FS_OK;
}
template <int N, typename T>
fs_status y_roots(std::vector<TwRoot> &out) {
  line_roots<Line<N>>(out);
  return FS_OK;
}
template <int N, typename T>
fs_status z_roots(std::vector<TwRoot> &out) {
  line_roots<Line<N / 2>>(out);
  for (int k = 0; k <= N / 2; ++k) out.push_back({k, N});
  return FS_OK;
}

// the attributes of the kernels a grid runs
template <int N, typename T>
fs_status x_attrs() {
  FS_CUDA(cudaFuncSetAttribute(k_lines_x_project<N, T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)XShape<N>::SMEM));
  // two 512-point CTAs need 202 KB together, more than the split the driver picks by itself
  FS_CUDA(cudaFuncSetAttribute(k_lines_x_project<N, T>, cudaFuncAttributePreferredSharedMemoryCarveout,
                               cudaSharedmemCarveoutMaxShared));
  return FS_OK;
}
template <int N, typename T>
fs_status y_attrs() {
  const int smem = (int)YShape<N, T>::SMEM;
  FS_CUDA(cudaFuncSetAttribute(k_lines_y<N, T, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  FS_CUDA(cudaFuncSetAttribute(k_lines_y<N, T, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
  return FS_OK;
}
template <int N, typename T>
fs_status z_attrs() {
  FS_CUDA(cudaFuncSetAttribute(k_lines_z_fwd<N / 2, T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)ZShape<N / 2>::SMEM));
  FS_CUDA(cudaFuncSetAttribute(k_lines_z_inv<N / 2, T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)ZShape<N / 2>::SMEM));
  return FS_OK;
}

template <int N, typename T>
fs_status z_fwd(fs_ctx *c, V16 *A, const V16 *tw) {
  const int nunit = 3 * c->nx * c->ny / (Num<T>::IS_DOUBLE ? 1 : 2);
  typedef ZShape<N / 2> Z;
  fs_launch(k_lines_z_fwd<N / 2, T>, fs_blocks(nunit, Z::LU), Z::THREADS, Z::SMEM, c->stream, c->grid_real, A, nunit,
            lines_nvp<T>(N), tw);
  FS_LAUNCH_CHECK();
  return FS_OK;
}
template <int N, typename T>
fs_status z_inv(fs_ctx *c, const V16 *A, const V16 *tw) {
  const int nunit = 3 * c->nx * c->ny / (Num<T>::IS_DOUBLE ? 1 : 2);
  typedef ZShape<N / 2> Z;
  fs_launch(k_lines_z_inv<N / 2, T>, fs_blocks(nunit, Z::LU), Z::THREADS, Z::SMEM, c->stream, A, c->grid_real, nunit,
            lines_nvp<T>(N), tw);
  FS_LAUNCH_CHECK();
  return FS_OK;
}
template <int N, typename T>
fs_status y_lines(fs_ctx *c, V16 *A, const V16 *tw, bool inv) {
  const int nv = lines_nv<T>(c->nz), nvp = lines_nvp<T>(c->nz), ncol = 3 * c->nx * nv;
  typedef YShape<N, T> Y;
  const size_t smem = Y::SMEM;
  // The inverse follows the x pass, for whose long lines the SMs give nearly all of their memory
  // to shared memory (51 to 101 KB a CTA from 256 points on). An SM is split anew only when it is
  // empty. Placed programmatically, while the last x CTAs run, the y CTAs kept the x pass's split,
  // and the chain handed it on, L1 short, up to the interpolation's gathers. Whole solves, us,
  // programmatic and plain: FP64 512^3 10,950 and 9,980, FP32 512 x 512 x 256 4,480 and 4,020, FP64
  // 512 x 64 x 64 258 and 240, 256 x 512 x 512 6,510 and 6,360, 320^3 3,190 and 3,140, 256^3 1,280
  // both; on shorter x lines a plain launch is 1 to 3 us more (FP32 64^3 59 and 61).
  if (inv && c->nx >= 256)
    k_lines_y<N, T, true><<<fs_blocks(ncol, Y::COLS), Y::THREADS, smem, c->stream>>>(A, ncol, nv, nvp, tw);
  else if (inv)
    fs_launch(k_lines_y<N, T, true>, fs_blocks(ncol, Y::COLS), Y::THREADS, smem, c->stream, A, ncol, nv, nvp, tw);
  else
    fs_launch(k_lines_y<N, T, false>, fs_blocks(ncol, Y::COLS), Y::THREADS, smem, c->stream, A, ncol, nv, nvp, tw);
  FS_LAUNCH_CHECK();
  return FS_OK;
}
template <int N, typename T>
fs_status x_lines(fs_ctx *c, V16 *A, const V16 *tw) {
  const double TwoPI = 2. * FS_PI;
  XArgs g;
  g.ny = c->ny;
  g.nv = lines_nv<T>(c->nz);
  g.nvp = lines_nvp<T>(c->nz);
  g.ncol = c->ny * g.nv;
  g.rstride = (size_t)c->ny * g.nvp;
  g.cstride = (size_t)c->nx * g.rstride;
  g.ffx = TwoPI / (c->nx * c->p.dx);
  g.ffy = TwoPI / (c->ny * c->p.dx);
  g.ffz = TwoPI / (c->nz * c->p.dx);
  const long double inv = 1.0L / ((long double)c->nx * c->ny * c->nz);
  g.inv_total = Num<T>::IS_DOUBLE ? (double)inv : (double)(float)inv;
  g.inv_total_lo = (double)(inv - (long double)g.inv_total);
  typedef XShape<N> X;
  fs_launch(k_lines_x_project<N, T>, fs_blocks(g.ncol, X::COLS), X::THREADS, X::SMEM, c->stream, A, g, tw);
  FS_LAUNCH_CHECK();
  return FS_OK;
}

// twiddle tables of the context's grid, at c->line_tw[prec][axis]
template <typename T>
fs_status lines_init_t(fs_ctx *c) {
  std::vector<TwRoot> roots;
  size_t off[3];
  off[0] = roots.size();
  FS_LINES_SWITCH(c->nx, x_roots, roots);
  off[1] = roots.size();
  FS_LINES_SWITCH(c->ny, y_roots, roots);
  off[2] = roots.size();
  FS_LINES_SWITCH(c->nz, z_roots, roots);
  std::vector<V16> h(roots.size());
  for (size_t i = 0; i < roots.size(); ++i) {
    const long double a = 2.0L * 3.14159265358979323846264338327950288L * roots[i].j / roots[i].n;
    const double w[2] = {(double)cosl(a), (double)-sinl(a)};
    if (Num<T>::IS_DOUBLE) {
      memcpy(&h[i], w, sizeof(V16));
    } else {
      const float p[4] = {(float)w[0], (float)w[0], (float)w[1], (float)w[1]};
      memcpy(&h[i], p, sizeof(V16));
    }
  }
  const int prec = Num<T>::IS_DOUBLE ? FS_PREC_FP64 : FS_PREC_FP32;
  V16 *d = nullptr;
  FS_CUDA(cudaMalloc(&d, sizeof(V16) * h.size()));
  for (int a = 0; a < 3; ++a) c->line_tw[prec][a] = d + off[a];
  c->bytes += sizeof(V16) * h.size();
  FS_CUDA(cudaMemcpy(d, h.data(), sizeof(V16) * h.size(), cudaMemcpyHostToDevice));
  return FS_OK;
}

// the attributes of the grid's kernels, which loads them: before the context's first solve at
// this precision (and before a capture), so that a context loads no kernel that it never runs
template <typename T>
fs_status lines_prepare_t(fs_ctx *c) {
  bool &ready = c->line_ready[Num<T>::IS_DOUBLE ? FS_PREC_FP64 : FS_PREC_FP32];
  if (ready) return FS_OK;
  FS_LINES_SWITCH(c->nx, x_attrs);
  FS_LINES_SWITCH(c->ny, y_attrs);
  FS_LINES_SWITCH(c->nz, z_attrs);
  ready = true;
  return FS_OK;
}

// u = Stokes solve of f, both [3][nx][ny][nz] in c->grid_real (in place); c->grid_cplx
// holds the half spectrum
template <typename T>
fs_status lines_flow_solve_t(fs_ctx *c) {
  // the single-kernel stages are recorded in FP32 on these grids only (filsim_gpu.h)
  auto timed = [](int n, int from) {
    const int odd = n / (n & -n);
    return odd == 1 ? n >= from : odd == 3 && n >= 96;
  };
  const bool kernel_stages = !Num<T>::IS_DOUBLE && timed(c->nx, 32) && timed(c->ny, 32) && timed(c->nz, 64);
  const int prec = Num<T>::IS_DOUBLE ? FS_PREC_FP64 : FS_PREC_FP32;
  const V16 *twx = (const V16 *)c->line_tw[prec][0], *twy = (const V16 *)c->line_tw[prec][1],
            *twz = (const V16 *)c->line_tw[prec][2];
  V16 *A = (V16 *)c->grid_cplx;
  {
    ProfScope ps(c, FS_STAGE_FFT_FWD);
    {
      ProfScope pk(c, FS_STAGE_K_FFT_Z_FWD, kernel_stages);
      FS_LINES_SWITCH(c->nz, z_fwd, c, A, twz);
    }
    ProfScope pk(c, FS_STAGE_K_FFT_Y_FWD, kernel_stages);
    FS_LINES_SWITCH(c->ny, y_lines, c, A, twy, false);
  }
  {
    ProfScope ps(c, FS_STAGE_PROJECT);
    FS_LINES_SWITCH(c->nx, x_lines, c, A, twx);
  }
  {
    ProfScope ps(c, FS_STAGE_FFT_INV);
    {
      ProfScope pk(c, FS_STAGE_K_FFT_Y_INV, kernel_stages);
      FS_LINES_SWITCH(c->ny, y_lines, c, A, twy, true);
    }
    ProfScope pk(c, FS_STAGE_K_FFT_Z_INV, kernel_stages);
    FS_LINES_SWITCH(c->nz, z_inv, c, A, twz);
  }
  return FS_OK;
}
