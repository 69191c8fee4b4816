// fs_fcm.cu -- Force Coupling Method mobility solve on sm_100a.
//
// Replaces Fcm::mobility_solve (FCMfunctions.cpp:175-464):
//   1. counting sort (BinKey): beads binned by the 16-point tile that
//      holds the start of their Gaussian stencil (gaussian_setup's index rule,
//      FCMfunctions.cpp:565-589).
//   2. k_records64 + k_spread64 (FP64) / k_spread_records32 + k_spread32 (FP32 chain):
//      CTAs over 16^3 grid tiles (FP64: half tiles) gather the monopole + rotlet
//      Gaussians of every bead whose stencil reaches them
//      (mono_and_dipole_force_distribution, :596-646); each lane owns grid points and
//      sums in registers (FP32: Kahan-compensated, on packed f32x2 pairs): no
//      atomics, bit-reproducible.
//   3.-5. the forward transforms, the Stokes projection of flow_solve (:648-736) and
//      the inverse transforms: the line transforms (fs_lines.cuh) on grids whose
//      lengths they take, the warp transform (fs_fft.cu) on the largest FP32 ones,
//      otherwise cuFFT with k_project / k_project_planes between.
//   6. k_interp64 / k_interp_q: one warp (or more) per bead (in spread-bin order for L2
//      locality) reduces U and Omega over the stencil (particle_velocities :740-770,
//      particle_rotations :774-808) with warp shuffles.
// FP64 mode follows the reference arithmetic; FP32 mode keeps grids, FFTs and
// weights in float, with Kahan-compensated spread sums and FP64 accumulation of
// the interpolation products.
#include "fs_internal.cuh"
#include "fs_sort.cuh"
#include <type_traits>
#include "fs_f32x2.cuh"

namespace {

struct FcmConsts {
  int N[3];
  int gnx, x0;  // x extent of the whole box and the grid's first plane in it (a slab window; else N[0], 0)
  int ngd, ngdh;
  int nbin[3];
  double dx;
  double anorm, anorm2, anormdip, anormdip2, sigmadipsq;
};

__host__ __device__ inline int wrap_int(int x, int n) {
  int r = x % n;
  return r < 0 ? r + n : r;
}
// x in (-n, 2n): one conditional add or subtract
__device__ __forceinline__ int wrap_near(int x, int n) {
  x += (x < 0) ? n : 0;
  return x >= n ? x - n : x;
}

// ---- 1. binning -------------------------------------------------------------
// key: the tile bin of the wrapped stencil start; sw: the wrapped stencil
// start per axis (gaussian_setup's index rule, FCMfunctions.cpp:565-585), kept
// for the spread and interpolation kernels so they need no integer division.
struct BinKey {
  const double *Y;
  FcmConsts c;
  int *sw_out;
  __device__ int operator()(int b) const {
    int bi[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      int xc = (int)(Y[3 * b + d] / c.dx);
      // the stencil start in the whole box, then in this grid (a slab window holds the
      // beads whose x start lies in its own planes; others are clamped, never out of range)
      int sw = wrap_int(xc - c.ngdh + 1, d == 0 ? c.gnx : c.N[d]) - (d == 0 ? c.x0 : 0);
      sw = sw < 0 ? 0 : (sw >= c.N[d] ? c.N[d] - 1 : sw);
      sw_out[3 * b + d] = sw;
      bi[d] = sw / FS_TILE;
    }
    return (bi[0] * c.nbin[1] + bi[1]) * c.nbin[2] + bi[2];
  }
};

// ---- 2. spread ----------------------------------------------------------------
// Both precisions first write one record per bead in sorted (bin) order: its stencil
// starts, F, T/2 and the Gaussian weights of its ngd stencil indices per axis
// (gaussian_setup, FCMfunctions.cpp:565-589), read by the spread and the interpolation.
//
// FP64 record (double4 units): [0] stencil starts and bead id (four ints), F0, F1;
// [1] F2, h0, h1, h2 (h = T / 2, GA_setup :536-547); then (g, d, r, r d) of axis a and
// stencil index i at 2 + a ngd + i.
__host__ __device__ inline int rec64_len(int ngd) { return 2 + 3 * ngd; }

__global__ void k_records64(const double *__restrict__ Y, const double *__restrict__ F, const double *__restrict__ T,
                            const int *__restrict__ sorted, const int *__restrict__ bead_sw, int np, FcmConsts c,
                            double4 *__restrict__ rec) {
  FS_AFTER_PREVIOUS();
  const int ngd = c.ngd, RL = rec64_len(ngd);
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long long)np * RL) return;
  const int q = (int)(t / RL), e = (int)(t - (long long)q * RL);
  const int b = sorted[q];
  double4 v;
  if (e == 0) {
    v.x = __hiloint2double(bead_sw[3 * b + 1], bead_sw[3 * b]);
    v.y = __hiloint2double(b, bead_sw[3 * b + 2]);
    v.z = F ? F[3 * b] : 0.0;
    v.w = F ? F[3 * b + 1] : 0.0;
  } else if (e == 1) {
    v.x = F ? F[3 * b + 2] : 0.0;
    v.y = T ? 0.5 * T[3 * b] : 0.0;
    v.z = T ? 0.5 * T[3 * b + 1] : 0.0;
    v.w = T ? 0.5 * T[3 * b + 2] : 0.0;
  } else {
    const int a = (e - 2) / ngd, i = (e - 2) - a * ngd;
    const double Yv = Y[3 * b + a];
    const int xg = (int)(Yv / c.dx) - c.ngdh + (i + 1);
    const double xx = ((double)xg) * c.dx - Yv;
    v.x = c.anorm * exp(-xx * xx / c.anorm2);
    v.y = c.anormdip * exp(-xx * xx / c.anormdip2);
    v.z = -xx / c.sigmadipsq;
    v.w = v.z * v.y;
  }
  rec[t] = v;
}

// The candidate bins of a tile per axis: its own and the ones before it that a stencil
// reaches (fs_cand_bins: K per axis), in the order (x, y, z); combination r < K^3 names, by
// its digit p of each axis, the bin K - 1 - p before the tile's own (empty when it would
// repeat a bin on an axis with fewer than K bins).
struct Cand {
  int rs[27], len[27];
};
__device__ __forceinline__ void cand_bins(Cand &cd, int tx, int ty, int tz, const int *__restrict__ bin_start,
                                          const FcmConsts &c) {
  const int K = fs_cand_bins(c.ngd), r = threadIdx.x;
  if (r >= K * K * K) return;
  const int tb[3] = {tx, ty, tz}, pick[3] = {r / (K * K), (r / K) % K, r % K};
  int bin = 0;
  bool valid = true;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const int back = K - 1 - pick[d];
    valid = valid && back < c.nbin[d];
    bin = bin * c.nbin[d] + wrap_int(tb[d] - back, c.nbin[d]);
  }
  cd.rs[r] = valid ? bin_start[bin] : 0;
  cd.len[r] = valid ? bin_start[bin + 1] - bin_start[bin] : 0;
}
// record of candidate q of the tile
__device__ __forceinline__ int cand_slot(const Cand &cd, int q) {
  int r = 0;
  while (q >= cd.len[r]) {
    q -= cd.len[r];
    ++r;
  }
  return cd.rs[r] + q;
}

// FP64 spread: one CTA (8 warps) per half tile of 8 x 16 x 16 points (ZL = 8; a quarter of 8 x
// 16 x 8 with ZL = 4). Warp w owns the 2 x 16 x ZL points x in {2 (w & 3), +1}, z in
// [ZL (w >> 2), +ZL); a lane owns one x, one y and the ZL z, 3 ZL sums in registers. Per
// staged bead that reaches the warp's points the lane forms the eight x-y factors of
//   f0 = F0 gx gy . gz + h2 ry dx dy . dz - h1 dx dy . rz dz
//   f1 = F1 gx gy . gz - h2 rx dx dy . dz + h0 dx dy . rz dz
//   f2 = F2 gx gy . gz + (h1 rx - h0 ry) dx dy . dz
// (mono_and_dipole_force_distribution, FCMfunctions.cpp:596-646, regrouped) and adds eight
// FMAs per point of the covered z quads, the z weights broadcast from shared memory. The
// candidates that reach the CTA are listed first, 256 at a time, then staged CH at a time in
// that (sorted) order, the sums kept throughout: no atomics, each point written once,
// bit-reproducible. Bound by issue at 24 warps per SM (80 registers) and the staging chain: 1.58
// ms at 512^3 / 131,072 beads and 0.288 ms at 256^3 / 30,720, where one grid point per lane with
// the Gaussians recomputed per tile took 2.38 and 0.52. Before the sums were chains of FMAs (a
// product, a sum and an addition each, eleven operations a point for eight) 1.63 and 0.301, and of
// that form without the list, every candidate staged, 1.83 and 0.36; at 128 registers and 16
// warps per SM 1.83, 0.32.
#define FS_SPREAD64_THREADS 256
constexpr int SPREAD64_CH = 32;  // beads staged at a time (64, at two CTAs per SM: 1.13 times as long at 512^3)
template <int ZL>
struct SpreadStage64 {
  static constexpr int CH = SPREAD64_CH;
  double xg[CH][8], xd[CH][8], xr[CH][8];
  double yg[CH][FS_TILE], yd[CH][FS_TILE], yr[CH][FS_TILE];
  double2 zgd[CH][2 * ZL];  // (g, d)
  double zrd[CH][2 * ZL];   // r d
  double2 f[CH][3];         // (F0, F1), (F2, h0), (h1, h2)
  // the beads of one batch of candidates that reach the CTA: record, covered x (8 bits) |
  // covered z (2 ZL bits) << 16
  int list[FS_SPREAD64_THREADS];
  unsigned lmask[FS_SPREAD64_THREADS];
  int count[FS_SPREAD64_THREADS / 32];
};
// points l < width from X0 on an axis of N points that a stencil of ngd from sw covers
__device__ __forceinline__ unsigned cover_mask(int X0, int sw, int N, int ngd, int width) {
  const int s0 = wrap_near(X0 - sw, N);  // stencil index of l = 0
  unsigned m = s0 < ngd ? (1u << (ngd - s0)) - 1u : 0u;
  if (N - s0 < width) m |= ((1u << ngd) - 1u) << (N - s0);
  return m & ((1u << width) - 1u);
}

template <int ZL>
__global__ void __launch_bounds__(FS_SPREAD64_THREADS, ZL == 4 ? 4 : 3)
    k_spread64(const int *__restrict__ bin_start, const double4 *__restrict__ rec, FcmConsts c,
               double *__restrict__ fgrid) {
  FS_AFTER_PREVIOUS();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int CH = SPREAD64_CH;
  typedef SpreadStage64<ZL> Stage;
  Stage &st = *reinterpret_cast<Stage *>(smem_raw);
  __shared__ Cand cd;
  constexpr int ZP = FS_TILE / (2 * ZL), ZT = 2 * ZL / 8;  // CTAs along a tile's z; z entries per staging thread
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int part = blockIdx.x % (2 * ZP), tile = blockIdx.x / (2 * ZP);
  const int tz = tile % c.nbin[2], ty = (tile / c.nbin[2]) % c.nbin[1], tx = tile / (c.nbin[2] * c.nbin[1]);
  const int X0[3] = {tx * FS_TILE + 8 * (part & 1), ty * FS_TILE, tz * FS_TILE + 2 * ZL * (part >> 1)};
  cand_bins(cd, tx, ty, tz, bin_start, c);
  __syncthreads();
  const int ngd = c.ngd, RL = rec64_len(ngd), K = fs_cand_bins(ngd), nr = K * K * K;
  int total = 0;
  for (int r = 0; r < nr; ++r) total += cd.len[r];
  const int xp = warp & 3, zh = warp >> 2, yl = lane & 15, xl = 2 * xp + (lane >> 4);
  double acc[ZL][3];
#pragma unroll
  for (int z = 0; z < ZL; ++z) acc[z][0] = acc[z][1] = acc[z][2] = 0.0;
  // candidates 256 at a time: those whose stencil reaches the CTA's points, in order
  for (int q0 = 0; q0 < total; q0 += FS_SPREAD64_THREADS) {
    int slot = 0;
    unsigned msk = 0;
    if (q0 + tid < total) {
      slot = cand_slot(cd, q0 + tid);
      const double2 hd = *reinterpret_cast<const double2 *>(rec + (size_t)slot * RL);
      const unsigned mx = cover_mask(X0[0], __double2loint(hd.x), c.N[0], ngd, 8);
      const unsigned my = cover_mask(X0[1], __double2hiint(hd.x), c.N[1], ngd, FS_TILE);
      const unsigned mz = cover_mask(X0[2], __double2loint(hd.y), c.N[2], ngd, 2 * ZL);
      if (mx && my && mz) msk = mx | (mz << 16);
    }
    const unsigned hit = __ballot_sync(0xffffffffu, msk != 0);
    if (lane == 0) st.count[warp] = __popc(hit);
    __syncthreads();  // counts; and the previous list and tables are no longer read
    int nhit = 0, at = 0;
#pragma unroll
    for (int w = 0; w < FS_SPREAD64_THREADS / 32; ++w) {
      const int k = st.count[w];
      if (w < warp) at += k;
      nhit += k;
    }
    if (msk) {
      at += __popc(hit & ((1u << lane) - 1u));
      st.list[at] = slot;
      st.lmask[at] = msk;
    }
    __syncthreads();
    for (int base = 0; base < nhit; base += CH) {
      const int nb = min(CH, nhit - base);
      if (base) __syncthreads();  // the previous tables are no longer read
      // eight threads per slot: thread j takes x = j, y in {j, j + 8}, z likewise
      for (int sl = tid >> 3; sl < nb; sl += FS_SPREAD64_THREADS / 8) {
        const int j = tid & 7;
        const double4 *rw = rec + (size_t)st.list[base + sl] * RL;
        const double4 hd = rw[0];
        const int swv[3] = {__double2loint(hd.x), __double2hiint(hd.x), __double2loint(hd.y)};
        constexpr int NE = 3 + ZT;
        double4 w[NE];
#pragma unroll
        for (int it = 0; it < NE; ++it) {
          const int a = it == 0 ? 0 : it < 3 ? 1 : 2, l = j + 8 * (it == 2 || it == 4), Nn = c.N[a];
          const int i = wrap_near(l + wrap_near(X0[a] - swv[a], Nn), Nn);
          w[it] = i < ngd ? rw[2 + a * ngd + i] : make_double4(0.0, 0.0, 0.0, 0.0);
        }
        if (j < 3) {
          const double4 h1 = rw[1];
          st.f[sl][j] = j == 0 ? make_double2(hd.z, hd.w) : j == 1 ? make_double2(h1.x, h1.y) : make_double2(h1.z, h1.w);
        }
        st.xg[sl][j] = w[0].x;
        st.xd[sl][j] = w[0].y;
        st.xr[sl][j] = w[0].z;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          st.yg[sl][j + 8 * h] = w[1 + h].x;
          st.yd[sl][j + 8 * h] = w[1 + h].y;
          st.yr[sl][j + 8 * h] = w[1 + h].z;
        }
#pragma unroll
        for (int h = 0; h < ZT; ++h) {
          st.zgd[sl][j + 8 * h] = make_double2(w[3 + h].x, w[3 + h].y);
          st.zrd[sl][j + 8 * h] = w[3 + h].w;
        }
      }
      __syncthreads();
      // staged beads reaching this warp's points
      static_assert(CH == 32, "one ballot covers the staged beads");
      const unsigned mm = lane < nb ? st.lmask[base + lane] : 0u;
      unsigned m = __ballot_sync(0xffffffffu, ((mm >> (2 * xp)) & 3u) && ((mm >> (16 + ZL * zh)) & ((1u << ZL) - 1u)));
      while (m) {
        const int sl = __ffs(m) - 1;
        m &= m - 1;
        const unsigned zm = st.lmask[base + sl] >> (16 + ZL * zh);
        const double gx = st.xg[sl][xl], dx = st.xd[sl][xl], rx = st.xr[sl][xl];
        const double gy = st.yg[sl][yl], dy = st.yd[sl][yl], ry = st.yr[sl][yl];
        const double2 f01 = st.f[sl][0], f2h0 = st.f[sl][1], h12 = st.f[sl][2];
        const double p = gx * gy, q = dx * dy;
        const double a0 = f01.x * p, a1 = f01.y * p, a2 = f2h0.x * p;
        const double b0 = h12.y * ry * q, b1 = -h12.y * rx * q, b2 = (h12.x * rx - f2h0.y * ry) * q;
        const double c0 = -h12.x * q, c1 = f2h0.y * q;
#pragma unroll
        for (int k = 0; k < ZL / 4; ++k) {
          if (ZL == 4 || ((zm >> (4 * k)) & 0xfu)) {
#pragma unroll
            for (int z = 4 * k; z < 4 * k + 4; ++z) {
              const double2 gd = st.zgd[sl][ZL * zh + z];
              const double rd = st.zrd[sl][ZL * zh + z];
              acc[z][0] = fma(a0, gd.x, fma(b0, gd.y, fma(c0, rd, acc[z][0])));
              acc[z][1] = fma(a1, gd.x, fma(b1, gd.y, fma(c1, rd, acc[z][1])));
              acc[z][2] = fma(a2, gd.x, fma(b2, gd.y, acc[z][2]));
            }
          }
        }
      }
    }
  }
  // through shared memory, as many components at a time as the tables have room for, so
  // that neighbouring lanes write whole rows of the CTA's z
  constexpr int RP = ZL + 1;  // pairs per row: ZL and a pad
  constexpr size_t ROWS = sizeof(double2) * 128 * RP;
  static_assert(sizeof(Stage) >= ROWS, "the tables hold one component");
  constexpr int NC = sizeof(Stage) >= 3 * ROWS ? 3 : 1;
  const size_t N = (size_t)c.N[0] * c.N[1] * c.N[2];
  double2 *T = reinterpret_cast<double2 *>(smem_raw);  // [component][128 (x, y)][RP]
  double *out = fgrid + ((size_t)X0[0] * c.N[1] + X0[1]) * c.N[2] + X0[2] + 2 * (tid % ZL);
#pragma unroll
  for (int a0 = 0; a0 < 3; a0 += NC) {
    __syncthreads();  // the tables, or the previous components, are no longer read
#pragma unroll
    for (int a = 0; a < NC; ++a)
#pragma unroll
      for (int z = 0; z < ZL; z += 2)
        T[(128 * a + 16 * xl + yl) * RP + ZL / 2 * zh + z / 2] = make_double2(acc[z][a0 + a], acc[z + 1][a0 + a]);
    __syncthreads();
#pragma unroll
    for (int a = 0; a < NC; ++a)
#pragma unroll
      for (int r = tid / ZL; r < 128; r += FS_SPREAD64_THREADS / ZL)
        *reinterpret_cast<double2 *>(out + (a0 + a) * N + ((size_t)(r >> 4) * c.N[1] + (r & 15)) * c.N[2]) =
            T[(128 * a + r) * RP + tid % ZL];
  }
}

// ---- 2b. FP32 spread on packed pairs -------------------------------------------
// The FP32 chain's spread. k_spread_records32 writes each bead's record with xx = xg dx - Y
// in double and the Gaussians in float.
// In k_spread32 a 16^3 tile is 16 column blocks, a warp each, shared out over 1, 2 or 4 CTAs. A
// CTA lists the beads whose stencil reaches its points, stages tables of them (by tile
// coordinate, from their records) and sums its columns; with the default 2 x 16 x 8 blocks,
// column q has x in [2 (q % 8), +2), z in [8 (q / 8), +8) and lane l owns x = 2 (q % 8) +
// (l & 1), the z pair 8 (q / 8) + 2 ((l >> 1) & 3) + {0, 1} and y = (l >> 3) + 4k, k < 4:
// eight points held as four packed pairs per component. Per staged bead reaching the warp's
// column the lane forms the x-z factors of its pair once, then each covered y row costs
// three packed FMA chains and three packed Kahan updates:
//   y = term + nc, t = s + y, nc = y - (t - s), s = t      (nc = -c of Kahan)
// The sums run over the candidates in sorted bead order and are written once
// per point (s + nc): no atomics, bit-reproducible.
// Bound by a CTA's chain (bins -> headers -> records -> tables) on small grids and by the
// packed updates (half of the lanes' points lie in a stencil) with that chain on large ones;
// staging only the beads of the list (20 to 25% of the candidates) is what helps both.
constexpr int SPREAD32_BATCH = 256;

// Record of the bead in sorted slot q (float4 units): [0] stencil starts and bead id
// (int), [1] F0, F1, F2, h0, [2] h1, h2, -, -, then (g, d, r, r d) for axis a and stencil
// index i at 3 + a ngd + i.
__host__ __device__ inline int spread_rec_len(int ngd) { return 3 + 3 * ngd; }

__global__ void k_spread_records32(const double *__restrict__ Y, const double *__restrict__ F,
                                   const double *__restrict__ T, const int *__restrict__ sorted,
                                   const int *__restrict__ bead_sw, int np, FcmConsts c, float4 *__restrict__ rec) {
  FS_AFTER_PREVIOUS();
  const int ngd = c.ngd, RL = spread_rec_len(ngd);
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long long)np * RL) return;
  const int q = (int)(t / RL), e = (int)(t - (long long)q * RL);
  const int bead = sorted[q];
  float4 v;
  if (e == 0) {
    v = make_float4(__int_as_float(bead_sw[3 * bead]), __int_as_float(bead_sw[3 * bead + 1]),
                    __int_as_float(bead_sw[3 * bead + 2]), __int_as_float(bead));
  } else if (e <= 2 && !F) {
    v = make_float4(0.f, 0.f, 0.f, 0.f);
  } else if (e == 1) {
    v = make_float4((float)F[3 * bead], (float)F[3 * bead + 1], (float)F[3 * bead + 2], (float)(0.5 * T[3 * bead]));
  } else if (e == 2) {
    v = make_float4((float)(0.5 * T[3 * bead + 1]), (float)(0.5 * T[3 * bead + 2]), 0.f, 0.f);
  } else {
    const int a = (e - 3) / ngd, i = (e - 3) - a * ngd;
    const double Yv = Y[3 * bead + a];
    const int xc = (int)(Yv / c.dx);
    const int xg = xc - c.ngdh + (i + 1);
    const double xx = ((double)xg) * c.dx - Yv;
    const float xf = (float)xx;
    const float g = (float)c.anorm * expf(-xf * xf / (float)c.anorm2);
    const float d = (float)c.anormdip * expf(-xf * xf / (float)c.anormdip2);
    const float r = -xf / (float)c.sigmadipsq;
    v = make_float4(g, d, r, r * d);
  }
  rec[t] = v;
}


// the staged chunk: tables by tile coordinate, built straight from the records in
// global memory (spread32_smem bytes of dynamic shared memory)
template <int CH>
struct SpreadStage32 {
  float4 xw[CH][FS_TILE];                    // (g, d, r, -) by tile-local x
  float zg[CH][FS_TILE], zd[CH][FS_TILE], zr[CH][FS_TILE];  // by tile-local z
  float4 yw[CH][FS_TILE];                    // (g, g, d, d) by tile-local y
  float2 yrd[CH][FS_TILE];                   // (r d, r d)
  float4 fh[CH], hh[CH];                     // (F0, F1, F2, h0), (h1, h2, -, -): h = T / 2
  // the beads of one batch of candidates that reach the CTA: record, covered x (16 bits) |
  // covered z (16 bits) << 16, y rows k with a covered y in [4k, 4k + 4)
  int list[SPREAD32_BATCH];
  unsigned lmask[SPREAD32_BATCH];
  unsigned char lrows[SPREAD32_BATCH];
  int count[SPREAD32_BATCH / 32];
};

// CX: the shape of a warp's column block, CX x 16 x (16 / CX) points (x, y, z), an autotuner
// knob (2, 4 or 8); a lane owns one x, one z pair and four y rows. NW: warps (column blocks)
// per CTA, PASSES: columns a warp does in turn on the same tables. Measured (us, 12-point
// stencils, 4 to 8 beads per tile), against a whole tile in two passes over all candidates:
//   tiles               27    64   216   512   864 (20-point)   4,096   32,768
//   before              31    39    22    35       109            234      927
//   4 warps, 1 pass     15    21    21    34        86            270     1487
//   8 warps, 1 pass     18    22    20    33        78            237     1308
//   8 warps, 2 passes   27    35    27    36        86            226      992
//   4 warps, 4 passes   53    68    47    57       121            254      909
// so quarter tiles below one tile per SM, then half tiles; the list is made once for a whole
// tile where the CTAs are enough without a split and a tile's beads few (half / whole: 343 tiles
// reached by 22 beads 25 / 28; 384 by 10, 20 and 27 22 / 18, 26 / 24, 30 / 30; 1,000 by 10, 27 and 40
// 41 / 32, 54 / 51, 68 / 72; 1,584 by 10, 27 and 40 56 / 40, 78 / 69, 97 / 99; 4,096 by 40 and 60
// 236 / 236, 333 / 339), and by four warps, which fit an SM more often, where the beads fit one
// stage and the CTAs are many waves (whole / by four warps: 1,584 tiles reached by 4 and 10 beads
// 34 / 30, 40 / 40; 4,096 by 10 and 20 95 / 83, 130 / 134; 8,000 by 20 and 27 237 / 223, 296 / 295;
// 21,952 by 27 and 40 780 / 752, 1,200 / 1,292).
template <int CH, int CX, int NW, int PASSES>
__global__ void __launch_bounds__(32 * NW, NW == 4 && PASSES == 4 ? 6 : 3)
    k_spread32(const int *__restrict__ bin_start, const float4 *__restrict__ rec, FcmConsts c,
               float *__restrict__ fgrid) {
  FS_AFTER_PREVIOUS();
  static_assert(CX == 2 || CX == 4 || CX == 8, "column widths");
  constexpr int CZ = FS_TILE / CX, NCX = FS_TILE / CX;  // z width; columns across x
  constexpr int NT = 32 * NW, PARTS = 16 / (NW * PASSES), COLS = NW * PASSES;  // columns per CTA
  constexpr int XW = NCX > COLS ? CX * COLS : FS_TILE, ZW = NCX > COLS ? CZ : CZ * (COLS / NCX);  // the CTA's points
  extern __shared__ __align__(16) unsigned char smem_raw[];
  SpreadStage32<CH> &st = *reinterpret_cast<SpreadStage32<CH> *>(smem_raw);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int part = blockIdx.x % PARTS, tile = blockIdx.x / PARTS;
  const int tz = tile % c.nbin[2], ty = (tile / c.nbin[2]) % c.nbin[1], tx = tile / (c.nbin[2] * c.nbin[1]);
  const int X0[3] = {tx * FS_TILE, ty * FS_TILE, tz * FS_TILE};
  const int xlo = NCX > COLS ? CX * ((part * COLS) % NCX) : 0, zlo = CZ * ((part * COLS) / NCX);
  const unsigned ctam = ((((1u << XW) - 1u) << xlo) & 0xffffu) | (((1u << ZW) - 1u) << (16 + zlo));
  __shared__ Cand cd;
  cand_bins(cd, tx, ty, tz, bin_start, c);
  __syncthreads();
  const int ngd = c.ngd, RL = spread_rec_len(ngd), K = fs_cand_bins(ngd), nr = K * K * K;
  int total = 0;
  for (int r = 0; r < nr; ++r) total += cd.len[r];
  const int ly = lane >> 3;
  int nhit = 0;
#pragma unroll 1
  for (int pass = 0; pass < PASSES; ++pass) {
    const int cx = (part * COLS + pass * NW + warp) % NCX, cz = (part * COLS + pass * NW + warp) / NCX;
    const unsigned warpm = (((1u << CX) - 1u) << (CX * cx)) | (((1u << CZ) - 1u) << (16 + CZ * cz));
    const int xl = CX * cx + (lane % CX), zl = CZ * cz + 2 * ((lane / CX) % (CZ / 2));
    f2p s[4][3], nc[4][3];
#pragma unroll
    for (int k = 0; k < 4; ++k)
#pragma unroll
      for (int a = 0; a < 3; ++a) s[k][a] = nc[k][a] = 0ull;
    // candidates SPREAD32_BATCH at a time: those whose stencil reaches the CTA's points, in order
    for (int q0 = 0; q0 < total; q0 += SPREAD32_BATCH) {
      if (pass == 0 || total > SPREAD32_BATCH) {  // else the first pass's list stands
        constexpr int H = SPREAD32_BATCH / NT;
        int slot[H];
        unsigned msk[H], rows[H], hit[H];
#pragma unroll
        for (int h = 0; h < H; ++h) {
          const int q = q0 + h * NT + tid;
          slot[h] = 0;
          msk[h] = rows[h] = 0;
          if (q < total) {
            slot[h] = cand_slot(cd, q);
            const float4 hd = __ldg(rec + (size_t)slot[h] * RL);
            const unsigned m = cover_mask(X0[0], __float_as_int(hd.x), c.N[0], ngd, FS_TILE) |
                               (cover_mask(X0[2], __float_as_int(hd.z), c.N[2], ngd, FS_TILE) << 16);
            const unsigned my = cover_mask(X0[1], __float_as_int(hd.y), c.N[1], ngd, FS_TILE);
#pragma unroll
            for (int k = 0; k < 4; ++k) rows[h] |= ((my >> (4 * k)) & 0xfu) ? (1u << k) : 0u;
            if ((m & ctam & 0xffffu) && (m & ctam) >> 16 && my) msk[h] = m;
          }
          hit[h] = __ballot_sync(0xffffffffu, msk[h] != 0);
          if (lane == 0) st.count[NW * h + warp] = __popc(hit[h]);
        }
        __syncthreads();  // counts; and the previous list and tables are no longer read
        int at[H];
        nhit = 0;
#pragma unroll
        for (int w = 0; w < SPREAD32_BATCH / 32; ++w) {
#pragma unroll
          for (int h = 0; h < H; ++h)
            if (w == NW * h + warp) at[h] = nhit;
          nhit += st.count[w];
        }
#pragma unroll
        for (int h = 0; h < H; ++h)
          if (msk[h]) {
            const int i = at[h] + __popc(hit[h] & ((1u << lane) - 1u));
            st.list[i] = slot[h];
            st.lmask[i] = msk[h];
            st.lrows[i] = (unsigned char)rows[h];
          }
        __syncthreads();
      }
      for (int base = 0; base < nhit; base += CH) {
        const int nb = min(CH, nhit - base);
        if (pass == 0 || total > SPREAD32_BATCH || nhit > CH) {  // else the first pass's tables stand
          if (base || pass) __syncthreads();  // the previous tables are no longer read
          // tables by tile coordinate, eight threads per slot (thread j takes x, y and z in
          // {j, j + 8}), each reading its slot's record from global memory; not copying the
          // records in first keeps a CTA at 57 KB of shared memory with 64 beads a stage
          for (int sl = tid >> 3; sl < nb; sl += NT / 8) {
            const int j = tid & 7;
            const float4 *rw = rec + (size_t)st.list[base + sl] * RL;
            const float4 hd = __ldg(rw);
            if (j == 0) st.fh[sl] = __ldg(rw + 1);
            if (j == 1) st.hh[sl] = __ldg(rw + 2);
            const int swv[3] = {__float_as_int(hd.x), __float_as_int(hd.y), __float_as_int(hd.z)};
            float4 w[6];
#pragma unroll
            for (int it = 0; it < 6; ++it) {
              const int a = it >> 1, l = j + 8 * (it & 1), Nn = c.N[a];
              const int i = wrap_near(l + wrap_near(X0[a] - swv[a], Nn), Nn);
              w[it] = i < ngd ? __ldg(rw + 3 + a * ngd + i) : make_float4(0.f, 0.f, 0.f, 0.f);
            }
            st.xw[sl][j] = w[0];
            st.xw[sl][j + 8] = w[1];
            st.yw[sl][j] = make_float4(w[2].x, w[2].x, w[2].y, w[2].y);
            st.yrd[sl][j] = make_float2(w[2].w, w[2].w);
            st.yw[sl][j + 8] = make_float4(w[3].x, w[3].x, w[3].y, w[3].y);
            st.yrd[sl][j + 8] = make_float2(w[3].w, w[3].w);
            st.zg[sl][j] = w[4].x;
            st.zd[sl][j] = w[4].y;
            st.zr[sl][j] = w[4].z;
            st.zg[sl][j + 8] = w[5].x;
            st.zd[sl][j + 8] = w[5].y;
            st.zr[sl][j + 8] = w[5].z;
          }
          __syncthreads();
        }
        // staged beads reaching this warp's column
        typedef typename std::conditional<CH == 64, unsigned long long, unsigned>::type mask_t;
        mask_t m = 0;
#pragma unroll
        for (int h = 0; h < CH / 32; ++h) {
          const int sl = 32 * h + lane;
          const unsigned mm = sl < nb ? st.lmask[base + sl] & warpm : 0u;
          m |= (mask_t)__ballot_sync(0xffffffffu, (mm & 0xffffu) && (mm >> 16)) << (32 * h % (8 * sizeof(mask_t)));
        }
        while (m) {
          const int sl = (CH == 64 ? __ffsll((long long)m) : __ffs((int)m)) - 1;
          m &= m - 1;
          const unsigned rows = st.lrows[base + sl];
          const float4 wx = st.xw[sl][xl];
          const float2 gz = *reinterpret_cast<const float2 *>(&st.zg[sl][zl]);
          const float2 dz = *reinterpret_cast<const float2 *>(&st.zd[sl][zl]);
          const float2 rz = *reinterpret_cast<const float2 *>(&st.zr[sl][zl]);
          const float4 fh = st.fh[sl];  // F0, F1, F2, h0 (h = T / 2, GA_setup :536-547)
          const float4 hh = st.hh[sl];  // h1, h2
          // per z of the pair: f_a = F_a gx gz, the rotlet factors (d = gdx gdz)
          const float gxz0 = wx.x * gz.x, gxz1 = wx.x * gz.y;
          const float dxz0 = wx.y * dz.x, dxz1 = wx.y * dz.y;
          const f2p f0 = f2_pack(fh.x * gxz0, fh.x * gxz1);
          const f2p f1 = f2_pack(fh.y * gxz0, fh.y * gxz1);
          const f2p f2v = f2_pack(fh.z * gxz0, fh.z * gxz1);
          const f2p h2d = f2_pack(hh.y * dxz0, hh.y * dxz1);
          const f2p mh0d = f2_pack(-fh.w * dxz0, -fh.w * dxz1);
          const f2p c0 = f2_pack(-hh.x * rz.x * dxz0, -hh.x * rz.y * dxz1);
          const f2p c1 = f2_pack((-hh.y * wx.z + fh.w * rz.x) * dxz0, (-hh.y * wx.z + fh.w * rz.y) * dxz1);
          const f2p c2 = f2_pack(hh.x * wx.z * dxz0, hh.x * wx.z * dxz1);
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            if (rows & (1u << k)) {
              const ulonglong2 gd = *reinterpret_cast<const ulonglong2 *>(&st.yw[sl][ly + 4 * k]);
              const f2p rd = *reinterpret_cast<const f2p *>(&st.yrd[sl][ly + 4 * k]);
              f2p y, t;
              // f0 g + h2d (r d) + c0 d
              y = f2_fma(f0, gd.x, f2_fma(h2d, rd, f2_fma(c0, gd.y, nc[k][0])));
              t = f2_add(s[k][0], y);
              nc[k][0] = f2_sub(y, f2_sub(t, s[k][0]));
              s[k][0] = t;
              // f1 g + c1 d
              y = f2_fma(f1, gd.x, f2_fma(c1, gd.y, nc[k][1]));
              t = f2_add(s[k][1], y);
              nc[k][1] = f2_sub(y, f2_sub(t, s[k][1]));
              s[k][1] = t;
              // f2 g + c2 d - h0d (r d)
              y = f2_fma(f2v, gd.x, f2_fma(mh0d, rd, f2_fma(c2, gd.y, nc[k][2])));
              t = f2_add(s[k][2], y);
              nc[k][2] = f2_sub(y, f2_sub(t, s[k][2]));
              s[k][2] = t;
            }
          }
        }
      }
    }
    const size_t N = (size_t)c.N[0] * c.N[1] * c.N[2];
    if constexpr (PASSES > 1) {  // one write per point, s - c (the tables are read again)
      float *out = fgrid + ((size_t)(X0[0] + xl) * c.N[1] + X0[1] + ly) * c.N[2] + X0[2] + zl;
#pragma unroll
      for (int k = 0; k < 4; ++k)
#pragma unroll
        for (int a = 0; a < 3; ++a)
          *reinterpret_cast<float2 *>(out + a * N + (size_t)(4 * k) * c.N[2]) = f2_unpack(f2_add(s[k][a], nc[k][a]));
    } else {
      // one write per point, s - c: through shared memory, so that neighbouring lanes write whole
      // rows of the CTA's z (a warp's own columns are parts of sectors)
      constexpr int XP = FS_TILE * ZW + 4;  // floats per x plane and component
      static_assert(PASSES > 1 || sizeof(SpreadStage32<CH>) >= sizeof(float) * 3 * XW * XP, "the tables hold the points");
      __syncthreads();
      float *T = reinterpret_cast<float *>(smem_raw);
#pragma unroll
      for (int k = 0; k < 4; ++k)
#pragma unroll
        for (int a = 0; a < 3; ++a)
          *reinterpret_cast<float2 *>(T + (a * XW + xl - xlo) * XP + (ly + 4 * k) * ZW + zl - zlo) =
              f2_unpack(f2_add(s[k][a], nc[k][a]));
      __syncthreads();
      constexpr int Q = ZW / 4;  // float4 per row
      for (int i = tid; i < 3 * XW * FS_TILE * Q; i += NT) {
        const int z4 = i % Q, y = (i / Q) % FS_TILE, ax = i / (Q * FS_TILE), a = ax / XW, x = ax - a * XW;
        const float4 v = *reinterpret_cast<const float4 *>(T + ax * XP + y * ZW + 4 * z4);
        *reinterpret_cast<float4 *>(fgrid + a * N + ((size_t)(X0[0] + xlo + x) * c.N[1] + X0[1] + y) * c.N[2] + X0[2] +
                                    zlo + 4 * z4) = v;
      }
    }
  }
}

// ---- 4. Stokes projection -----------------------------------------------------
template <typename R>
struct Cplx;
template <>
struct Cplx<double> { typedef double2 T; };
template <>
struct Cplx<float> { typedef float2 T; };

template <typename R>
__device__ inline void project_mode(R q1, R q2, R q3, R a1, R a2, R a3, R total, R &u1, R &u2, R &u3) {
  const R qq = q2 * q2 + q1 * q1 + (R)1e-18;
  const R norm = (R)1.0 / (qq + q3 * q3);
  const R kdotf = (q1 * a1 + q2 * a2 + q3 * a3) * norm;
  u1 = norm * (a1 - q1 * kdotf) / total;
  u2 = norm * (a2 - q2 * kdotf) / total;
  u3 = norm * (a3 - q3 * kdotf) / total;
}

template <typename R>
__device__ inline R wavenumber(int i, int n, R ff) {
  return (R)((i <= n / 2) ? i : i - n) * ff;
}

// modes with 0 < kz < nz/2 (each stored once in the half spectrum)
template <typename R>
__global__ void k_project(typename Cplx<R>::T *__restrict__ fh, size_t NH, int nx, int ny, int nz, int nzh, R ffx,
                          R ffy, R ffz, R total) {
  FS_AFTER_PREVIOUS();
  typedef typename Cplx<R>::T C;
  size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= NH) return;
  const int k = (int)(idx % nzh);
  if (k == 0 || 2 * k == nz) return;
  const int j = (int)((idx / nzh) % ny);
  const int i = (int)(idx / ((size_t)nzh * ny));
  const R q1 = wavenumber<R>(i, nx, ffx), q2 = wavenumber<R>(j, ny, ffy), q3 = (R)k * ffz;
  C a = fh[idx], b = fh[NH + idx], d = fh[2 * NH + idx];
  C ua, ub, ud;
  project_mode<R>(q1, q2, q3, a.x, b.x, d.x, total, ua.x, ub.x, ud.x);
  project_mode<R>(q1, q2, q3, a.y, b.y, d.y, total, ua.y, ub.y, ud.y);
  fh[idx] = ua;
  fh[NH + idx] = ub;
  fh[2 * NH + idx] = ud;
}

// kz = 0 and kz = nz/2 planes. The reference's inverse real transform uses
// only the real part of the last axis's DC and Nyquist coefficients after the
// complex transforms of the other axes, which equals inverting the Hermitian
// part of these planes: u_sym(i,j) = (u(i,j) + conj(u(-i,-j))) / 2. Writing
// that exactly Hermitian plane makes the C2R result well defined.
template <typename R>
__global__ void k_project_planes(typename Cplx<R>::T *__restrict__ fh, size_t NH, int nx, int ny, int nz, int nzh,
                                 R ffx, R ffy, R ffz, R total) {
  FS_AFTER_PREVIOUS();
  typedef typename Cplx<R>::T C;
  const int ij = blockIdx.x * blockDim.x + threadIdx.x;
  if (ij >= nx * ny) return;
  const int kp = blockIdx.y == 0 ? 0 : nz / 2;
  if (blockIdx.y == 1 && (nz % 2 != 0 || nz / 2 == 0)) return;
  const int i = ij / ny, j = ij % ny;
  const int ip = (nx - i) % nx, jp = (ny - j) % ny;
  const int ijp = ip * ny + jp;
  if (ijp < ij) return;  // the partner handles the pair
  const size_t m = (size_t)ij * nzh + kp, mp = (size_t)ijp * nzh + kp;
  const R q3 = (R)kp * ffz;
  C u[3], up[3];
  {
    const R q1 = wavenumber<R>(i, nx, ffx), q2 = wavenumber<R>(j, ny, ffy);
    C a = fh[m], b = fh[NH + m], d = fh[2 * NH + m];
    project_mode<R>(q1, q2, q3, a.x, b.x, d.x, total, u[0].x, u[1].x, u[2].x);
    project_mode<R>(q1, q2, q3, a.y, b.y, d.y, total, u[0].y, u[1].y, u[2].y);
  }
  {
    const R q1 = wavenumber<R>(ip, nx, ffx), q2 = wavenumber<R>(jp, ny, ffy);
    C a = fh[mp], b = fh[NH + mp], d = fh[2 * NH + mp];
    project_mode<R>(q1, q2, q3, a.x, b.x, d.x, total, up[0].x, up[1].x, up[2].x);
    project_mode<R>(q1, q2, q3, a.y, b.y, d.y, total, up[0].y, up[1].y, up[2].y);
  }
  const bool zero_mode = (kp == 0 && ij == 0);
#pragma unroll
  for (int cpt = 0; cpt < 3; ++cpt) {
    C s;
    s.x = (R)0.5 * (u[cpt].x + up[cpt].x);
    s.y = (R)0.5 * (u[cpt].y - up[cpt].y);
    if (zero_mode) s.x = s.y = (R)0;
    if (ijp == ij) s.y = (R)0;
    fh[(size_t)cpt * NH + m] = s;
    if (ijp != ij) {
      C sc;
      sc.x = s.x;
      sc.y = -s.y;
      fh[(size_t)cpt * NH + mp] = sc;
    }
  }
}

// ---- 6. interpolation -------------------------------------------------------
// U and Omega of a bead from its stencil (particle_velocities :740-770,
// particle_rotations :774-808): SPLIT warps per bead, in spread-bin order, weights from the
// bead's record. interp_finish reduces the warps' lane sums (shuffles, then the bead's
// warps in order) and writes; every thread of the CTA calls it.
template <int WPB, int SPLIT>
__device__ __forceinline__ void interp_finish(double (&v)[6], bool on, int b, double dx, double *__restrict__ V,
                                              double *__restrict__ W) {
  __shared__ double part[SPLIT > 1 ? WPB : 1][6];
  const int lane = threadIdx.x & 31, wl = threadIdx.x >> 5;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
#pragma unroll
    for (int k = 0; k < 6; ++k) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
  if constexpr (SPLIT > 1) {
    if (lane == 0)
      for (int k = 0; k < 6; ++k) part[wl][k] = v[k];
    __syncthreads();
    if (wl % SPLIT == 0 && lane == 0)
#pragma unroll
      for (int w = 1; w < SPLIT; ++w)
        for (int k = 0; k < 6; ++k) v[k] += part[wl + w][k];
  }
  if (on && wl % SPLIT == 0 && lane == 0) {
    const double norm = dx * dx * dx;
    for (int k = 0; k < 3; ++k) {
      V[3 * b + k] = v[k] * norm;
      W[3 * b + k] = -0.5 * v[3 + k] * norm;
    }
  }
}

// FP64. A lane owns an aligned pair of z points and some of the stencil's y indices j, and
// runs along x: per (j, pair) the eight sums over i
//   Sg_c = sum gx u_c,  Sd_c = sum dx u_c (c = 0, 1, 2),  Sr_c = sum rx dx u_c (c = 1, 2)
// need only the x weights, broadcast from shared memory, one FMA per point each; the y and
// z weights are applied afterwards:
//   V_c += gy gz Sg_c,  W0 += ry dy dz Sd_2 - dy rz dz Sd_1,
//   W1 += dy rz dz Sd_0 - dy dz Sr_2,  W2 += dy dz Sr_1 - ry dy dz Sd_0.
// The run of ngd points from zs touches P = (ngd + (zs & 1) + 1) / 2 pairs (a pair that a
// short axis wraps onto twice has disjoint weights the two times); 32 / P rows j at once.
// Bound by the latency of its gathers, eighteen in flight a lane: 0.72 ms at 512^3 / 131,072
// beads, 0.156 ms at 256^3 / 30,720 (one point at a time with all weights from shared memory:
// 1.16, 0.26; steps of 2, 4, 12 along x in place of 6: 0.86, 0.81, 0.86 and 0.184, 0.171, 0.184);
// with the x-y products tabled per warp and the pairs walked across them 0.97, 0.21.
struct InterpWarp64 {
  double xg[FS_NGD_MAX], xd[FS_NGD_MAX], xr[FS_NGD_MAX];  // g, d, r d
  double yg[FS_NGD_MAX], yd[FS_NGD_MAX], yr[FS_NGD_MAX];
  long long xoff[FS_NGD_MAX];
};
// MASK (velocities that a caller gives): the pair's point off the run is dropped from the sums and
// not only given a weight of zero, which would not do where it is no finite number. After a
// solve, whose velocities are finite all or none, it would only cost (a bead's warps at 20
// points 76 -> 132 us for 1,480 beads).
template <int WPB, int SPLIT, bool MASK>
__global__ void __launch_bounds__(32 * WPB) k_interp64(const double *__restrict__ u, const double4 *__restrict__ rec,
                                                       int np, FcmConsts c, double *__restrict__ V,
                                                       double *__restrict__ W) {
  FS_AFTER_PREVIOUS();
  __shared__ InterpWarp64 sw[WPB];
  const int lane = threadIdx.x & 31, wl = threadIdx.x >> 5;
  const int slot = (blockIdx.x * WPB + wl) / SPLIT, ws = wl % SPLIT;
  const bool on = slot < np;  // warp-uniform
  InterpWarp64 &s = sw[wl];
  double acc[6] = {0, 0, 0, 0, 0, 0};  // V, W
  int b = 0;
  if (on) {
    const int ngd = c.ngd, Nz = c.N[2];
    const double4 *rw = rec + (size_t)slot * rec64_len(ngd);
    const double2 hd = *reinterpret_cast<const double2 *>(rw);
    const int sx = __double2loint(hd.x), sy = __double2hiint(hd.x), zs = __double2loint(hd.y);
    b = __double2hiint(hd.y);
    rw += 2;
    if (lane < ngd) {
      const double4 x = rw[lane], y = rw[ngd + lane];
      s.xg[lane] = x.x;
      s.xd[lane] = x.y;
      s.xr[lane] = x.w;
      s.yg[lane] = y.x;
      s.yd[lane] = y.y;
      s.yr[lane] = y.w;
      const int ix = sx + lane;
      s.xoff[lane] = (long long)(ix >= c.N[0] ? ix - c.N[0] : ix) * c.N[1] * Nz;
    }
    const int odd = zs & 1, P = (ngd + odd + 1) >> 1, G = 32 / P;
    const int pr = lane % P, g = lane / P;
    double gz[2], dz[2], rz[2];
    bool in[2];
#pragma unroll
    for (int t = 0; t < 2; ++t) {
      const int k = 2 * pr + t - odd;
      in[t] = k >= 0 && k < ngd;
      const double4 z = rw[2 * ngd + (in[t] ? k : 0)];
      gz[t] = in[t] ? z.x : 0.0;
      dz[t] = in[t] ? z.y : 0.0;
      rz[t] = in[t] ? z.w : 0.0;
    }
    int z0 = zs - odd + 2 * pr;
    if (z0 >= Nz) z0 -= Nz;
    __syncwarp();
    const size_t N = (size_t)c.N[0] * c.N[1] * Nz;
    const int i0 = ws * ngd / SPLIT, i1 = (ws + 1) * ngd / SPLIT;
    for (int j = g; j < ngd && g < G; j += G) {
      const int iy = sy + j;
      const double *base = u + (size_t)(iy >= c.N[1] ? iy - c.N[1] : iy) * Nz + z0;
      double2 Sg[3], Sd[3], Sr[2];
#pragma unroll
      for (int a = 0; a < 3; ++a) Sg[a] = Sd[a] = Sr[a < 2 ? a : 0] = make_double2(0.0, 0.0);
      auto add = [](double2 &t, double w, const double2 &m) {
        t.x += w * m.x;
        t.y += w * m.y;
      };
#pragma unroll (SPLIT > 1 ? 4 : 6)
      for (int i = i0; i < i1; ++i) {
        const double *q = base + s.xoff[i];
        const double2 u0 = __ldg(reinterpret_cast<const double2 *>(q)),
                      u1 = __ldg(reinterpret_cast<const double2 *>(q + N)),
                      u2 = __ldg(reinterpret_cast<const double2 *>(q + 2 * N));
        const double wg = s.xg[i], wd = s.xd[i], wr = s.xr[i];
        add(Sg[0], wg, u0);
        add(Sg[1], wg, u1);
        add(Sg[2], wg, u2);
        add(Sd[0], wd, u0);
        add(Sd[1], wd, u1);
        add(Sd[2], wd, u2);
        add(Sr[0], wr, u1);
        add(Sr[1], wr, u2);
      }
      if constexpr (MASK) {
        auto drop = [&](double2 &t) {
          if (!in[0]) t.x = 0.0;
          if (!in[1]) t.y = 0.0;
        };
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          drop(Sg[a]);
          drop(Sd[a]);
          if (a < 2) drop(Sr[a]);
        }
      }
      const double yg = s.yg[j], yd = s.yd[j], yr = s.yr[j];
#pragma unroll
      for (int a = 0; a < 3; ++a) acc[a] += yg * (gz[0] * Sg[a].x + gz[1] * Sg[a].y);
      acc[3] += yr * (dz[0] * Sd[2].x + dz[1] * Sd[2].y) - yd * (rz[0] * Sd[1].x + rz[1] * Sd[1].y);
      acc[4] += yd * ((rz[0] * Sd[0].x + rz[1] * Sd[0].y) - (dz[0] * Sr[1].x + dz[1] * Sr[1].y));
      acc[5] += yd * (dz[0] * Sr[0].x + dz[1] * Sr[0].y) - yr * (dz[0] * Sd[0].x + dz[1] * Sd[0].y);
    }
  }
  interp_finish<WPB, SPLIT>(acc, on, b, c.dx, V, W);
}

// FP32, float4 gathers along z. The stencil's z run of ngd points starting at zs lies in
// nq = ceil(((zs & 3) + ngd) / 4) aligned quads of four points (a quad that a short axis
// wraps onto twice has disjoint weights the two times). A lane takes (ij, quad) slots: one
// 16-byte load per component, z weights per quad position (zero off the run), the quad's
// four products summed in FP32 and the sum added in FP64. 0.525 ms at 512^3 / 131,072
// beads; the FP64 kernel's walk with packed FP32 pairs and FP64 flushes every four x
// points: 0.62.
// SINGLE (boxes with Nz < ngd + 6, whose runs can wrap onto a quad twice): the points of the
// run alone and each product added in FP64, as these boxes were always summed.
constexpr int IQ_MAX = (FS_NGD_MAX + 6) / 4;  // quads a z run of ngd points can touch
struct InterpQuad {
  float4 wg[IQ_MAX], wd[IQ_MAX], wr[IQ_MAX];  // g, gd, r of the quad's four points (0 off the run)
  int zq[IQ_MAX];                              // the quad's first z index
};
struct XY32 {
  float gg, dd, rx, ry;  // gx gy, gdx gdy, rx, ry of one (i, j) of the x-y stencil
};
__host__ __device__ constexpr size_t interp_q_xy_offset() { return (sizeof(InterpQuad) + 15) / 16 * 16; }
__host__ __device__ constexpr size_t interp_q_warp_bytes(int ngd) {
  return (interp_q_xy_offset() + (size_t)ngd * ngd * (sizeof(XY32) + sizeof(long long)) + 31) / 32 * 32;
}

template <int WPB, int SPLIT, bool SINGLE>
__global__ void __launch_bounds__(32 * WPB) k_interp_q(const float *__restrict__ u, const float4 *__restrict__ rec,
                                                       int np, FcmConsts c, double *__restrict__ V,
                                                       double *__restrict__ W) {
  FS_AFTER_PREVIOUS();
  extern __shared__ __align__(32) unsigned char interp_smem[];
  const int lane = threadIdx.x & 31, wl = threadIdx.x >> 5;
  const int slot = (blockIdx.x * WPB + wl) / SPLIT, ws = wl % SPLIT;
  const bool on = slot < np;  // warp-uniform
  const int ngd = c.ngd, n2 = ngd * ngd, Nz = c.N[2];
  // the warps of one bead share its tables, each filling a part
  unsigned char *base = interp_smem + (size_t)(wl / SPLIT) * interp_q_warp_bytes(ngd);
  InterpQuad &q = *reinterpret_cast<InterpQuad *>(base);
  XY32 *xy = reinterpret_cast<XY32 *>(base + interp_q_xy_offset());
  long long *off = reinterpret_cast<long long *>(xy + n2);
  double acc[6] = {0, 0, 0, 0, 0, 0};  // V, W
  int b = 0, nq = 1, zs = 0;
  if (on) {
    const float4 *rw = rec + (size_t)slot * spread_rec_len(ngd);
    const float4 hd = __ldg(rw);
    const int sx = __float_as_int(hd.x), sy = __float_as_int(hd.y);
    zs = __float_as_int(hd.z);
    b = __float_as_int(hd.w);
    nq = ((zs & 3) + ngd + 3) >> 2;
    if (lane < nq && ws == 0) {
      int z0 = (zs & ~3) + 4 * lane;
      if (z0 >= Nz) z0 -= Nz;
      float w[3][4];
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        const int k = 4 * lane + t - (zs & 3);
        const float4 wz = k >= 0 && k < ngd ? __ldg(rw + 3 + 2 * ngd + k) : make_float4(0.f, 0.f, 0.f, 0.f);
        w[0][t] = wz.x;
        w[1][t] = wz.y;
        w[2][t] = wz.z;
      }
      q.wg[lane] = make_float4(w[0][0], w[0][1], w[0][2], w[0][3]);
      q.wd[lane] = make_float4(w[1][0], w[1][1], w[1][2], w[1][3]);
      q.wr[lane] = make_float4(w[2][0], w[2][1], w[2][2], w[2][3]);
      q.zq[lane] = z0;
    }
    for (int ij = lane + 32 * ws; ij < n2; ij += 32 * SPLIT) {
      const int i = ij / ngd, j = ij - i * ngd;
      const float4 wx = __ldg(rw + 3 + i), wy = __ldg(rw + 3 + ngd + j);
      XY32 e;
      e.gg = wx.x * wy.x;
      e.dd = wx.y * wy.y;
      e.rx = wx.z;
      e.ry = wy.z;
      xy[ij] = e;
      const int ix = sx + i, iy = sy + j;
      off[ij] = ((long long)(ix >= c.N[0] ? ix - c.N[0] : ix) * c.N[1] + (iy >= c.N[1] ? iy - c.N[1] : iy)) * Nz;
    }
  }
  if constexpr (SPLIT > 1)
    __syncthreads();
  else
    __syncwarp();
  if (on) {
    const size_t N = (size_t)c.N[0] * c.N[1] * Nz;
    const float *ux = u, *uy = u + N, *uz = u + 2 * N;
    // slot sl = ij * nq + qi; a step advances (ij, qi) by (step / nq, step % nq)
    constexpr int STEP = 32 * SPLIT;
    const int nslot = n2 * nq, dij = STEP / nq, dq = STEP - dij * nq;
    const int first = lane + 32 * ws;
    int ij = first / nq, qi = first - ij * nq;
    for (int sl = first; sl < nslot; sl += STEP) {
      const XY32 e = xy[ij];
      const long long m = off[ij] + q.zq[qi];
      const float4 a0 = __ldg(reinterpret_cast<const float4 *>(ux + m));
      const float4 a1 = __ldg(reinterpret_cast<const float4 *>(uy + m));
      const float4 a2 = __ldg(reinterpret_cast<const float4 *>(uz + m));
      const float4 g = q.wg[qi], gd = q.wd[qi], r = q.wr[qi];
      if constexpr (SINGLE) {
        const int k0 = 4 * qi - (zs & 3);  // stencil index of the quad's first point
        auto add = [&](int k, float x0, float x1, float x2, float gz, float gdz, float zz) {
          if (k < 0 || k >= ngd) return;
          const float temp = e.gg * gz;  // (gx gy) gz, the reference's order
          const float tempd = e.dd * gdz;
          acc[0] += (double)(x0 * temp);
          acc[1] += (double)(x1 * temp);
          acc[2] += (double)(x2 * temp);
          acc[3] += (double)((x2 * e.ry - x1 * zz) * tempd);
          acc[4] += (double)((x0 * zz - x2 * e.rx) * tempd);
          acc[5] += (double)((x1 * e.rx - x0 * e.ry) * tempd);
        };
        add(k0, a0.x, a1.x, a2.x, g.x, gd.x, r.x);
        add(k0 + 1, a0.y, a1.y, a2.y, g.y, gd.y, r.y);
        add(k0 + 2, a0.z, a1.z, a2.z, g.z, gd.z, r.z);
        add(k0 + 3, a0.w, a1.w, a2.w, g.w, gd.w, r.w);
      } else {
        float p0 = 0.f, p1 = 0.f, p2 = 0.f, p3 = 0.f, p4 = 0.f, p5 = 0.f;
        auto add = [&](float x0, float x1, float x2, float gz, float gdz, float zz) {
          const float temp = e.gg * gz;  // (gx gy) gz, the reference's order
          const float tempd = e.dd * gdz;
          p0 += x0 * temp;
          p1 += x1 * temp;
          p2 += x2 * temp;
          p3 += (x2 * e.ry - x1 * zz) * tempd;
          p4 += (x0 * zz - x2 * e.rx) * tempd;
          p5 += (x1 * e.rx - x0 * e.ry) * tempd;
        };
        add(a0.x, a1.x, a2.x, g.x, gd.x, r.x);
        add(a0.y, a1.y, a2.y, g.y, gd.y, r.y);
        add(a0.z, a1.z, a2.z, g.z, gd.z, r.z);
        add(a0.w, a1.w, a2.w, g.w, gd.w, r.w);
        acc[0] += (double)p0;
        acc[1] += (double)p1;
        acc[2] += (double)p2;
        acc[3] += (double)p3;
        acc[4] += (double)p4;
        acc[5] += (double)p5;
      }
      qi += dq;
      ij += dij;
      if (qi >= nq) {
        qi -= nq;
        ++ij;
      }
    }
  }
  interp_finish<WPB, SPLIT>(acc, on, b, c.dx, V, W);
}

// Launched plainly: its many CTAs (885,000 at 512 x 384 x 384) each do one load and one store a
// thread, and the wait of programmatic serialization in all of them costs more than it saves: an
// FP32 flow solve with its two conversions 3.68 ms plain, 4.16 with it; at 64^3 39 and 38 us.
template <typename A, typename B>
__global__ void k_convert(const A *__restrict__ in, B *__restrict__ out, size_t n) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = (B)in[i];
}

__global__ void k_friction(const double *__restrict__ F, const double *__restrict__ T, double *__restrict__ V,
                           double *__restrict__ W, int n3, double a1, double a2) {
  FS_AFTER_PREVIOUS();
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n3) {
    V[i] = a1 * F[i];
    W[i] = a2 * T[i];
  }
}

FcmConsts make_consts(const fs_ctx *c) {
  FcmConsts k;
  k.N[0] = c->nx;
  k.N[1] = c->ny;
  k.N[2] = c->nz;
  k.gnx = c->slab_nx > 0 ? c->slab_nx : c->nx;
  k.x0 = c->slab_nx > 0 ? c->slab_x0 : 0;
  k.ngd = c->p.ngd;
  k.ngdh = c->p.ngd / 2;
  for (int d = 0; d < 3; ++d) k.nbin[d] = c->nbin[d];
  k.dx = c->p.dx;
  const double PI = FS_PI;
  k.sigmadipsq = c->p.sigma_dip * c->p.sigma_dip;
  k.anormdip = 1.0 / sqrt(2.0 * PI * k.sigmadipsq);
  k.anormdip2 = 2.0 * k.sigmadipsq;
  const double sigmasq = c->p.sigma * c->p.sigma;
  k.anorm = 1.0 / sqrt(2.0 * PI * sigmasq);
  k.anorm2 = 2.0 * sigmasq;
  return k;
}

fs_status ensure_plans(fs_ctx *c, int prec) {
  if (c->plan_ok[prec]) return FS_OK;
  int n[3] = {c->nx, c->ny, c->nz};
  size_t ws = 0;
  if (cufftCreate(&c->plan_fwd[prec]) != CUFFT_SUCCESS) return FS_ERR_CUFFT;
  if (cufftCreate(&c->plan_inv[prec]) != CUFFT_SUCCESS) return FS_ERR_CUFFT;
  cufftType tf = prec == FS_PREC_FP64 ? CUFFT_D2Z : CUFFT_R2C;
  cufftType ti = prec == FS_PREC_FP64 ? CUFFT_Z2D : CUFFT_C2R;
  if (cufftMakePlanMany(c->plan_fwd[prec], 3, n, NULL, 1, 0, NULL, 1, 0, tf, 3, &ws) != CUFFT_SUCCESS)
    return FS_ERR_CUFFT;
  c->bytes += ws;
  if (cufftMakePlanMany(c->plan_inv[prec], 3, n, NULL, 1, 0, NULL, 1, 0, ti, 3, &ws) != CUFFT_SUCCESS)
    return FS_ERR_CUFFT;
  c->bytes += ws;
  if (cufftSetStream(c->plan_fwd[prec], c->stream) != CUFFT_SUCCESS) return FS_ERR_CUFFT;
  if (cufftSetStream(c->plan_inv[prec], c->stream) != CUFFT_SUCCESS) return FS_ERR_CUFFT;
  c->plan_ok[prec] = true;
  return FS_OK;
}

// the grid runs this library's transforms (fs_lines.cuh) at this precision; else cuFFT
bool own_transform(const fs_ctx *c, int prec) {
  return c->line_tw[prec][0] && (prec == FS_PREC_FP64 || c->tune_fft32 == 0);
}

fs_status prepare_transform(fs_ctx *c, int prec) {
  if (prec == FS_PREC_FP64) return lines_prepare64(c);
  return fft32_preferred(c) ? FS_OK : lines_prepare32(c);
}

template <typename R>
fs_status flow_solve_t(fs_ctx *c) {
  const int prec = sizeof(R) == 8 ? FS_PREC_FP64 : FS_PREC_FP32;
  if (own_transform(c, prec)) {
    FS_TRY(prepare_transform(c, prec));
    if (prec == FS_PREC_FP64) return lines_flow_solve64(c);
    return fft32_preferred(c) ? fft32_flow_solve(c) : lines_flow_solve32(c);
  }
  FS_TRY(ensure_plans(c, prec));
  cufftResult r;
  {
    ProfScope ps(c, FS_STAGE_FFT_FWD);
    if (prec == FS_PREC_FP64)
      r = cufftExecD2Z(c->plan_fwd[prec], (cufftDoubleReal *)c->grid_real, (cufftDoubleComplex *)c->grid_cplx);
    else
      r = cufftExecR2C(c->plan_fwd[prec], (cufftReal *)c->grid_real, (cufftComplex *)c->grid_cplx);
  }
  if (r != CUFFT_SUCCESS) return FS_ERR_CUFFT;
  const double TwoPI = 2. * FS_PI;
  const R ffx = (R)(TwoPI / (c->nx * c->p.dx)), ffy = (R)(TwoPI / (c->ny * c->p.dx)),
          ffz = (R)(TwoPI / (c->nz * c->p.dx));
  const R total = (R)((double)c->nx * (double)c->ny * (double)c->nz);
  typedef typename Cplx<R>::T C;
  C *fh = (C *)c->grid_cplx;
  {
    ProfScope ps(c, FS_STAGE_PROJECT);
    fs_launch(k_project<R>, fs_blocks((long long)c->NH, 256), 256, 0, c->stream, fh, c->NH, c->nx, c->ny, c->nz,
              c->nzh, ffx, ffy, ffz, total);
    FS_LAUNCH_CHECK();
    dim3 gp(fs_blocks((long long)c->nx * c->ny, 256), 2);
    fs_launch(k_project_planes<R>, gp, 256, 0, c->stream, fh, c->NH, c->nx, c->ny, c->nz, c->nzh, ffx, ffy, ffz,
              total);
    FS_LAUNCH_CHECK();
  }
  {
    ProfScope ps(c, FS_STAGE_FFT_INV);
    if (prec == FS_PREC_FP64)
      r = cufftExecZ2D(c->plan_inv[prec], (cufftDoubleComplex *)c->grid_cplx, (cufftDoubleReal *)c->grid_real);
    else
      r = cufftExecC2R(c->plan_inv[prec], (cufftComplex *)c->grid_cplx, (cufftReal *)c->grid_real);
  }
  if (r != CUFFT_SUCCESS) return FS_ERR_CUFFT;
  return FS_OK;
}

// bins the beads of Y, sorts them and writes their records (F, T: null where only the
// weights are read)
template <typename R>
fs_status bin_t(fs_ctx *c, const FcmConsts &k, const double *Y, const double *F, const double *T, int np) {
  FS_TRY(fs_sort_run(&c->bins, BinKey{Y, k, c->bead_sw}, np, c->stream));
  if (np <= 0) return FS_OK;
  if (sizeof(R) == 4)
    fs_launch(k_spread_records32, fs_blocks((long long)np * spread_rec_len(k.ngd), 256), 256, 0, c->stream, Y, F, T,
              c->bins.sorted, c->bead_sw, np, k, (float4 *)c->bead_rec);
  else
    fs_launch(k_records64, fs_blocks((long long)np * rec64_len(k.ngd), 256), 256, 0, c->stream, Y, F, T,
              c->bins.sorted, c->bead_sw, np, k, (double4 *)c->bead_rec);
  FS_LAUNCH_CHECK();
  return FS_OK;
}

// binning and the spread of the force grid into c->grid_real (R precision)
template <typename R>
fs_status spread_t(fs_ctx *c, const FcmConsts &k, const double *Y, const double *F, const double *T, int np) {
  FS_TRY(bin_t<R>(c, k, Y, F, T, np));
  ProfScope pk(c, FS_STAGE_K_SPREAD);
  const int ch = c->tune_spread_chunk, cx = c->tune_spread_cols;
  if (sizeof(R) == 4) {
    const float4 *rec = (const float4 *)c->bead_rec;
    // beads whose stencil reaches a tile, if they lie evenly
    const double e = (k.ngd + FS_TILE - 1) / (double)FS_TILE, reach = (double)np / c->nbins * (e * e * e);
    const int per_sm = c->nbins / c->num_sms;
    const bool quarter = per_sm < 1, sparse = (reach <= 12 && per_sm >= 10) || (reach <= 28 && per_sm >= 40),
               whole = reach <= (per_sm >= 10 ? 48 : 20) && per_sm >= 2;
#define FS_SPREAD32_LAUNCH1(CHV, CXV, NWV, PV)                                                                    \
  {                                                                                                               \
    constexpr size_t bytes = sizeof(SpreadStage32<CHV>);                                                          \
    if (bytes > 48 * 1024)                                                                                        \
      FS_CUDA(cudaFuncSetAttribute((const void *)k_spread32<CHV, CXV, NWV, PV>,                                   \
                                   cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));                     \
    fs_launch(k_spread32<CHV, CXV, NWV, PV>, 16 / (NWV * PV) * c->nbins, 32 * NWV, bytes, c->stream, \
              c->bins.start, rec, k, (float *)c->grid_real); \
  }
#define FS_SPREAD32_LAUNCH(CHV, CXV)                      \
  {                                                       \
    if (quarter) FS_SPREAD32_LAUNCH1(CHV, CXV, 4, 1)      \
    else if (sparse) FS_SPREAD32_LAUNCH1(CHV, CXV, 4, 4)  \
    else if (whole) FS_SPREAD32_LAUNCH1(CHV, CXV, 8, 2)   \
    else FS_SPREAD32_LAUNCH1(CHV, CXV, 8, 1)              \
  }
    if (ch == 32 && cx == 2) FS_SPREAD32_LAUNCH(32, 2)
    else if (ch == 32 && cx == 8) FS_SPREAD32_LAUNCH(32, 8)
    else if (ch == 32) FS_SPREAD32_LAUNCH(32, 4)
    else if (cx == 2) FS_SPREAD32_LAUNCH(64, 2)
    else if (cx == 8) FS_SPREAD32_LAUNCH(64, 8)
    else FS_SPREAD32_LAUNCH(64, 4)
#undef FS_SPREAD32_LAUNCH
#undef FS_SPREAD32_LAUNCH1
  } else {
    const double4 *rec = (const double4 *)c->bead_rec;
    double *f = (double *)c->grid_real;
    // half tiles, or quarter tiles where the half tiles would not fill the SMs three times
    // (quarter / half, us, tiles reached by 10 and 27 beads: 64 tiles 12 / 15, 14 / 17; 216 19 / 16, 23 /
    // 25; 343 23 / 23, 30 / 32; 512 30 / 28, 39 / 39; 4,096 181 / 161, 247 / 229)
    if (2 * c->nbins < 3 * c->num_sms)
      fs_launch(k_spread64<4>, 4 * c->nbins, FS_SPREAD64_THREADS, sizeof(SpreadStage64<4>), c->stream, c->bins.start,
                rec, k, f);
    else
      fs_launch(k_spread64<8>, 2 * c->nbins, FS_SPREAD64_THREADS, sizeof(SpreadStage64<8>), c->stream, c->bins.start,
                rec, k, f);
  }
  FS_LAUNCH_CHECK();
  return FS_OK;
}

// Warps a bead is split over. FP64 (16 warps an SM): four up to 4 beads per SM, two up to 8
// (four / two / one warp, 256^3, 12 points: 592 beads 21 / 23 / 23 us, 740 29 / 25 / 25, 1,000 34 / 27 /
// 28, 1,480 44 / 40 / 34). FP32, short stencils (27 warps an SM): four up to 6.75, two up to 13.5 (740
// beads 17 / 21 / 27, 1,000 20 / 23 / 29, 1,480 27 / 25 / 32, 2,000 29 / 29 / 34, 2,960 37 / 39 / 38). From 15
// points on a bead's FP32 tables, which its warps share, leave an SM less than 40 warps of whole
// beads, so beads are always split (256^3, 20 points: 1,480 beads 55 / 60 / 101, 6,000 104 / 117 / 216,
// 12,000 179 / 184 / 277, 100,000 1,305 / 1,272 / 1,512).
int interp_split(const fs_ctx *c, int prec, int np) {
  if (prec == FS_PREC_FP32 && c->p.ngd >= 15) return np <= 40 * c->num_sms ? 4 : 2;
  const int warps = (prec == FS_PREC_FP32 ? 27 : 16) * c->num_sms;
  return 4 * np <= warps ? 4 : 2 * np <= warps ? 2 : 1;
}
bool interp_single(const fs_ctx *c) { return c->nz < c->p.ngd + 6; }  // FP32: k_interp_q's SINGLE

// interpolation of U, Omega from the velocity grid in c->grid_real (R precision); the
// beads must have been binned (bin_t) at this precision. given: the grid is a caller's
template <typename R>
fs_status interp_t(fs_ctx *c, const FcmConsts &k, double *V, double *W, int np, bool given) {
  if (np <= 0) return FS_OK;
  ProfScope ps(c, FS_STAGE_INTERP);
  ProfScope pk(c, FS_STAGE_K_INTERP);
  const int split = interp_split(c, sizeof(R) == 4 ? FS_PREC_FP32 : FS_PREC_FP64, np);
  const size_t wb = sizeof(R) == 4 ? interp_q_warp_bytes(k.ngd) : 0;  // dynamic shared memory per bead of a CTA
  // the forms for single points (FP32) and with MASK (FP64) exist with four warps
  const bool other = sizeof(R) == 4 ? interp_single(c) : given;
  const int wpb = split > 1 || other ? 4 : (c->tune_interp_wpb == 16 && 16 * wb > FS_SMEM_MAX) ? 8 : c->tune_interp_wpb;
#define FS_INTERP_LAUNCH(WPB, SPLIT, OTHER)                                                                     \
  if constexpr (sizeof(R) == 4)                                                                                 \
    fs_launch(k_interp_q<WPB, SPLIT, OTHER>, fs_blocks(np, WPB / SPLIT), 32 * WPB, WPB / SPLIT * wb, c->stream, \
              (const float *)c->grid_real, (const float4 *)c->bead_rec, np, k, V, W);                           \
  else                                                                                                          \
    fs_launch(k_interp64<WPB, SPLIT, OTHER>, fs_blocks(np, WPB / SPLIT), 32 * WPB, 0, c->stream,                \
              (const double *)c->grid_real, (const double4 *)c->bead_rec, np, k, V, W)
  if (other && split == 4) {
    FS_INTERP_LAUNCH(4, 4, true);
  } else if (other && split == 2) {
    FS_INTERP_LAUNCH(4, 2, true);
  } else if (other) {
    FS_INTERP_LAUNCH(4, 1, true);
  } else if (split == 4) {
    FS_INTERP_LAUNCH(4, 4, false);
  } else if (split == 2) {
    FS_INTERP_LAUNCH(4, 2, false);
  } else if (wpb == 4) {
    FS_INTERP_LAUNCH(4, 1, false);
  } else if (wpb == 16) {
    FS_INTERP_LAUNCH(16, 1, false);
  } else {
    FS_INTERP_LAUNCH(8, 1, false);
  }
#undef FS_INTERP_LAUNCH
  FS_LAUNCH_CHECK();
  return FS_OK;
}

template <typename R>
fs_status mobility_t(fs_ctx *c, const double *Y, const double *F, const double *T, double *V, double *W, int np) {
  FcmConsts k = make_consts(c);
  {
    ProfScope ps(c, FS_STAGE_SPREAD);
    FS_TRY(spread_t<R>(c, k, Y, F, T, np));
  }
  FS_TRY(flow_solve_t<R>(c));
  FS_TRY(interp_t<R>(c, k, V, W, np, false));
  c->last_grid_prec = sizeof(R) == 8 ? FS_PREC_FP64 : FS_PREC_FP32;
  return FS_OK;
}

}  // namespace

fs_status fcm_init(fs_ctx *c) {
  c->nx = c->p.npts_x;
  c->ny = c->p.npts_y;
  c->nz = c->p.npts_z;
  c->nzh = c->nz / 2 + 1;
  c->N = (size_t)c->nx * c->ny * c->nz;
  c->NH = (size_t)c->nx * c->ny * c->nzh;
  for (int d = 0; d < 3; ++d) c->nbin[d] = (d == 0 ? c->nx : d == 1 ? c->ny : c->nz) / FS_TILE;
  c->nbins = c->nbin[0] * c->nbin[1] * c->nbin[2];
  c->last_grid_prec = -1;
  FS_CUDA(cudaMalloc(&c->grid_real, sizeof(double) * 3 * c->N));
  // the line transforms round their rows of nz / 2 + 1 values up to even
  const size_t ncplx = 3 * (size_t)c->nx * c->ny * ((c->nzh + 1) & ~1);
  FS_CUDA(cudaMalloc(&c->grid_cplx, sizeof(double2) * ncplx));
  c->bytes += sizeof(double) * 3 * c->N + sizeof(double2) * ncplx;
  FS_TRY(fs_sort_alloc(&c->bins, c->nbins, c->max_beads, &c->bytes));
  FS_TRY(fs_sort_prepare<BinKey>());
  FS_CUDA(cudaMalloc(&c->bead_sw, sizeof(int) * 3 * (size_t)(c->max_beads > 0 ? c->max_beads : 1)));
  c->bytes += sizeof(int) * 3 * (size_t)c->max_beads;
  {
    // the beads' records of either precision (the FP64 ones are the larger)
    const size_t bytes = sizeof(double4) * (size_t)(c->max_beads > 0 ? c->max_beads : 1) * rec64_len(c->p.ngd);
    FS_CUDA(cudaMalloc(&c->bead_rec, bytes));
    c->bytes += bytes;
  }
  // the attributes are per kernel, shared by every context: set for the largest ngd
  // (capped at what a CTA may ask for; larger launches take 8 warps per CTA)
  auto smem = [](const void *fn, size_t bytes) {
    return cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)(bytes < (size_t)FS_SMEM_MAX ? bytes : (size_t)FS_SMEM_MAX));
  };
  FS_CUDA(smem((const void *)k_spread64<4>, sizeof(SpreadStage64<4>)));
  FS_CUDA(smem((const void *)k_spread64<8>, sizeof(SpreadStage64<8>)));
  const size_t wq = interp_q_warp_bytes(FS_NGD_MAX);
  FS_CUDA(smem((const void *)k_interp_q<4, 1, false>, 4 * wq));
  FS_CUDA(smem((const void *)k_interp_q<4, 1, true>, 4 * wq));
  FS_CUDA(smem((const void *)k_interp_q<8, 1, false>, 8 * wq));
  FS_CUDA(smem((const void *)k_interp_q<16, 1, false>, 16 * wq));
  c->tune_spread_chunk = 32;
  c->tune_spread_cols = 2;  // 2 x 16 x 8 blocks: fs_autotune's choice at 384^3 and 512^3
  c->tune_interp_wpb = 4;  // the fastest at 256^3 and 512^3 in both precisions (512^3 FP64 before six x steps: 833, 873, 911 us)
  c->tune_fft32 = 0;
  if (lines_supported(c)) {
    FS_TRY(lines_init64(c));
    FS_TRY(lines_init32(c));
  }
  return fft32_init(c);
}

bool lines_supported(const fs_ctx *c) { return line_length(c->nx) && line_length(c->ny) && line_length(c->nz); }

void fcm_free(fs_ctx *c) {
  for (int p = 0; p < 2; ++p)
    if (c->plan_ok[p]) {
      cufftDestroy(c->plan_fwd[p]);
      cufftDestroy(c->plan_inv[p]);
      c->plan_ok[p] = false;
    }
  cudaFree(c->grid_real);
  cudaFree(c->grid_cplx);
  c->grid_real = c->grid_cplx = nullptr;
  fft32_free(c);
  for (int p = 0; p < 2; ++p) {
    cudaFree(c->line_tw[p][0]);  // the three axes' tables are one allocation
    for (int a = 0; a < 3; ++a) c->line_tw[p][a] = nullptr;
  }
  fs_sort_free(&c->bins);
  cudaFree(c->bead_sw);
  c->bead_sw = nullptr;
  cudaFree(c->bead_rec);
  c->bead_rec = nullptr;
}

bool fcm_interp_wpb_used(const fs_ctx *c, int np) {
  return interp_split(c, c->precision, np) == 1 && !(c->precision == FS_PREC_FP32 && interp_single(c));
}

fs_status fcm_set_stream(fs_ctx *c, cudaStream_t st) {
  const int prec = c->precision;
  if (own_transform(c, prec)) return prepare_transform(c, prec);  // no cuFFT plan
  FS_TRY(ensure_plans(c, prec));
  if (cufftSetStream(c->plan_fwd[prec], st) != CUFFT_SUCCESS) return FS_ERR_CUFFT;
  if (cufftSetStream(c->plan_inv[prec], st) != CUFFT_SUCCESS) return FS_ERR_CUFFT;
  return FS_OK;
}

fs_status fcm_mobility(fs_ctx *c, const double *Y, const double *F, const double *T, double *V, double *W, int np) {
  if (c->precision == FS_PREC_FP32) return mobility_t<float>(c, Y, F, T, V, W, np);
  return mobility_t<double>(c, Y, F, T, V, W, np);
}

fs_status fcm_friction(fs_ctx *c, const double *F, const double *T, double *V, double *W, int np) {
  const double PI = FS_PI, a = c->p.a, mu = c->p.mu;
  const double a1 = 1. / (6 * PI * a * mu);
  const double a2 = 1. / (8 * PI * a * a * a * mu);
  if (np > 0) {
    ProfScope ps(c, FS_STAGE_FRICTION);
    fs_launch(k_friction, fs_blocks(3 * np, 256), 256, 0, c->stream, F, T, V, W, 3 * np, a1, a2);
    FS_LAUNCH_CHECK();
  }
  return FS_OK;
}

fs_status fcm_interpolate_only(fs_ctx *c, const double *u, const double *Y, int np, double *V, double *W) {
  FcmConsts k = make_consts(c);
  const size_t n = 3 * c->N;
  FS_TRY(c->precision == FS_PREC_FP32 ? bin_t<float>(c, k, Y, nullptr, nullptr, np)
                                      : bin_t<double>(c, k, Y, nullptr, nullptr, np));
  if (c->precision == FS_PREC_FP32) {
    k_convert<double, float><<<fs_blocks((long long)n, 256), 256, 0, c->stream>>>(u, (float *)c->grid_real, n);
    FS_LAUNCH_CHECK();
    FS_TRY(interp_t<float>(c, k, V, W, np, true));
  } else {
    FS_CUDA(cudaMemcpyAsync(c->grid_real, u, sizeof(double) * n, cudaMemcpyDeviceToDevice, c->stream));
    FS_TRY(interp_t<double>(c, k, V, W, np, true));
  }
  c->last_grid_prec = -1;
  return FS_OK;
}

fs_status fcm_spread_only(fs_ctx *c, const double *Y, const double *F, const double *T, int np, double *f) {
  FcmConsts k = make_consts(c);
  const size_t n = 3 * c->N;
  if (c->precision == FS_PREC_FP32) {
    FS_TRY(spread_t<float>(c, k, Y, F, T, np));
    k_convert<float, double><<<fs_blocks((long long)n, 256), 256, 0, c->stream>>>((const float *)c->grid_real, f, n);
    FS_LAUNCH_CHECK();
  } else {
    FS_TRY(spread_t<double>(c, k, Y, F, T, np));
    FS_CUDA(cudaMemcpyAsync(f, c->grid_real, sizeof(double) * n, cudaMemcpyDeviceToDevice, c->stream));
  }
  c->last_grid_prec = -1;
  return FS_OK;
}

fs_status fcm_flow_solve_only(fs_ctx *c, const double *f, double *u) {
  const size_t n = 3 * c->N;
  if (c->precision == FS_PREC_FP32) {
    // FP32 chain: f rounded to float, solved, widened back
    k_convert<double, float><<<fs_blocks((long long)n, 256), 256, 0, c->stream>>>(f, (float *)c->grid_real, n);
    FS_LAUNCH_CHECK();
    FS_TRY(flow_solve_t<float>(c));
    k_convert<float, double><<<fs_blocks((long long)n, 256), 256, 0, c->stream>>>((const float *)c->grid_real, u, n);
    FS_LAUNCH_CHECK();
    c->last_grid_prec = FS_PREC_FP32;
    return FS_OK;
  }
  FS_CUDA(cudaMemcpyAsync(c->grid_real, f, sizeof(double) * n, cudaMemcpyDeviceToDevice, c->stream));
  FS_TRY(flow_solve_t<double>(c));
  FS_CUDA(cudaMemcpyAsync(u, c->grid_real, sizeof(double) * n, cudaMemcpyDeviceToDevice, c->stream));
  c->last_grid_prec = FS_PREC_FP64;
  return FS_OK;
}
