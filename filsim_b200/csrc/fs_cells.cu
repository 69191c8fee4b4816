// fs_cells.cu -- cell linked list and collision barrier on sm_100a.
//
// LinkedList::link (CollisionBarrierFilament.cpp:370-433) head-inserts beads
// into cells, so each cell's list runs from the largest bead id down. A
// counting sort by (cell, id) produces the same lists: head[c] is the last
// bead of the cell's segment and list[b] the one before it. k_cell_lists
// writes head/list exactly as the reference holds them.
//
// LinkedList::apply_collision_barrier (:24-271) walks cells in order, and for
// each bead i the rest of its own cell and the 13 half-shell neighbour cells,
// adding the pair force to i and subtracting it from j. k_barrier gives each
// bead a group of lanes that collects every interaction it takes part in (as i
// and as j), orders them as the reference visits them (cell of i, list
// position of i, neighbour slot, list position of j) and folds them in that order, so each bead's total is bit-identical to the
// reference's sequential accumulation. Pair arithmetic uses explicit
// round-to-nearest intrinsics (no FMA contraction) to match the reference's
// x86-64 doubles.
#include "fs_internal.cuh"
#include "fs_events.cuh"
#include "fs_sort.cuh"

fs_status fs_exclusive_scan(const int *in, int *out, int n, int *block_sums, cudaStream_t st);

namespace {

struct BarrierConsts {
  double L[3];
  int M[3];
  double chiRnm2, den, cap, cap2, fs;
  int nt, initial_friction_steps;
  int mode, np;  // pair filter (FS_BARRIER_*) and bead count
};

// bulkmap neighbour offsets (CollisionBarrierFilament.cpp:326-338) of slots 1..13, after slot
// 0 (the cell itself); two bits per slot and dimension hold the offset plus one
struct NbPack {
  unsigned d[3];
};
__host__ __device__ constexpr NbPack nb_pack() {
  const int off[14][3] = {{0, 0, 0},  {1, 0, 0},  {1, 1, 0},  {0, 1, 0}, {-1, 1, 0}, {1, 0, -1}, {1, 1, -1},
                          {0, 1, -1}, {-1, 1, -1}, {1, 0, 1}, {1, 1, 1}, {0, 1, 1},  {-1, 1, 1}, {0, 0, 1}};
  NbPack p = {{0, 0, 0}};
  for (int s = 0; s < 14; ++s)
    for (int d = 0; d < 3; ++d) p.d[d] |= (unsigned)(off[s][d] + 1) << (2 * s);
  return p;
}
__device__ __forceinline__ int nb_off(int slot, int d) {
  constexpr NbPack p = nb_pack();
  const unsigned w = d == 0 ? p.d[0] : d == 1 ? p.d[1] : p.d[2];
  return (int)((w >> (2 * slot)) & 3u) - 1;
}

__device__ __forceinline__ int icell(const int *M, int x, int y, int z) {
  int xx = (x + M[0]) % M[0], yy = (y + M[1]) % M[1], zz = (z + M[2]) % M[2];
  return xx + yy * M[0] + zz * M[0] * M[1];
}

__global__ void k_bulkmap(int Mx, int My, int Mz, int *__restrict__ map) {
  FS_AFTER_PREVIOUS();
  int c = blockIdx.x * blockDim.x + threadIdx.x;
  int M[3] = {Mx, My, Mz};
  if (c >= Mx * My * Mz) return;
  int x = c % Mx, y = (c / Mx) % My, z = c / (Mx * My);
  for (int nb = 0; nb < 13; ++nb) map[13 * c + nb] = icell(M, x + nb_off(nb + 1, 0), y + nb_off(nb + 1, 1), z + nb_off(nb + 1, 2));
}

// cell of an unwrapped position (CollisionBarrierFilament.cpp:387-409)
struct CellKey {
  const double *Xs;
  BarrierConsts k;
  __device__ int operator()(int b) const {
    const int large_number = 100000;
    int ci[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const double x = Xs[3 * b + d];
      const int w = __double2int_rz(__dadd_rn(__ddiv_rn(x, k.L[d]), (double)large_number)) - large_number;
      const double xr = __dsub_rn(x, __dmul_rn(k.L[d], (double)w));
      int cc = __double2int_rz(__dmul_rn(__ddiv_rn(xr, k.L[d]), (double)k.M[d]));
      cc = cc >= k.M[d] ? k.M[d] - 1 : cc;
      cc = cc < 0 ? 0 : cc;
      ci[d] = cc;
    }
    return ci[0] + ci[1] * k.M[0] + ci[2] * k.M[0] * k.M[1];
  }
};

__global__ void k_cell_lists(const int *__restrict__ start, const int *__restrict__ sorted, int ncell,
                             int *__restrict__ head, int *__restrict__ list, int *__restrict__ rank_desc,
                             int *__restrict__ flags) {
  FS_AFTER_PREVIOUS();
  int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= ncell) return;
  int s = start[c], e = start[c + 1];
  head[c] = (e > s) ? sorted[e - 1] : -1;
  if (e - s >= 4096) atomicOr(&flags[FLAG_CAPACITY], 1);
  for (int p = s; p < e; ++p) {
    int b = sorted[p];
    list[b] = (p > s) ? sorted[p - 1] : -1;
    rank_desc[b] = e - 1 - p;
  }
}

// minimum-image separation of a pair and its square as the reference computes them
// (CollisionBarrierFilament.cpp:80-100). Below 0.49 L the quotient plus one half lies within
// (0, 1), so its floor is 0 and the separation is x itself: the division is left out.
__device__ __forceinline__ double pair_dist(const BarrierConsts &k, const double *Yi, const double *Yj, double *d) {
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const double x = __dsub_rn(Yi[a], Yj[a]);
    d[a] = x;
    if (!(fabs(x) < 0.49 * k.L[a])) {
      const double s = floor(__dadd_rn(__ddiv_rn(x, k.L[a]), 0.5));
      d[a] = __dsub_rn(x, __dmul_rn(k.L[a], s));
    }
  }
  return __dadd_rn(__dadd_rn(__dmul_rn(d[0], d[0]), __dmul_rn(d[1], d[1])), __dmul_rn(d[2], d[2]));
}

// force of a pair inside the barrier range (CollisionBarrierFilament.cpp:101-149)
__device__ __forceinline__ void pair_force(const BarrierConsts &k, double *d, double rijsq, double *f) {
  if (rijsq < k.cap2) {
    double rij = __dsqrt_rn(rijsq);
#pragma unroll
    for (int a = 0; a < 3; ++a) d[a] = __dmul_rn(__ddiv_rn(d[a], rij), k.cap);
    rijsq = k.cap2;
  }
  double prefac = __dsub_rn(k.chiRnm2, rijsq);
  prefac = __ddiv_rn(prefac, k.den);
  prefac = __dmul_rn(prefac, prefac);
  prefac = __dmul_rn(prefac, prefac);
  prefac = __dmul_rn(prefac, k.fs);
#pragma unroll
  for (int a = 0; a < 3; ++a) f[a] = __dmul_rn(prefac, d[a]);
}

__device__ __forceinline__ unsigned long long ev_key(int cell, int pos_i, int slot, int pos_j) {
  return ((((unsigned long long)cell * 4096ull + (unsigned long long)pos_i) * 16ull + (unsigned long long)slot) *
          4096ull) + (unsigned long long)pos_j;
}

// pairs the barrier skips: neighbours on one filament (CollisionBarrierFilament.cpp:57),
// and per mode swimmer-network pairs (apply_collision_barrier_not_swimmer, :474-477)
// or pairs with one of the last two beads (apply_collision_barrier_not_test_particles, :754)
__device__ __forceinline__ bool excluded(const BarrierConsts &k, const int *fil_id, const int *seg_id, int i, int j) {
  if (k.mode == FS_BARRIER_NOT_SWIMMER && ((fil_id[i] == 0) != (fil_id[j] == 0))) return true;
  if (k.mode == FS_BARRIER_NOT_TEST_PARTICLES && (i >= k.np - 2 || j >= k.np - 2)) return true;
  return (fil_id[j] == fil_id[i] && abs(seg_id[j] - seg_id[i]) == 1) && !(k.nt < k.initial_friction_steps);
}

// Pairs inside the range, b as i, in the reference's order: pairs == nullptr counts them per
// bead, else writes them from pair_off[b]
__global__ void __launch_bounds__(128) k_pairs(const double *__restrict__ Y, int np, BarrierConsts k,
                                               const int *__restrict__ cell_of, const int *__restrict__ start,
                                               const int *__restrict__ sorted, const int *__restrict__ rank_desc,
                                               const int *__restrict__ map, const int *__restrict__ fil_id,
                                               const int *__restrict__ seg_id, int *__restrict__ pair_count,
                                               const int *__restrict__ pair_off, int *__restrict__ pairs,
                                               int max_pairs) {
  FS_AFTER_PREVIOUS();
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= np) return;
  const int cb = cell_of[b], p_asc = start[cb + 1] - 1 - rank_desc[b];
  const double Yb[3] = {Y[3 * b], Y[3 * b + 1], Y[3 * b + 2]};
  int n = 0;
  double d[3];
  for (int slot = 0; slot < 14; ++slot) {
    const int cj = slot == 0 ? cb : map[13 * cb + slot - 1], qs = start[cj];
    const int qe = slot == 0 ? p_asc : start[cj + 1];  // own cell: ascending positions below b's
    for (int q = qe - 1; q >= qs; --q) {
      const int j = sorted[q];
      if (excluded(k, fil_id, seg_id, b, j)) continue;
      const double Yj[3] = {Y[3 * j], Y[3 * j + 1], Y[3 * j + 2]};
      if (!(pair_dist(k, Yb, Yj, d) < k.chiRnm2)) continue;
      if (pairs && pair_off[b] + n < max_pairs) {
        pairs[2 * (pair_off[b] + n)] = b;
        pairs[2 * (pair_off[b] + n) + 1] = j;
      }
      ++n;
    }
  }
  if (!pairs && pair_count) pair_count[b] = n;
}

// Barrier forces: G lanes per bead. Each lane walks some of the 28 cell ranges in which the
// bead takes part (as i: slots 0..13; as j: the cells whose slot is its own cell), the pairs
// in range are ordered by their keys, and the forces, a lane each, are folded in that order.
// Bound by the latency of cell -> range -> bead -> position, so by how many of a bead's cells
// are looked at together. With a lane for every range (G = 32) while the beads' warps fit the
// chip in about one wave, 8 lanes beyond: with the launch before it, 480 beads 15.5 us (8
// lanes 19.3), 3,840 beads 16.5 (20.8), 16,384 beads 24.0 (20.3), 131,072 beads 98 (62). A
// thread per bead over all ranges took 53 us for 480 beads and 89 us for 131,072.
constexpr int BARRIER_WIDE_PER_SM = 48;  // beads per SM
template <int G>
__global__ void __launch_bounds__(128) k_barrier(const double *__restrict__ Y, double *__restrict__ F, int np,
                                                 BarrierConsts k, const int *__restrict__ cell_of,
                                                 const int *__restrict__ start, const int *__restrict__ sorted,
                                                 const int *__restrict__ rank_desc, const int *__restrict__ fil_id,
                                                 const int *__restrict__ seg_id,
                                                 unsigned long long *__restrict__ min_bits, int *__restrict__ flags) {
  FS_AFTER_PREVIOUS();
  constexpr int BEADS = 128 / G;
  __shared__ unsigned long long s_key[BEADS][FS_MAX_EVENTS];
  __shared__ int s_other[BEADS][FS_MAX_EVENTS];  // the other bead; complemented where b is j
  __shared__ unsigned char s_ord[BEADS][FS_MAX_EVENTS];
  __shared__ int s_n[BEADS];
  const int l = threadIdx.x % G, w = threadIdx.x / G;
  const int b = blockIdx.x * BEADS + w;
  const bool live = b < np;
  if (l == 0) s_n[w] = 0;
  __syncwarp();
  double Yb[3] = {0.0, 0.0, 0.0}, d[3], local_min = 100000.0;
  if (live) {
    const int cb = cell_of[b], pb = rank_desc[b];
#pragma unroll
    for (int a = 0; a < 3; ++a) Yb[a] = Y[3 * b + a];
    const int cx = cb % k.M[0], cyz = cb / k.M[0], cy = cyz % k.M[1], cz = cyz / k.M[1];
    for (int s = l; s < 28; s += G) {
      const bool as_i = s < 14;
      const int slot = as_i ? s : s - 14, sg = as_i ? 1 : -1;
      int x = cx + sg * nb_off(slot, 0), y = cy + sg * nb_off(slot, 1), z = cz + sg * nb_off(slot, 2);
      x = x < 0 ? x + k.M[0] : x >= k.M[0] ? x - k.M[0] : x;
      y = y < 0 ? y + k.M[1] : y >= k.M[1] ? y - k.M[1] : y;
      z = z < 0 ? z + k.M[2] : z >= k.M[2] ? z - k.M[2] : z;
      const int cell = x + (y + z * k.M[1]) * k.M[0];
      int qs = start[cell], qe = start[cell + 1];
      const int e = qe;
      if (slot == 0) {  // own cell: b is i to the ascending positions below its own, j to those above
        if (as_i) qe = e - 1 - pb;
        else qs = e - pb;
      }
      for (int q = qs; q < qe; ++q) {
        const int j = sorted[q];
        if (excluded(k, fil_id, seg_id, b, j)) continue;
        const double Yj[3] = {Y[3 * j], Y[3 * j + 1], Y[3 * j + 2]};
        const double rsq = as_i ? pair_dist(k, Yb, Yj, d) : pair_dist(k, Yj, Yb, d);
        if (rsq < k.chiRnm2) {
          const int n = atomicAdd(&s_n[w], 1);
          if (n < FS_MAX_EVENTS) {
            s_key[w][n] = as_i ? ev_key(cb, pb, slot, e - 1 - q) : ev_key(cell, e - 1 - q, slot, pb);
            s_other[w][n] = as_i ? j : ~j;
          }
        }
        if (as_i && rsq < local_min) local_min = rsq;
      }
    }
  }
  __syncwarp();
  int n = s_n[w];
  if (n > FS_MAX_EVENTS) {
    if (l == 0) atomicOr(&flags[FLAG_CAPACITY], 1);
    n = FS_MAX_EVENTS;
  }
  for (int e = l; e < n; e += G) s_ord[w][event_place(s_key[w], n, e)] = (unsigned char)e;
  __syncwarp();
  // fold in order: adding -f equals subtracting f exactly
  double acc[3] = {0.0, 0.0, 0.0};
  for (int c0 = 0; __any_sync(0xffffffffu, c0 < n); c0 += G) {
    double f[3] = {0.0, 0.0, 0.0};
    if (c0 + l < n) {
      const int o = s_other[w][s_ord[w][c0 + l]], j = o < 0 ? ~o : o;
      const double Yj[3] = {Y[3 * j], Y[3 * j + 1], Y[3 * j + 2]};
      const double rsq = o >= 0 ? pair_dist(k, Yb, Yj, d) : pair_dist(k, Yj, Yb, d);
      pair_force(k, d, rsq, f);
      if (o < 0)
#pragma unroll
        for (int a = 0; a < 3; ++a) f[a] = -f[a];
    }
    for (int e = 0; __any_sync(0xffffffffu, c0 + e < n) && e < G; ++e) {
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        const double v = __shfl_sync(0xffffffffu, f[a], e, G);
        if (c0 + e < n) acc[a] = __dadd_rn(acc[a], v);
      }
    }
  }
  if (live && l < 3) {
    const double v = l == 0 ? acc[0] : l == 1 ? acc[1] : acc[2];
    F[3 * b + l] = __dadd_rn(F[3 * b + l], v);
  }
  // the minimum squared distance: an atomic per warp, and only below what is there already
  unsigned long long mb = fs_dbits(local_min);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const unsigned long long other = __shfl_xor_sync(0xffffffffu, mb, o);
    mb = other < mb ? other : mb;
  }
  if ((threadIdx.x & 31) == 0 && mb < *(volatile unsigned long long *)min_bits) atomicMin(min_bits, mb);
}

__global__ void k_pair_pos(const int *__restrict__ cell_of, const int *__restrict__ start,
                           const int *__restrict__ rank_desc, const int *__restrict__ count, int np,
                           int *__restrict__ by_pos) {
  FS_AFTER_PREVIOUS();
  int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b < np) by_pos[start[cell_of[b]] + rank_desc[b]] = count[b];
}

__global__ void k_pair_off(const int *__restrict__ cell_of, const int *__restrict__ start,
                           const int *__restrict__ rank_desc, const int *__restrict__ off_by_pos, int np,
                           int *__restrict__ off) {
  FS_AFTER_PREVIOUS();
  int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b < np) off[b] = off_by_pos[start[cell_of[b]] + rank_desc[b]];
}

// local minimum starts at 100000 as in apply_collision_barrier (CollisionBarrierFilament.cpp:41)
__global__ void k_set_min_init(unsigned long long *bits) {
  FS_AFTER_PREVIOUS(); *bits = fs_dbits(100000.0); }

BarrierConsts make_bconsts(const fs_ctx *c, int nt) {
  BarrierConsts k;
  for (int d = 0; d < 3; ++d) {
    k.L[d] = c->L[d];
    k.M[d] = c->M[d];
  }
  const double Rnm = 2 * c->p.a;
  const double Rnm2 = Rnm * Rnm;
  k.chiRnm2 = 1.21 * Rnm2;
  k.den = k.chiRnm2 - Rnm2;
  k.cap = c->p.barrier_distance_cap;
  k.cap2 = k.cap * k.cap;
  k.fs = c->p.barrier_fs_over_2a;
  k.nt = nt;
  k.initial_friction_steps = c->p.initial_friction_steps;
  k.mode = FS_BARRIER_ALL;
  k.np = 0;
  return k;
}

}  // namespace

fs_status cells_init(fs_ctx *c) {
  const double Rref = c->p.cell_width;
  for (int d = 0; d < 3; ++d) {
    c->M[d] = (int)(c->L[d] / Rref);
    if (c->M[d] < 1) return FS_ERR_INVALID_ARG;
  }
  c->ncell = c->M[0] * c->M[1] * c->M[2];
  FS_TRY(fs_sort_alloc(&c->cells, c->ncell, c->max_beads, &c->bytes));
  FS_TRY(fs_sort_prepare<CellKey>());
  const int nb = c->max_beads > 0 ? c->max_beads : 1;
  FS_CUDA(cudaMalloc(&c->head, sizeof(int) * c->ncell));
  FS_CUDA(cudaMalloc(&c->list, sizeof(int) * nb));
  FS_CUDA(cudaMalloc(&c->map, sizeof(int) * 13 * (size_t)c->ncell));
  FS_CUDA(cudaMalloc(&c->cell_rank, sizeof(int) * nb));
  FS_CUDA(cudaMalloc(&c->pair_count, sizeof(int) * (size_t)(nb + 1)));
  FS_CUDA(cudaMalloc(&c->pair_off, sizeof(int) * (size_t)(nb + 1)));
  FS_CUDA(cudaMalloc(&c->min_dist2_bits, sizeof(unsigned long long)));
  FS_CUDA(cudaMalloc(&c->pair_scan_tmp, sizeof(int) * (size_t)((nb + 1) / 4096 + 2)));
  c->bytes += sizeof(int) * ((size_t)14 * c->ncell + 4 * (size_t)nb);
  fs_launch(k_bulkmap, fs_blocks(c->ncell, 256), 256, 0, c->stream, c->M[0], c->M[1], c->M[2], c->map);
  FS_LAUNCH_CHECK();
  c->cells_np = -1;
  return FS_OK;
}

void cells_free(fs_ctx *c) {
  fs_sort_free(&c->cells);
  cudaFree(c->head);
  cudaFree(c->list);
  cudaFree(c->map);
  cudaFree(c->cell_rank);
  cudaFree(c->pair_count);
  cudaFree(c->pair_off);
  cudaFree(c->min_dist2_bits);
  cudaFree(c->pair_scan_tmp);
}

fs_status cells_link(fs_ctx *c, const double *Xs, int np) {
  ProfScope ps(c, FS_STAGE_LINK);
  BarrierConsts k = make_bconsts(c, 0);
  FS_TRY(fs_sort_run(&c->cells, CellKey{Xs, k}, np, c->stream));
  fs_launch(k_cell_lists, fs_blocks(c->ncell, 256), 256, 0, c->stream, c->cells.start, c->cells.sorted, c->ncell,
            c->head, c->list, c->cell_rank, c->flags);
  FS_LAUNCH_CHECK();
  c->cells_np = np;
  return FS_OK;
}

fs_status cells_barrier(fs_ctx *c, const double *Y, double *F, int np, int nt, const int *fil_id,
                        const int *seg_id, int *pairs_d, int max_pairs, int *npairs_h, int mode) {
  if (c->cells_np != np) return FS_ERR_STATE;
  ProfScope ps(c, FS_STAGE_BARRIER);
  BarrierConsts k = make_bconsts(c, nt);
  k.mode = mode;
  k.np = np;
  fs_launch(k_set_min_init, 1, 1, 0, c->stream, c->min_dist2_bits);
  FS_LAUNCH_CHECK();
  c->min_dist2_valid = true;
  if (np == 0) return FS_OK;
  const int T = 128;
  if (npairs_h) {
    fs_launch(k_pairs, fs_blocks(np, T), T, 0, c->stream, Y, np, k, c->cells.key, c->cells.start, c->cells.sorted,
              c->cell_rank, c->map, fil_id, seg_id, c->pair_count, nullptr, nullptr, 0);
    FS_LAUNCH_CHECK();
    // offsets in the reference's visiting order of the i beads
    fs_launch(k_pair_pos, fs_blocks(np, 256), 256, 0, c->stream, c->cells.key, c->cells.start, c->cell_rank,
              c->pair_count, np, c->pair_off);
    FS_LAUNCH_CHECK();
    FS_CUDA(cudaMemsetAsync(c->pair_off + np, 0, sizeof(int), c->stream));
    FS_TRY(fs_exclusive_scan(c->pair_off, c->pair_count, np + 1, c->pair_scan_tmp, c->stream));
    FS_CUDA(cudaMemcpyAsync(npairs_h, c->pair_count + np, sizeof(int), cudaMemcpyDeviceToHost, c->stream));
    fs_launch(k_pair_off, fs_blocks(np, 256), 256, 0, c->stream, c->cells.key, c->cells.start, c->cell_rank,
              c->pair_count, np, c->pair_off);
    FS_LAUNCH_CHECK();
    fs_launch(k_pairs, fs_blocks(np, T), T, 0, c->stream, Y, np, k, c->cells.key, c->cells.start, c->cells.sorted,
              c->cell_rank, c->map, fil_id, seg_id, nullptr, c->pair_off, pairs_d, max_pairs);
    FS_LAUNCH_CHECK();
    FS_CUDA(cudaStreamSynchronize(c->stream));
    return FS_OK;
  }
  if (np <= BARRIER_WIDE_PER_SM * c->num_sms)
    fs_launch(k_barrier<32>, fs_blocks(np, T / 32), T, 0, c->stream, Y, F, np, k, c->cells.key, c->cells.start,
              c->cells.sorted, c->cell_rank, fil_id, seg_id, c->min_dist2_bits, c->flags);
  else
    fs_launch(k_barrier<8>, fs_blocks(np, T / 8), T, 0, c->stream, Y, F, np, k, c->cells.key, c->cells.start,
              c->cells.sorted, c->cell_rank, fil_id, seg_id, c->min_dist2_bits, c->flags);
  FS_LAUNCH_CHECK();
  return FS_OK;
}
