// fs_sort.cuh -- the counting sort's steps that form the items' keys, as templates on K, a
// value whose (device) K::operator()(i) is the key of item i (fs_sort.cu: the other steps).
#pragma once
#include "fs_internal.cuh"

fs_status fs_sort_finish(fs_sort *s, int n, cudaStream_t st);  // scan, scatter and ranks of counted keys

// One launch for keys and counts: with the link's own kernels 512^3 / 131,072 beads took 161 us
// in two, 155 in one.
// keys of n items, their counts and each item's slot among its key's (in arrival order)
template <typename K>
__global__ void k_sort_count(K key_of, int *__restrict__ key, int n, int *__restrict__ count, int *__restrict__ slot) {
  FS_AFTER_PREVIOUS();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int k = key_of(i);
  key[i] = k;
  slot[i] = atomicAdd(&count[k], 1);
}

// The whole sort in one CTA: counts, then starts, in shared memory (nkeys + 1 ints), then
// the placed items (n ints). Bound by its chain of barriers: with the key kernel and the
// lists of LinkedList::link 17 us at 480 beads / 2,197 cells, 27 at 4,000 / 39,304, where
// the separate launches take 34 and 42; both limits are what shared memory holds.
constexpr int SORT1_THREADS = 1024, SORT1_ITEMS = 4096, SORT1_KEYS = 40960;
template <typename K>
__global__ void __launch_bounds__(SORT1_THREADS) k_sort_one(K key_of, int *__restrict__ key, int n, int nkeys,
                                                            int *__restrict__ start, int *__restrict__ sorted) {
  FS_AFTER_PREVIOUS();
  extern __shared__ int sort_smem[];
  __shared__ int warp_tot[32];
  int *cnt = sort_smem, *placed = sort_smem + nkeys + 1;
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  constexpr int PER = SORT1_ITEMS / SORT1_THREADS;
  for (int k = t; k <= nkeys; k += SORT1_THREADS) cnt[k] = 0;
  __syncthreads();
  int ks[PER], slot[PER];
#pragma unroll
  for (int q = 0; q < PER; ++q) {
    const int i = t + q * SORT1_THREADS;
    ks[q] = i < n ? key_of(i) : -1;
    if (i < n) key[i] = ks[q];
    slot[q] = i < n ? atomicAdd(&cnt[ks[q]], 1) : 0;
  }
  __syncthreads();
  // exclusive scan in place, thread t over keys [t c, (t + 1) c)
  // (c odd: the threads' strided accesses fall on different banks)
  const int c = ((nkeys + SORT1_THREADS) / SORT1_THREADS) | 1, k0 = min(t * c, nkeys + 1), k1 = min(k0 + c, nkeys + 1);
  int sum = 0;
  for (int k = k0; k < k1; ++k) sum += cnt[k];
  int incl = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  if (lane == 31) warp_tot[w] = incl;
  __syncthreads();
  if (w == 0) {
    const int x = warp_tot[lane];
    int ix = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, ix, o);
      if (lane >= o) ix += y;
    }
    warp_tot[lane] = ix - x;
  }
  __syncthreads();
  int run = incl - sum + warp_tot[w];
  for (int k = k0; k < k1; ++k) {
    const int v = cnt[k];
    cnt[k] = run;
    run += v;
  }
  __syncthreads();
  for (int k = t; k <= nkeys; k += SORT1_THREADS) start[k] = cnt[k];
#pragma unroll
  for (int q = 0; q < PER; ++q)
    if (ks[q] >= 0) placed[cnt[ks[q]] + slot[q]] = t + q * SORT1_THREADS;
  __syncthreads();
#pragma unroll
  for (int q = 0; q < PER; ++q) {
    if (ks[q] < 0) continue;
    const int i = t + q * SORT1_THREADS, s0 = cnt[ks[q]], s1 = cnt[ks[q] + 1];
    int r = 0;
    for (int p = s0; p < s1; ++p) r += placed[p] < i;
    sorted[s0 + r] = i;
  }
}

template <typename K>
fs_status fs_sort_prepare() {
  FS_CUDA(cudaFuncSetAttribute(k_sort_one<K>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)(sizeof(int) * (SORT1_KEYS + 1 + SORT1_ITEMS))));
  return FS_OK;
}

// sorts items 0 .. n - 1 by (key, id): s->key, s->start and s->sorted
template <typename K>
fs_status fs_sort_run(fs_sort *s, const K &key_of, int n, cudaStream_t st) {
  const int nk1 = s->nkeys + 1;
  // one CTA as far as its shared memory goes (see k_sort_one)
  if (n <= SORT1_ITEMS && s->nkeys <= SORT1_KEYS) {
    fs_launch(k_sort_one<K>, 1, SORT1_THREADS, sizeof(int) * (nk1 + (n > 0 ? n : 1)), st, key_of, s->key, n, s->nkeys,
              s->start, s->sorted);
    FS_LAUNCH_CHECK();
    return FS_OK;
  }
  FS_CUDA(cudaMemsetAsync(s->count, 0, sizeof(int) * nk1, st));
  if (n > 0) {
    fs_launch(k_sort_count<K>, fs_blocks(n, 256), 256, 0, st, key_of, s->key, n, s->count, s->slot);
    FS_LAUNCH_CHECK();
  }
  return fs_sort_finish(s, n, st);
}
