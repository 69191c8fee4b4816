// fs_sort.cu -- deterministic counting sort of items by integer key.
//
// keys and count (an atomic per item, which also gives the item a slot of its key) -> exclusive
// scan -> scatter to the slots -> rank of each item by id among its key's. The slots depend
// on atomic timing; the ranks make the output a pure function of the keys: items ascend by
// (key, id). This is the order the collision linked list of LinkedList::link
// (CollisionBarrierFilament.cpp:370-433) encodes in reverse. Small sorts run all steps in
// one CTA. The steps that form the keys are templates on them (fs_sort.cuh).
#include "fs_internal.cuh"

fs_status fs_exclusive_scan(const int *in, int *out, int n, int *block_sums, cudaStream_t st);

#define SCAN_THREADS 1024
#define SCAN_ITEMS 4
#define SCAN_SPAN (SCAN_THREADS * SCAN_ITEMS)

// exclusive scan of in[0..n) into out, block totals into bsum
__global__ void __launch_bounds__(SCAN_THREADS) k_scan_block(const int *in, int *out, int n, int *bsum) {
  FS_AFTER_PREVIOUS();
  __shared__ int warp_tot[32];
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  const long long base = (long long)blockIdx.x * SCAN_SPAN + (long long)t * SCAN_ITEMS;
  int v[SCAN_ITEMS];
  int s = 0;
#pragma unroll
  for (int i = 0; i < SCAN_ITEMS; ++i) {
    long long idx = base + i;
    v[i] = idx < n ? in[idx] : 0;
    s += v[i];
  }
  int incl = s;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    int y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  if (lane == 31) warp_tot[w] = incl;
  __syncthreads();
  if (w == 0) {
    int x = lane < (SCAN_THREADS / 32) ? warp_tot[lane] : 0;
    int ix = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      int y = __shfl_up_sync(0xffffffffu, ix, o);
      if (lane >= o) ix += y;
    }
    warp_tot[lane] = ix - x;
  }
  __syncthreads();
  int run = incl - s + warp_tot[w];
  if (t == SCAN_THREADS - 1 && bsum) bsum[blockIdx.x] = run + s;
#pragma unroll
  for (int i = 0; i < SCAN_ITEMS; ++i) {
    long long idx = base + i;
    if (idx < n) out[idx] = run;
    run += v[i];
  }
}

__global__ void k_scan_add(int *__restrict__ out, int n, const int *__restrict__ bsum) {
  FS_AFTER_PREVIOUS();
  long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx < n) out[idx] += bsum[idx / SCAN_SPAN];
}

__global__ void k_sort_scatter(const int *__restrict__ key, const int *__restrict__ slot, int n,
                               const int *__restrict__ start, int *__restrict__ placed) {
  FS_AFTER_PREVIOUS();
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) placed[start[key[i]] + slot[i]] = i;
}

// position of item i among its key's items by id (a thread per item: a shell sort by one
// thread per key took 15 to 27 us at 8 to 30 items a key, this 3 to 5)
__global__ void k_sort_rank(const int *__restrict__ key, int n, const int *__restrict__ start,
                            const int *__restrict__ placed, int *__restrict__ sorted) {
  FS_AFTER_PREVIOUS();
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int k = key[i], s0 = start[k], s1 = start[k + 1];
  int r = 0;
  for (int p = s0; p < s1; ++p) r += placed[p] < i;
  sorted[s0 + r] = i;
}

fs_status fs_sort_alloc(fs_sort *s, int nkeys, int max_items, size_t *bytes) {
  s->nkeys = nkeys;
  int nblk = (nkeys + 1 + SCAN_SPAN - 1) / SCAN_SPAN;
  if (nblk > SCAN_SPAN) return FS_ERR_INVALID_ARG;
  FS_CUDA(cudaMalloc(&s->key, sizeof(int) * (size_t)(max_items > 0 ? max_items : 1)));
  FS_CUDA(cudaMalloc(&s->count, sizeof(int) * (size_t)(nkeys + 1)));
  FS_CUDA(cudaMalloc(&s->start, sizeof(int) * (size_t)(nkeys + 1)));
  FS_CUDA(cudaMalloc(&s->slot, sizeof(int) * (size_t)(max_items > 0 ? max_items : 1)));
  FS_CUDA(cudaMalloc(&s->placed, sizeof(int) * (size_t)(max_items > 0 ? max_items : 1)));
  FS_CUDA(cudaMalloc(&s->sorted, sizeof(int) * (size_t)(max_items > 0 ? max_items : 1)));
  FS_CUDA(cudaMalloc(&s->block_sums, sizeof(int) * (size_t)(nblk + 1)));
  *bytes += sizeof(int) * ((size_t)4 * (max_items > 0 ? max_items : 1) + 2 * (size_t)(nkeys + 1) + nblk + 1);
  return FS_OK;
}

void fs_sort_free(fs_sort *s) {
  cudaFree(s->key);
  cudaFree(s->count);
  cudaFree(s->start);
  cudaFree(s->slot);
  cudaFree(s->placed);
  cudaFree(s->sorted);
  cudaFree(s->block_sums);
  s->key = s->count = s->start = s->slot = s->placed = s->sorted = s->block_sums = nullptr;
}

fs_status fs_sort_finish(fs_sort *s, int n, cudaStream_t st) {
  FS_TRY(fs_exclusive_scan(s->count, s->start, s->nkeys + 1, s->block_sums, st));
  if (n > 0) {
    fs_launch(k_sort_scatter, fs_blocks(n, 256), 256, 0, st, s->key, s->slot, n, s->start, s->placed);
    FS_LAUNCH_CHECK();
    fs_launch(k_sort_rank, fs_blocks(n, 256), 256, 0, st, s->key, n, s->start, s->placed, s->sorted);
    FS_LAUNCH_CHECK();
  }
  return FS_OK;
}

// exclusive scan of n ints (n <= SCAN_SPAN^2); block_sums needs n/SCAN_SPAN+1 ints
fs_status fs_exclusive_scan(const int *in, int *out, int n, int *block_sums, cudaStream_t st) {
  if (n <= 0) return FS_OK;
  int nblk = (n + SCAN_SPAN - 1) / SCAN_SPAN;
  if (nblk > SCAN_SPAN) return FS_ERR_INVALID_ARG;
  fs_launch(k_scan_block, nblk, SCAN_THREADS, 0, st, in, out, n, block_sums);
  FS_LAUNCH_CHECK();
  if (nblk > 1) {
    fs_launch(k_scan_block, 1, SCAN_THREADS, 0, st, block_sums, block_sums, nblk, nullptr);
    FS_LAUNCH_CHECK();
    fs_launch(k_scan_add, fs_blocks(n, 256), 256, 0, st, out, n, block_sums);
    FS_LAUNCH_CHECK();
  }
  return FS_OK;
}
