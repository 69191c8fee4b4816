// fs_events.cuh -- the order of a bead's collision events (k_barrier), in plain C++ so that the
// host can check it too.
#pragma once

// Place of event e among the n events of keys key[]: by key, then by index. The index makes
// the places a permutation of 0 .. n - 1 whatever the keys, so every entry below n of a list
// filled by place is written. Equal keys do occur: where an axis has one cell, a neighbour
// slot names the bead's own cell and the bead meets itself under one key as i and as j; and the
// positions of more than 4,096 beads in a cell overflow their part of the key.
__host__ __device__ __forceinline__ int event_place(const unsigned long long *key, int n, int e) {
  const unsigned long long mine = key[e];
  int place = 0;
  for (int o = 0; o < n; ++o) place += key[o] < mine || (key[o] == mine && o < e);
  return place;
}
