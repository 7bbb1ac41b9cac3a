// Stable counting sort of positions by key (stable_sort.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "internal.h"

namespace ss {

struct StableSortPlan {
  bool ok;         // false: more than 4096 buckets of 4096 keys
  int f, NB;       // 2^f keys per bucket, buckets
  int ranges, range;  // level-1 blocks and the elements each owns
};

struct SortArgs {
  const int32_t *keys;     // [nnz]
  const int32_t *payload;  // [nnz]
  const void *vals;        // gathered by position into out_vals, or null
  int K, nnz, vsize;
  int32_t *out_indptr, *perm, *out_payload;  // [K + 1], [nnz], [nnz]
  void *out_vals;
  // filled by stable_sort
  int f, F, NB, nb_bits, ranges, range;
  int32_t *cnt, *count, *start, *order;
  int2 *rec;      // position, payload
  int32_t *rkey;
};

StableSortPlan stable_sort_plan(int K, int nnz);
size_t stable_sort_ws(const StableSortPlan &p, int nnz);
// perm = positions grouped by key in [0, K), in input order inside a key;
// elements with other keys land past out_indptr[K] as -1, their values as 0.
ss_status stable_sort(const StableSortPlan &p, SortArgs &a, void *ws, cudaStream_t s);

}  // namespace ss
