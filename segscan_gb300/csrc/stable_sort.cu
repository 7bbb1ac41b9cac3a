// Stable counting sort of positions by key, in two levels: COO -> CSR (key =
// row, payload = column).
//
// Reference semantics: compressedRow (test-cg/include/dataloader/
// dataloader.hpp:109-121): entries of one row keep their input order.  Each
// level keeps that order by ranking, so no row's entries are sorted
// afterwards, and neither a long row nor sorted input is a special case:
//  * a block gives every warp a contiguous piece of its elements; the warp
//    ranks 32 of them at a time (ballots per digit bit) against a table of
//    counts of its own in shared memory, and the tables' prefix over warps
//    and digits gives each element its place;
//  * level 1: digit = bucket of F = 2^f consecutive keys.  Each block owns a
//    contiguous range of elements, whose count per bucket is known from a
//    counting pass, so its runs start at fixed places (no atomics on the
//    cursors, which would order the runs by chance);
//  * level 2: digit = key inside the bucket, a block per bucket, 8192 records
//    at a time; a longer bucket carries its cursors from chunk to chunk.
// Values are gathered by position at the end.
//
// 4.62 M shuffled edges of 1 M power-law rows, values included: 1130 -> 175
// us, where the one-level sort (atomic scatter, then a sort per row) spent
// 904 us in bitonic sorts of the rows above 32 entries.  Bound by shared
// memory passes and barriers (24 K cycles a tile of 4096, 5 K of them bank
// conflicts of the scatter), not by DRAM (300 MB of traffic).  The transpose
// keeps its own sort (transpose.cu): its columns are short and its rows
// ordered, which needs no ranking (165 us there, 188 by this one).
#include <algorithm>
#include <climits>

#include "stable_sort.cuh"

namespace ss {

namespace {

constexpr int NB_MAX = 4096, F_LOG2_MAX = 12;
constexpr int PT = 512, PER1 = 8;   // level 1: threads, elements per thread and tile
constexpr int T2 = 512, PER2 = 16;  // level 2: threads, records per thread and chunk
constexpr int CHUNK2 = T2 * PER2;

size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

// Exclusive prefix sums of x[0, n) in place by the whole block; returns the
// total.  The caller synchronises before; wbuf: 33 ints.
__device__ int block_exclusive(int32_t *x, int n, int32_t *wbuf) {
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, W = blockDim.x >> 5;
  const int seg = ((n + W - 1) / W + 31) & ~31;
  const int lo = min(wid * seg, n), hi = min(lo + seg, n);
  int carry = 0;
  for (int b = lo; b < hi; b += 32) {
    const int i = b + lane;
    const int v0 = i < hi ? x[i] : 0;
    int v = v0;
    #pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, v, off);
      if (lane >= off) v += y;
    }
    if (i < hi) x[i] = carry + v - v0;
    carry += __shfl_sync(0xffffffffu, v, 31);
  }
  if (lane == 0) wbuf[wid] = carry;
  __syncthreads();
  if (wid == 0) {
    const int w = lane < W ? wbuf[lane] : 0;
    int v = w;
    #pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, v, off);
      if (lane >= off) v += y;
    }
    wbuf[lane] = v - w;
    if (lane == 31) wbuf[32] = v;
  }
  __syncthreads();
  const int pre = wbuf[wid];
  for (int i = lo + lane; i < hi; i += 32) x[i] += pre;
  const int total = wbuf[32];
  __syncthreads();
  return total;
}

// Ranks of a warp's N x 32 elements (step by step in input order) among the
// earlier elements of the same digit (< 0: none) in the warp's piece.  hist
// is the warp's own table of counts, two 16-bit counts a word.  The lanes of
// one digit are found with a ballot per digit bit (match_any takes about 40
// cycles of an SM each: 12,000 cycles of a tile's 28,000), and the counts are
// taken by atomics whose results are used at the end, so their latency is
// not paid once per step.
template <int N>
__device__ __forceinline__ void warp_ranks(uint32_t *hist, const int (&d)[N], int (&rank)[N], int lane, int bits) {
  unsigned m[N];
  #pragma unroll
  for (int k = 0; k < N; k++) m[k] = __ballot_sync(0xffffffffu, d[k] >= 0);
  for (int b = 0; b < bits; b++) {
    #pragma unroll
    for (int k = 0; k < N; k++) {
      const bool on = (d[k] >> b) & 1;
      const unsigned v = __ballot_sync(0xffffffffu, on);
      m[k] &= on ? v : ~v;
    }
  }
  #pragma unroll
  for (int k = 0; k < N; k++) {
    const int sh = (d[k] & 1) * 16;
    rank[k] = 0;
    if (d[k] >= 0 && (m[k] & ((1u << lane) - 1u)) == 0u)  // the first of its digit counts for all
      rank[k] = (int)((atomicAdd(hist + (d[k] >> 1), (unsigned)__popc(m[k]) << sh) >> sh) & 0xffffu);
    __syncwarp();  // the next step's counts come after this step's
  }
  #pragma unroll
  for (int k = 0; k < N; k++)
    rank[k] = __shfl_sync(0xffffffffu, rank[k], max(__ffs(m[k]) - 1, 0)) + __popc(m[k] & ((1u << lane) - 1u));
}

// Turns the W warps' counts of the digits 2i and 2i + 1 into their exclusive
// prefix over the warps; returns both totals packed.  (A tile has at most
// 8192 elements, so no half carries into the other.)
template <int W>
__device__ __forceinline__ uint32_t warps_prefix(uint32_t *hist, int words, int i) {
  uint32_t c[W], run = 0;
  #pragma unroll
  for (int w = 0; w < W; w++) c[w] = hist[w * words + i];
  #pragma unroll
  for (int w = 0; w < W; w++) {
    hist[w * words + i] = run;
    run += c[w];
  }
  return run;
}
__device__ __forceinline__ int half_of(const uint32_t *hist, int d) {
  return reinterpret_cast<const uint16_t *>(hist)[d];
}

// ---------------------------------------------------------------------
// level 1
// ---------------------------------------------------------------------
__global__ void __launch_bounds__(1024) range_count_kernel(SortArgs a) {
  extern __shared__ int32_t h[];
  for (int i = threadIdx.x; i < a.NB; i += 1024) h[i] = 0;
  __syncthreads();
  const long long r0 = (long long)blockIdx.x * a.range;
  const int lo = (int)min(r0, (long long)a.nnz), hi = (int)min(r0 + a.range, (long long)a.nnz);
  for (long long b = lo + (long long)threadIdx.x; b < hi; b += 4096) {
    int c[4];
    #pragma unroll
    for (int u = 0; u < 4; u++) c[u] = b + u * 1024 < hi ? __ldg(a.keys + b + u * 1024) : -1;
    #pragma unroll
    for (int u = 0; u < 4; u++)
      if ((unsigned)c[u] < (unsigned)a.K) atomicAdd(h + (c[u] >> a.f), 1);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < a.NB; i += 1024) a.cnt[(size_t)i * a.ranges + blockIdx.x] = h[i];
}

// A warp per bucket: the ranges' counts become their exclusive prefix.
__global__ void __launch_bounds__(256) range_prefix_kernel(SortArgs a) {
  const int b = (blockIdx.x * 256 + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (b >= a.NB) return;
  int32_t *c = a.cnt + (size_t)b * a.ranges;
  int carry = 0;
  for (int i0 = 0; i0 < a.ranges; i0 += 32) {
    const int i = i0 + lane;
    const int v0 = i < a.ranges ? c[i] : 0;
    int v = v0;
    #pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, v, off);
      if (lane >= off) v += y;
    }
    if (i < a.ranges) c[i] = carry + v - v0;
    carry += __shfl_sync(0xffffffffu, v, 31);
  }
  if (lane == 0) a.count[b] = carry;
}

// A tile of PT * PER1 elements per round: ranked, grouped by bucket in shared
// memory and written out as one contiguous run per bucket.
__global__ void __launch_bounds__(PT, 2) partition_kernel(SortArgs a) {
  constexpr int TILE = PT * PER1, W = PT / 32;
  extern __shared__ int32_t sm[];
  int32_t *lst = sm;                   // [NB + 1] the tile's count, then start, per bucket
  int32_t *base = lst + a.NB + 1;      // [NB] where the tile's run of a bucket goes
  int32_t *s_pay = base + a.NB;        // [TILE] staged payloads
  int32_t *s_key = s_pay + TILE;       // [TILE] staged keys
  uint32_t *hist = (uint32_t *)(s_key + TILE);  // [W][words] counts of each warp
  const int words = (a.NB + 1) / 2;
  uint16_t *s_pos = (uint16_t *)(hist + W * words);  // [TILE] staged positions in the tile
  __shared__ int32_t wbuf[33];
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  // bucket starts; every block scans the same counts, the first one keeps them
  for (int i = tid; i < a.NB; i += PT) base[i] = a.count[i];
  __syncthreads();
  const int total = block_exclusive(base, a.NB, wbuf);
  if (blockIdx.x == 0) {
    for (int i = tid; i < a.NB; i += PT) a.start[i] = base[i];
    if (tid == 0) a.start[a.NB] = total;
    if (tid == 0) a.out_indptr[a.K] = total;
    for (long long q = (long long)total + tid; q < a.nnz; q += PT) {  // elements with keys outside [0, K)
      a.perm[q] = -1;
      a.out_payload[q] = -1;
      if (a.out_vals && a.vsize == 4) ((uint32_t *)a.out_vals)[q] = 0u;
      else if (a.out_vals) ((uint16_t *)a.out_vals)[q] = 0;
    }
  }
  if (blockIdx.x == 0) {
    // the order in which level 2 takes the buckets: those longer than a chunk
    // first, since a late one would run alone (147 -> 103 us on power-law rows)
    for (int i = tid; i < a.NB; i += PT) s_key[i] = a.count[i] > CHUNK2;
    __syncthreads();
    const int nlong = block_exclusive(s_key, a.NB, wbuf);
    for (int i = tid; i < a.NB; i += PT)
      a.order[a.count[i] > CHUNK2 ? s_key[i] : nlong + i - s_key[i]] = i;
    __syncthreads();
  }
  for (int i = tid; i < a.NB; i += PT) base[i] += a.cnt[(size_t)i * a.ranges + blockIdx.x];
  const long long r0 = (long long)blockIdx.x * a.range;
  const int lo = (int)min(r0, (long long)a.nnz), hi = (int)min(r0 + a.range, (long long)a.nnz);
  for (long long t0 = lo; t0 < hi; t0 += TILE) {
    const int b0 = (int)t0, n = min(TILE, hi - b0);
    for (int i = tid; i < W * words; i += PT) hist[i] = 0u;
    int key[PER1], pay[PER1];
    const int e0 = wid * (PER1 * 32) + lane;  // a warp's elements are consecutive
    #pragma unroll
    for (int k = 0; k < PER1; k++) {
      const int e = e0 + k * 32;
      key[k] = e < n ? __ldg(a.keys + b0 + e) : -1;
      pay[k] = e < n ? __ldg(a.payload + b0 + e) : 0;
    }
    __syncthreads();
    int dig[PER1], rank[PER1];
    #pragma unroll
    for (int k = 0; k < PER1; k++) dig[k] = (unsigned)key[k] < (unsigned)a.K ? key[k] >> a.f : -1;
    warp_ranks<PER1>(hist + wid * words, dig, rank, lane, a.nb_bits);
    __syncthreads();
    for (int i = tid; i < words; i += PT) {
      const uint32_t both = warps_prefix<W>(hist, words, i);
      lst[2 * i] = both & 0xffff;
      if (2 * i + 1 < a.NB) lst[2 * i + 1] = both >> 16;
    }
    __syncthreads();
    const int valid = block_exclusive(lst, a.NB, wbuf);
    if (tid == 0) lst[a.NB] = valid;
    for (int d = tid; d < a.NB; d += PT) base[d] -= lst[d];  // place of the run's element i: base + i
    #pragma unroll
    for (int k = 0; k < PER1; k++) {
      if (dig[k] >= 0) {
        const int q = lst[dig[k]] + half_of(hist + wid * words, dig[k]) + rank[k];
        s_pos[q] = (uint16_t)(e0 + k * 32);
        s_pay[q] = pay[k];
        s_key[q] = key[k];
      }
    }
    __syncthreads();
    for (int i = tid; i < valid; i += PT) {
      const int c = s_key[i];
      const int q = base[c >> a.f] + i;
      a.rec[q] = make_int2(b0 + s_pos[i], s_pay[i]);
      a.rkey[q] = c;
    }
    __syncthreads();
    for (int d = tid; d < a.NB; d += PT) base[d] += lst[d + 1];
    __syncthreads();
  }
}

// ---------------------------------------------------------------------
// level 2
// ---------------------------------------------------------------------
__device__ __forceinline__ void copy_value(const SortArgs &a, int q, int p) {
  if (a.vsize == 4) ((uint32_t *)a.out_vals)[q] = __ldg((const uint32_t *)a.vals + p);
  else ((uint16_t *)a.out_vals)[q] = __ldg((const unsigned short *)a.vals + p);
}

__global__ void __launch_bounds__(T2, 2) bucket_kernel(SortArgs a) {
  constexpr int W = T2 / 32, H = 8;  // H records per thread ranked at a time
  extern __shared__ int32_t sm[];
  int32_t *tot = sm;               // [F + 2] counts, then starts, per key
  int32_t *s_pos = tot + a.F + 2;  // [CHUNK2]
  int32_t *s_pay = s_pos + CHUNK2;
  uint32_t *hist = (uint32_t *)(s_pay + CHUNK2);  // [W][words]
  __shared__ int32_t wbuf[33];
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int b = __ldg(a.order + blockIdx.x);
  const int c0 = b << a.f, nf = min(a.F, a.K - c0), words = (nf + 1) / 2;
  const int s0 = __ldg(a.start + b), n = __ldg(a.start + b + 1) - s0;
  const bool one = n <= CHUNK2;
  if (!one) {  // longer than a chunk: every key's start first
    for (int i = tid; i < nf; i += T2) tot[i] = 0;
    __syncthreads();
    for (long long i0 = tid; i0 < n; i0 += 8 * T2) {
      int c[8];
      #pragma unroll
      for (int u = 0; u < 8; u++) c[u] = i0 + u * T2 < n ? __ldg(a.rkey + s0 + i0 + u * T2) - c0 : -1;
      #pragma unroll
      for (int u = 0; u < 8; u++)
        if (c[u] >= 0) atomicAdd(tot + c[u], 1);
    }
    __syncthreads();
    block_exclusive(tot, nf, wbuf);
    for (int i = tid; i < nf; i += T2) a.out_indptr[c0 + i] = s0 + tot[i];
  }
  for (long long t0 = 0; t0 < n || t0 == 0; t0 += CHUNK2) {
    const int b0 = (int)t0;
    const int m = min(CHUNK2, n - b0);
    const int steps = (m + T2 - 1) / T2;  // 32-element steps per warp
    for (int i = tid; i < W * words; i += T2) hist[i] = 0u;
    int kr[PER2];  // key | rank << 16 (F <= 4096, ranks below 512), -1 none
    const int e0 = wid * steps * 32 + lane;
    #pragma unroll
    for (int k = 0; k < PER2; k++) {
      const int e = e0 + k * 32;
      kr[k] = k < steps && e < m ? __ldg(a.rkey + s0 + b0 + e) - c0 : -1;
    }
    __syncthreads();
    #pragma unroll
    for (int k0 = 0; k0 < PER2; k0 += H) {
      if (k0 >= steps) break;
      int d[H], r[H];
      #pragma unroll
      for (int k = 0; k < H; k++) d[k] = kr[k0 + k];
      warp_ranks<H>(hist + wid * words, d, r, lane, a.f);
      #pragma unroll
      for (int k = 0; k < H; k++)
        if (d[k] >= 0) kr[k0 + k] = d[k] | (r[k] << 16);
    }
    __syncthreads();
    for (int i = tid; i < words; i += T2) {
      const uint32_t both = warps_prefix<W>(hist, words, i);
      if (one) {
        tot[2 * i] = both & 0xffff;
        tot[2 * i + 1] = both >> 16;
      } else {
        // the cursors move past this chunk after its records are placed
        s_pos[2 * i] = both & 0xffff;
        s_pos[2 * i + 1] = both >> 16;
      }
    }
    __syncthreads();
    if (one) {
      block_exclusive(tot, nf, wbuf);
      for (int i = tid; i < nf; i += T2) a.out_indptr[c0 + i] = s0 + tot[i];
    }
    #pragma unroll
    for (int k0 = 0; k0 < PER2; k0 += H) {
      if (k0 >= steps) break;
      int2 rec[H];
      #pragma unroll
      for (int k = 0; k < H; k++)
        rec[k] = kr[k0 + k] >= 0 ? __ldg(a.rec + s0 + b0 + e0 + (k0 + k) * 32) : make_int2(0, 0);
      #pragma unroll
      for (int k = 0; k < H; k++) {
        if (kr[k0 + k] < 0) continue;
        const int d = kr[k0 + k] & 0xffff;
        const int q = tot[d] + half_of(hist + wid * words, d) + (kr[k0 + k] >> 16);
        if (one) {
          s_pos[q] = rec[k].x;
          s_pay[q] = rec[k].y;
        } else {
          a.perm[s0 + q] = rec[k].x;
          a.out_payload[s0 + q] = rec[k].y;
          if (a.out_vals) copy_value(a, s0 + q, rec[k].x);
        }
      }
    }
    __syncthreads();
    if (!one) {
      for (int d = tid; d < nf; d += T2) tot[d] += s_pos[d];
      __syncthreads();
      continue;
    }
    for (int i0 = tid; i0 < m; i0 += 8 * T2) {
      uint32_t v[8];
      if (a.out_vals) {
        #pragma unroll
        for (int u = 0; u < 8; u++) {
          const int i = i0 + u * T2;
          const int p = i < m ? s_pos[i] : 0;
          v[u] = a.vsize == 4 ? __ldg((const uint32_t *)a.vals + p) : __ldg((const unsigned short *)a.vals + p);
        }
      }
      #pragma unroll
      for (int u = 0; u < 8; u++) {
        const int i = i0 + u * T2;
        if (i >= m) break;
        a.perm[s0 + i] = s_pos[i];
        a.out_payload[s0 + i] = s_pay[i];
        if (a.out_vals) {
          if (a.vsize == 4) ((uint32_t *)a.out_vals)[s0 + i] = v[u];
          else ((uint16_t *)a.out_vals)[s0 + i] = (uint16_t)v[u];
        }
      }
    }
  }
}

// One key per bucket: level 1 has put everything in its place.
__global__ void __launch_bounds__(256) single_key_kernel(SortArgs a) {
  const int total = __ldg(a.start + a.NB);
  const long long stride = (long long)gridDim.x * 256, i0 = blockIdx.x * 256ll + threadIdx.x;
  for (long long i = i0; i < a.K; i += stride) a.out_indptr[i] = __ldg(a.start + i);
  for (long long q = i0; q < total; q += stride) {
    const int2 r = __ldg(a.rec + q);
    const int p = r.x;
    a.perm[q] = p;
    a.out_payload[q] = r.y;
    if (a.out_vals) copy_value(a, (int)q, p);
  }
}

size_t partition_smem(int NB) {
  return (size_t)(2 * NB + 1 + 2 * PT * PER1 + (PT / 32) * ((NB + 1) / 2)) * 4 + (size_t)PT * PER1 * 2;
}
size_t bucket_smem(int F) { return (size_t)(F + 2 + 2 * CHUNK2 + (T2 / 32) * ((F + 1) / 2)) * 4; }

}  // namespace

StableSortPlan stable_sort_plan(int K, int nnz) {
  StableSortPlan p{};
  if (K <= 0 || nnz <= 0) return p;  // nothing to sort (and no ranges to divide the elements by)
  // buckets of at most 6144 elements on average (a chunk holds 8192), more
  // keys per bucket where there would be too many buckets
  int f = F_LOG2_MAX;
  const double avg = (double)nnz / K;
  while (f > 0 && (double)(1 << f) * avg > 6144.0) f--;
  long long nb = ((long long)K + (1LL << f) - 1) >> f;
  while (nb > NB_MAX && f < F_LOG2_MAX) {
    f++;
    nb = ((long long)K + (1LL << f) - 1) >> f;
  }
  p.ok = nb <= NB_MAX;
  p.f = f;
  p.NB = (int)nb;
  // level 1: one range per resident block (two per SM while both blocks' count
  // tables fit)
  const int tile = PT * PER1, tiles = ceil_div(nnz, tile);
  p.ranges = std::max(1, std::min(tiles, sm_count() * (partition_smem(p.NB) <= 112 * 1024 ? 2 : 1)));
  p.range = ceil_div(tiles, p.ranges) * tile;
  p.ranges = ceil_div(nnz, p.range);
  return p;
}

size_t stable_sort_ws(const StableSortPlan &p, int nnz) {
  return align256((size_t)p.NB * p.ranges * 4) + 3 * align256((size_t)(p.NB + 1) * 4) + align256((size_t)nnz * 8) + align256((size_t)nnz * 4);
}

ss_status stable_sort(const StableSortPlan &p, SortArgs &a, void *ws, cudaStream_t s) {
  char *w = (char *)ws;
  a.cnt = (int32_t *)w; w += align256((size_t)p.NB * p.ranges * 4);
  a.count = (int32_t *)w; w += align256((size_t)(p.NB + 1) * 4);
  a.start = (int32_t *)w; w += align256((size_t)(p.NB + 1) * 4);
  a.order = (int32_t *)w; w += align256((size_t)(p.NB + 1) * 4);
  a.rec = (int2 *)w; w += align256((size_t)a.nnz * 8);
  a.rkey = (int32_t *)w;
  a.f = p.f; a.F = 1 << p.f; a.nb_bits = ilog2(p.NB); a.NB = p.NB; a.ranges = p.ranges; a.range = p.range;
  ss_status st = allow_smem((const void *)partition_kernel, partition_smem(NB_MAX), "stable sort partition");
  if (st == SS_OK) st = allow_smem((const void *)bucket_kernel, bucket_smem(1 << F_LOG2_MAX), "stable sort buckets");
  if (st == SS_OK) st = launch("stable sort counts", range_count_kernel, p.ranges, 1024, (size_t)p.NB * 4, s, a);
  if (st == SS_OK) st = launch("stable sort prefix", range_prefix_kernel, ceil_div(p.NB, 8), 256, 0, s, a);
  if (st == SS_OK) st = launch("stable sort partition", partition_kernel, p.ranges, PT, partition_smem(p.NB), s, a);
  if (st != SS_OK) return st;
  if (p.f == 0)
    return launch("stable sort", single_key_kernel, std::min(ceil_div(a.nnz, 256), sm_count() * 8), 256, 0, s, a);
  return launch("stable sort buckets", bucket_kernel, p.NB, T2, bucket_smem(a.F), s, a);
}

}  // namespace ss
