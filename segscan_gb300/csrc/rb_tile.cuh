// Row-balanced sequential SpMM (rbsr): groups of rows, staged.
//
// Reference counterpart: csrspmm_seqreduce_rowbalance_cg_kernel
// (test-cg/include/spmm/spmm_cg.cuh:593-662).
//
// A group of G lanes along N (E = V * NV columns a lane) owns a few
// consecutive rows, about as many as fill its stage.  It stages their columns
// and values in shared memory, marks each row's last nonzero with row + 1 and
// walks them four at a time across the row ends, so a batch of gathers is
// full whatever the row lengths, and the chain row pointer -> column -> B row
// is paid once per few rows instead of once per row.  Longer rows go through
// the stage piece by piece.  Every row is summed in order by one group, so
// the result does not depend on the tuple.  Groups share nothing: no block
// barrier.
//
// us, a row per team before -> staged: Poisson 200 K x 16, N = 64 94 -> 71;
// 200 K x 1.5, N = 32 31 -> 21; banded 120 K x 20, N = 128 BF16 97 -> 69,
// N = 64 FP32 57 -> 54.  In the last L1 serves 56 % of the sectors (614 MB of
// gathered rows) and L2 the other 301 MB at 5.7 TB/s; issue is 50 % busy.
#pragma once

#include "eb_tile.cuh"

namespace ss {

struct RowArgs {
  const int32_t *indptr, *cols;
  const void *vals, *B;
  void *C;
  int M, K, N, nnz;
  int rows;        // rows per group at a time
  int block_rows;  // rows per block, where the rows are about even
  long long share;  // cost of a block above which they are not (0: not looked at)
  int kahan;
  float keep_frac;
};

constexpr int ROW_CAP = 64;  // nonzeros a group stages
constexpr int ROW_COST = 2;  // a row's own cost (its store, the walk's bookkeeping), in nonzeros

template <typename T, typename TC, int G, int V, int NV, bool ADDC>
struct RowWalk {
  const RowArgs &a;
  const char *Bj[NV];
  char *Cj[NV];
  uint32_t ldb, ldc;
  uint64_t keep, strm;
  float acc[NV][V], comp[NV][V];

  __device__ __forceinline__ RowWalk(const RowArgs &a_, int lane, int col0, const bool (&act)[NV])
      : a(a_), ldb((uint32_t)a_.N * (uint32_t)sizeof(T)), ldc((uint32_t)a_.N * (uint32_t)sizeof(TC)),
        keep(policy_keep(a_.keep_frac)), strm(policy_stream()) {
    #pragma unroll
    for (int j = 0; j < NV; j++) {
      // lanes past the last column repeat one that this lane (or lane 0) has
      // (accumulating, they leave the walk to the others: they could read a
      // row after another lane's store)
      const int cj = act[j] ? col0 + j * G * V : act[0] ? col0 : col0 - lane * V;
      Bj[j] = (const char *)((const T *)a.B + cj);
      Cj[j] = (char *)((TC *)a.C + cj) - ldc;
    }
    clear<V, NV>(acc);
    clear<V, NV>(comp);
  }
  __device__ __forceinline__ void fetch(RawVec<T, V> (&raw)[NV], int c) {
    #pragma unroll
    for (int j = 0; j < NV; j++) load_raw<T, V>((const T *)(Bj[j] + (uint64_t)(uint32_t)c * ldb), raw[j], keep);
  }
  __device__ __forceinline__ void fetch_old(OldVec<TC, V> (&old)[NV], int end) {
    #pragma unroll
    for (int j = 0; j < NV; j++)
      load_old_if<TC, V>((const TC *)(Cj[j] + (uint64_t)(uint32_t)end * ldc), old[j], end);
  }
  // one nonzero; a marked one ends its row
  __device__ __forceinline__ void consume(const RawVec<T, V> (&raw)[NV], const OldVec<TC, V> (&old)[NV], float v,
                                          int end, bool kah) {
    #pragma unroll
    for (int j = 0; j < NV; j++) {
      float b[V];
      unpack_raw<T, V>(raw[j], b);
      if (kah) {
        kahan_fma<V>(acc[j], comp[j], v, b);
      } else {
        #pragma unroll
        for (int i = 0; i < V; i++) acc[j][i] = fmaf(v, b[i], acc[j][i]);
      }
      TC *d = (TC *)(Cj[j] + (uint64_t)(uint32_t)end * ldc);
      if (ADDC) {
        float x[V];
        unpack_old<TC, V>(old[j], x);
        #pragma unroll
        for (int i = 0; i < V; i++) x[i] += acc[j][i];
        store_vec_if<TC, V>(d, x, strm, end);
      } else {
        store_vec_if<TC, V>(d, acc[j], strm, end);
      }
      #pragma unroll
      for (int i = 0; i < V; i++) {
        acc[j][i] = end ? 0.f : acc[j][i];
        comp[j][i] = end ? 0.f : comp[j][i];
      }
    }
  }
};

// A block per SM walks a contiguous range of rows, its groups side by side, so
// that rows with near columns share the SM's L1.  The ranges have equal numbers
// of rows, or, where one of those costs more than a.share, equal cost: rows
// whose lengths follow their index would leave most SMs waiting for a few.
template <typename T, typename TC, int G, int V, int NV, bool ADDC>
__global__ void __launch_bounds__(ADDC ? 768 : 1024, 1) rb_tile_kernel(RowArgs a) {
  constexpr int COLS = G * V * NV, CAP = ROW_CAP, PAD = CAP + 4, IT = CAP / G;
  extern __shared__ __align__(16) int32_t smem[];
  const int NG = blockDim.x / G;
  const int tid = threadIdx.x, wl = tid & 31, lane = tid & (G - 1), g = tid / G;
  int32_t *s_col = smem + g * PAD;
  float *s_val = (float *)(smem + NG * PAD) + g * PAD;
  int32_t *s_info = smem + 2 * NG * PAD + g * PAD;
  const unsigned mask = G >= 32 ? 0xffffffffu : (((1u << (G & 31)) - 1u) << (wl & ~(G - 1)));
  const int col0 = blockIdx.y * COLS + lane * V;
  bool act[NV];
  #pragma unroll
  for (int j = 0; j < NV; j++) act[j] = col0 + j * G * V < a.N;
  RowWalk<T, TC, G, V, NV, ADDC> w(a, lane, col0, act);
  auto clamped = [&](int r) { return max(0, min(__ldg(a.indptr + r), a.nnz)); };
  // this block's rows and the rows of a unit (in shared memory: the walk needs
  // the registers)
  __shared__ int s_rows[3];
  __shared__ int s_next;
  const int blocks = gridDim.x;
  if (tid < 2) s_rows[tid] = (int)min((long long)(blockIdx.x + tid) * a.block_rows, (long long)a.M);
  if (tid == 0) { s_rows[2] = a.rows; s_next = NG; }
  if (a.share) {
    auto at_block = [&](int b) { return (int)min((long long)b * a.block_rows, (long long)a.M); };
    bool over = false;  // every block looks at all of them, and so decides alike
    for (int b = tid; b <= blocks; b += blockDim.x) {
      const int r = at_block(b), p = clamped(r);
      smem[b] = p;
      if (b < blocks) {
        const int r1 = at_block(b + 1);
        over |= (long long)clamped(r1) - p + (long long)ROW_COST * (r1 - r) > a.share;
      }
    }
    if (__syncthreads_or(over)) {
      // cut where the cost of the rows before reaches the block's part of it:
      // first among the rows looked at, then between two of them
      const int part = blockIdx.x + (tid >> 5);
      if (tid < 64 && part < blocks) {
        const long long key = part * (a.nnz + (long long)ROW_COST * a.M) / blocks;
        int lo = 0, hi = blocks;  // the first at or past it is in [lo, hi]
        auto narrow = [&](auto cost) {
          while (lo < hi) {
            const int at = lo + (int)((long long)(hi - lo) * wl / 32);
            const unsigned m = __ballot_sync(0xffffffffu, cost(at) >= key);
            const int f = m ? __ffs(m) - 1 : 32;
            const int below = __shfl_sync(0xffffffffu, at, max(f - 1, 0)), past = __shfl_sync(0xffffffffu, at, f & 31);
            if (f < 32) hi = past;
            if (f > 0) lo = below + 1;
          }
        };
        narrow([&](int b) { return smem[b] + (long long)ROW_COST * at_block(b); });
        hi = at_block(lo);
        lo = lo > 0 ? at_block(lo - 1) : 0;
        narrow([&](int r) { return clamped(r) + (long long)ROW_COST * r; });
        if (wl == 0) s_rows[tid >> 5] = lo;
      }
      __syncthreads();
      if (tid == 0) {
        // units that about fill a stage at these rows' mean length, and some
        // for every group
        const int rows = s_rows[1] - s_rows[0];
        const int nnz = clamped(s_rows[1]) - clamped(s_rows[0]);
        s_rows[2] = max(1, min(min(G, rows / NG), (int)((long long)ROW_CAP * rows / max(nnz, 1))));
      }
    }
  }
  // groups take the block's rows from a counter, so a long row holds up only
  // the group that has it
  __syncthreads();
  for (int unit = g;;) {
    const int b_hi = s_rows[1], rows = s_rows[2];
    const long long r_at = s_rows[0] + (long long)unit * rows;
    if (r_at >= b_hi) break;
    if (lane == 0) unit = atomicAdd(&s_next, 1);
    unit = __shfl_sync(mask, unit, 0, G);
    const int r0 = (int)r_at, nr = min(rows, b_hi - r0);
    // the rows' pointers, a row per lane (at most G rows at a time)
    int rs = 0, re = 0;
    if (lane < nr) {
      rs = clamped(r0 + lane);
      re = max(rs, clamped(r0 + lane + 1));
    }
    const int ps = __shfl_sync(mask, rs, 0, G);
    int pe = re;
    #pragma unroll
    for (int off = G >> 1; off > 0; off >>= 1) pe = max(pe, __shfl_xor_sync(mask, pe, off));
    const bool longs = __any_sync(mask, re - rs > a.kahan);  // a compensated row among these
    if (!ADDC) {
      unsigned todo = __ballot_sync(mask, lane < nr && re == rs);
      while (todo) {
        const int rz = r0 + ((__ffs(todo) - 1) & (G - 1));
        todo &= todo - 1;
        #pragma unroll
        for (int j = 0; j < NV; j++) {
          float z[V];
          #pragma unroll
          for (int i = 0; i < V; i++) z[i] = 0.f;
          if (act[j]) store_vec<TC, V>((TC *)a.C + (int64_t)rz * a.N + col0 + j * G * V, z, w.strm);
        }
      }
    }
    int row = r0;  // slow path: the row being summed, and whether with compensation
    bool at_start = true, kah = false;
    for (int base = ps; base < pe; base += CAP) {
      const int n = min(CAP, pe - base);
      bool bad = longs;
      int c[IT];
      float v[IT];
      #pragma unroll
      for (int k = 0; k < IT; k++) {
        const int i = k * G + lane;
        c[k] = 0;
        v[k] = 0.f;
        if (i < n) {
          c[k] = ld_idx(a.cols + base + i, w.strm);
          v[k] = load_val<T>((const T *)a.vals, (int64_t)base + i, w.strm);
        }
      }
      __syncwarp(mask);  // the last chunk's entries have been read
      #pragma unroll
      for (int k = 0; k < IT; k++) {
        const int i = k * G + lane;
        if ((unsigned)c[k] >= (unsigned)a.K) {
          c[k] = -1;
          v[k] = 0.f;  // (Inf and NaN times the zero row would not vanish)
          bad = true;
        }
        s_col[i] = c[k];
        s_val[i] = v[k];
        s_info[i] = 0;
      }
      __syncwarp(mask);
      const unsigned pos = (unsigned)(re - 1 - base);
      if (re > rs && pos < (unsigned)n) s_info[pos] = r0 + lane + 1;
      bad = __any_sync(mask, bad);
      __syncwarp(mask);  // the marks are visible to the group
      if (ADDC && !act[0]) continue;
      if (!bad) {
        at_start = true;  // for a later chunk: look the row up
        int q = 0;
        #pragma unroll 1
        for (; q + 4 <= n; q += 4) {
          RawVec<T, V> raw[4][NV];
          OldVec<TC, V> old[ADDC ? 4 : 1][NV];
          const int4 c4 = *reinterpret_cast<const int4 *>(s_col + q);
          w.fetch(raw[0], c4.x); w.fetch(raw[1], c4.y); w.fetch(raw[2], c4.z); w.fetch(raw[3], c4.w);
          const float4 v4 = *reinterpret_cast<const float4 *>(s_val + q);
          const int4 i4 = *reinterpret_cast<const int4 *>(s_info + q);
          if constexpr (ADDC) {
            w.fetch_old(old[0], i4.x); w.fetch_old(old[1], i4.y);
            w.fetch_old(old[2], i4.z); w.fetch_old(old[3], i4.w);
          }
          w.consume(raw[0], old[0], v4.x, i4.x, false);
          w.consume(raw[1], old[ADDC ? 1 : 0], v4.y, i4.y, false);
          w.consume(raw[2], old[ADDC ? 2 : 0], v4.z, i4.z, false);
          w.consume(raw[3], old[ADDC ? 3 : 0], v4.w, i4.w, false);
        }
        if (q < n) {  // the last one to three, gathered together
          RawVec<T, V> raw[3][NV];
          OldVec<TC, V> old[ADDC ? 3 : 1][NV];
          const int4 c4 = *reinterpret_cast<const int4 *>(s_col + q);  // zeros past n
          const float4 v4 = *reinterpret_cast<const float4 *>(s_val + q);
          const int4 i4 = *reinterpret_cast<const int4 *>(s_info + q);
          w.fetch(raw[0], c4.x);
          if (q + 1 < n) w.fetch(raw[1], c4.y);
          if (q + 2 < n) w.fetch(raw[2], c4.z);
          if constexpr (ADDC) {
            w.fetch_old(old[0], i4.x); w.fetch_old(old[1], i4.y); w.fetch_old(old[2], i4.z);
          }
          w.consume(raw[0], old[0], v4.x, i4.x, false);
          if (q + 1 < n) w.consume(raw[1], old[ADDC ? 1 : 0], v4.y, i4.y, false);
          if (q + 2 < n) w.consume(raw[2], old[ADDC ? 2 : 0], v4.z, i4.z, false);
        }
      } else {
        // compensated rows, or columns outside [0, K); a long row is a chain of
        // such steps, so more gathers go together
        constexpr int SU = V * NV <= 4 && !ADDC ? 8 : 4;
        #pragma unroll 1
        for (int q = 0; q < n; q += SU) {
          RawVec<T, V> raw[SU][NV];
          #pragma unroll
          for (int u = 0; u < SU; u++) {
            const int cu = q + u < n ? s_col[q + u] : -1;
            #pragma unroll
            for (int j = 0; j < NV; j++) zero_raw<T, V>(raw[u][j]);
            if (cu >= 0) w.fetch(raw[u], cu);
          }
          #pragma unroll
          for (int u = 0; u < SU; u++) {
            if (q + u >= n) break;
            if (at_start) {  // the first nonzero of a row
              while (row < r0 + nr - 1 && clamped(row + 1) <= base + q + u) row++;
              kah = clamped(row + 1) - clamped(row) > a.kahan;
              at_start = false;
            }
            const int end = s_info[q + u];
            OldVec<TC, V> old[NV];
            if constexpr (ADDC) w.fetch_old(old, end);
            w.consume(raw[u], old, s_val[q + u], end, kah);
            at_start = end != 0;
          }
        }
      }
    }
  }
}

template <typename T, typename TC>
inline void *rb_tile_ptr(int G, int V, int NV, bool addc) {
#define SS_RBT(g, v, nv)            \
  if (G == g && V == v && NV == nv) \
    return addc ? (void *)rb_tile_kernel<T, TC, g, v, nv, true> : (void *)rb_tile_kernel<T, TC, g, v, nv, false>;
#define SS_RBT_G(v) SS_RBT(8, v, 1) SS_RBT(16, v, 1)
  SS_RBT_G(2) SS_RBT(16, 2, 2)
  SS_RBT_G(4) SS_RBT(32, 4, 1)
  if constexpr (sizeof(T) == 2) { SS_RBT_G(8) SS_RBT(32, 8, 1) }
#undef SS_RBT_G
#undef SS_RBT
  return nullptr;
}

void *rb_tile_kernel_f32(int G, int V, int NV, bool addc);
void *rb_tile_kernel_bf16(int G, int V, int NV, bool addc);
void *rb_tile_kernel_bf16_f32(int G, int V, int NV, bool addc);
void *rb_tile_kernel_f16(int G, int V, int NV, bool addc);
void *rb_tile_kernel_f16_f32(int G, int V, int NV, bool addc);

}  // namespace ss
