// segment_coo over block tiles: the sequential family's default.
//
// Reference counterparts: segscan_sr_kernel and its variants
// (new-cg/include/segscan/segscan.cuh:357-815).
//
// The layout of the tile walk (eb_tile.cuh): a block takes a tile of
// consecutive elements, equal pieces go to groups of G lanes along N, an
// element whose successor has another id is marked with its id + 1 (the
// index itself says where segments end, so no search), a group's first
// segment end and its last partial go to shared memory and are combined in
// order, and segments that straddle tiles are put together by fix_kernel.  The rows of src stream in order, eight ahead where the registers
// allow.  Sum, max and mean; sums of every element with compensation where
// the tuple's chunk is longer than the threshold.
//
// Bound by DRAM: 4.62 M x 64 FP32, 225 us, 6.5 TB/s of algorithmic bytes
// (95 % of a copy; the group walk took 257 us).
#pragma once

#include "eb_tile.cuh"

namespace ss {

struct SegTileArgs {
  const void *src;
  const int32_t *index;
  float *dst;
  int2 *span;           // [tiles] segment that starts in the tile and goes on (or -1), its last tile
  int *hcnt, *tcnt;     // [tiles] elements of a tile's first / last segment (means)
  float *heads, *tails;  // [tiles * N] their partials
  int M, nnz, N, piece, tiles, phases, reduce, kahan;  // piece: elements per group
  uint32_t inv_piece;
};

enum { SEG_ADD = 0, SEG_KADD = 1, SEG_MAXV = 2 };
template <int N> struct Op { static constexpr int value = N; };

template <int OP>
__device__ __forceinline__ void seg_op(float &acc, float &comp, float x) {
  if (OP == SEG_MAXV) acc = fmaxf(acc, x);
  else if (OP == SEG_KADD) kahan_add(acc, comp, x);
  else acc += x;
}

// The last set bit of `bits` in [lo, pos), or lo - 1.
__device__ __forceinline__ int prev_bit(const uint32_t *bits, int lo, int pos) {
  for (int w = (pos - 1) >> 5; w >= lo >> 5; w--) {
    uint32_t b = bits[w];
    if (w == pos >> 5) b &= (1u << (pos & 31)) - 1u;
    if (b) return max(w * 32 + 31 - __clz(b), lo - 1);
  }
  return lo - 1;
}

template <int G, int V, int NV, bool ADDC>
__device__ __forceinline__ void seg_store(const SegTileArgs &a, int row, float (&acc)[NV][V], int count, int col0,
                                          const bool (&act)[NV], uint64_t pol) {
  if ((unsigned)row >= (unsigned)a.M) return;
  float *dst = a.dst + (int64_t)row * a.N + col0;
  #pragma unroll
  for (int j = 0; j < NV; j++) {
    if (!act[j]) continue;
    float x[V];
    #pragma unroll
    for (int i = 0; i < V; i++) x[i] = a.reduce == SS_MEAN ? acc[j][i] / (float)count : acc[j][i];
    if (ADDC) {
      float prev[V];
      load_old<float, V>(dst + j * G * V, prev);
      #pragma unroll
      for (int i = 0; i < V; i++) x[i] += prev[i];
    }
    store_vec<float, V>(dst + j * G * V, x, pol);
  }
}

// One group's piece of m elements, from element p0 of the tile.  Marks: id + 1
// at the last element of a segment, -1 where the id is outside [0, M), 0
// inside a segment; bits has a bit for each mark (a mean's lengths come from
// it at the segment ends: counting in the loop took 15 instructions a row).
// Returns the first mark.
template <typename T, int G, int V, int NV, int OP, bool MEAN, bool ADDC>
__device__ __forceinline__ int seg_walk(const SegTileArgs &a, const T *src, int m, const int32_t *sinfo,
                                        const uint32_t *bits, int p0, float *shead, float *stail, int lane, int col0, const bool (&act)[NV],
                                        uint64_t strm) {
  constexpr int U = V * NV <= 4 ? 8 : 4;
  const char *Sj[NV];
  char *Dj[NV];
  const uint32_t lds = (uint32_t)a.N * (uint32_t)sizeof(T), ldd = (uint32_t)a.N * 4u;
  #pragma unroll
  for (int j = 0; j < NV; j++) {
    // lanes past the last column repeat one that this lane (or lane 0) has
    // (accumulating, they leave the walk to the others)
    const int cj = act[j] ? col0 + j * G * V : act[0] ? col0 : col0 - lane * V;
    Sj[j] = (const char *)(src + cj);
    Dj[j] = (char *)(a.dst + cj) - ldd;
  }
  const float ident = OP == SEG_MAXV ? -INFINITY : 0.f;
  float acc[NV][V], comp[NV][V];
  #pragma unroll
  for (int j = 0; j < NV; j++)
    #pragma unroll
    for (int i = 0; i < V; i++) { acc[j][i] = ident; comp[j][i] = 0.f; }
  int hr = 0;
  auto consume = [&](const RawVec<T, V> (&raw)[NV], const OldVec<float, V> (&old)[NV], int e, int end) {
    #pragma unroll
    for (int j = 0; j < NV; j++) {
      float b[V];
      unpack_raw<T, V>(raw[j], b);
      #pragma unroll
      for (int i = 0; i < V; i++) seg_op<OP>(acc[j][i], comp[j][i], b[i]);
    }
    const int out = hr ? end : 0;  // a segment end after the first: stored here
    #pragma unroll
    for (int j = 0; j < NV; j++) {
      if (end != out) store_smem<V>(shead + j * G * V, acc[j]);
      float *d = (float *)(Dj[j] + (uint64_t)(uint32_t)end * ldd);
      if (MEAN && out > 0) {
        asm volatile("");  // stays a branch; in place, so that no row pays for copies
        const float len = (float)(p0 + e - prev_bit(bits, p0, p0 + e));
        #pragma unroll
        for (int i = 0; i < V; i++) acc[j][i] = acc[j][i] / len;
      }
      if (ADDC) {
        float prev[V];
        unpack_old<float, V>(old[j], prev);
        #pragma unroll
        for (int i = 0; i < V; i++) acc[j][i] = out > 0 ? acc[j][i] + prev[i] : acc[j][i];
      }
      store_vec_if<float, V>(d, acc[j], strm, out);
      #pragma unroll
      for (int i = 0; i < V; i++) {
        acc[j][i] = end ? ident : acc[j][i];
        comp[j][i] = end ? 0.f : comp[j][i];
      }
    }
    hr = hr ? hr : end;
  };
  auto load_row = [&](RawVec<T, V> (&raw)[NV], int e) {
    #pragma unroll
    for (int j = 0; j < NV; j++) load_raw<T, V>((const T *)(Sj[j] + (uint64_t)(uint32_t)e * lds), raw[j], strm);
  };
  auto load_prev = [&](OldVec<float, V> (&old)[NV], int end) {
    #pragma unroll
    for (int j = 0; j < NV; j++)
      load_old_if<float, V>((const float *)(Dj[j] + (uint64_t)(uint32_t)end * ldd), old[j], end);
  };
  int q = 0;
  #pragma unroll 1
  for (; q + U <= m; q += U) {
    RawVec<T, V> raw[U][NV];
    OldVec<float, V> old[ADDC ? U : 1][NV];
    #pragma unroll
    for (int u = 0; u < U; u++) load_row(raw[u], q + u);
    int is[U];
    #pragma unroll
    for (int u = 0; u < U; u += 4) {
      const int4 i4 = *reinterpret_cast<const int4 *>(sinfo + q + u);
      is[u] = i4.x; is[u + 1] = i4.y; is[u + 2] = i4.z; is[u + 3] = i4.w;
    }
    if constexpr (ADDC) {
      #pragma unroll
      for (int u = 0; u < U; u++) load_prev(old[u], is[u]);
    }
    #pragma unroll
    for (int u = 0; u < U; u++) consume(raw[u], old[ADDC ? u : 0], q + u, is[u]);
  }
  #pragma unroll 1
  for (; q < m; q++) {
    RawVec<T, V> raw[NV];
    OldVec<float, V> old[NV];
    load_row(raw, q);
    if constexpr (ADDC) load_prev(old, sinfo[q]);
    consume(raw, old, q, sinfo[q]);
  }
  #pragma unroll
  for (int j = 0; j < NV; j++) store_smem<V>(stail + j * G * V, acc[j]);
  return hr;
}

template <typename T, int G, int V, int NV, bool ADDC>
__global__ void __launch_bounds__(TW_T, (ADDC || V * NV > 4 ? 3 : 4)) seg_tile_kernel(SegTileArgs a) {
  constexpr int NG = TW_T / G, E = V * NV, COLS = G * E, EW = (NG + 31) / 32;
  extern __shared__ __align__(16) int32_t smem[];
  __shared__ int s_last;  // last tile of the segment that leaves this one
  __shared__ uint32_t s_ends[EW];
  __shared__ int s_hn[NG], s_tn[NG];
  const int S = a.piece, TILE = NG * S;
  int32_t *s_info = smem;                        // [NG][S + 4]
  float *s_head = (float *)(smem + NG * (S + 4));  // [NG][COLS]
  float *s_tail = s_head + NG * COLS;
  uint32_t *s_bits = (uint32_t *)(s_tail + NG * COLS);  // [TILE / 32] elements that end a segment
  const int tid = threadIdx.x, wl = tid & 31;
  const int phase = blockIdx.x / a.tiles;
  const int tile = blockIdx.x - phase * a.tiles;
  const int ts = tile * TILE;
  const int n = min(TILE, a.nnz - ts), te = ts + n;
  const uint64_t strm = policy_stream();
  const int lane = tid & (G - 1), g = tid / G;
  const int col0 = phase * COLS + lane * V;
  bool act[NV];
  #pragma unroll
  for (int j = 0; j < NV; j++) act[j] = col0 + j * G * V < a.N;
  if (tid < EW) s_ends[tid] = 0;
  grid_dependents_launch();  // fix_kernel, which waits for this grid

  // segment ends, and the empty segments after each of them
  auto zero_gap = [&](int lo, int hi) {  // the whole warp; lo, hi uniform
    lo = max(lo, 0);
    hi = min(hi, a.M - 1);
    float z[NV][V];
    clear<V, NV>(z);
    for (int r = lo + wl / G; r <= hi; r += 32 / G) {
      float *d = a.dst + (int64_t)r * a.N + col0;
      #pragma unroll
      for (int j = 0; j < NV; j++)
        if (act[j]) store_vec<float, V>(d + j * G * V, z[j], strm);
    }
  };
  for (int e0 = 0; e0 < TILE; e0 += TW_T) {
    const int e = e0 + tid, p = ts + e;
    int mark = 0, id = 0, next = 0;
    bool gap = false;
    if (e < n) {
      id = ld_idx(a.index + p, strm);
      next = p + 1 < a.nnz ? ld_idx(a.index + p + 1, strm) : a.M;
      const bool end = p + 1 >= a.nnz || next != id;
      mark = !end ? 0 : (unsigned)id < (unsigned)a.M ? id + 1 : -1;
      gap = !ADDC && next > id && (unsigned)next - (unsigned)id > 1u;
    }
    if (e < TILE) s_info[e + 4 * piece_of(e, a.inv_piece)] = mark;
    const unsigned ends = __ballot_sync(0xffffffffu, mark != 0);
    if (wl == 0 && e < TILE) s_bits[e >> 5] = ends;
    unsigned todo = __ballot_sync(0xffffffffu, gap);
    while (todo) {
      const int s = __ffs(todo) - 1;
      todo &= todo - 1;
      zero_gap(__shfl_sync(0xffffffffu, id, s) + 1, __shfl_sync(0xffffffffu, next, s) - 1);
    }
  }
  if (!ADDC && tile == 0 && tid < 32) zero_gap(0, __ldg(a.index) - 1);
  const int r_in = __ldg(a.index + ts), r_out = __ldg(a.index + te - 1);
  const bool has_head = ts > 0 && __ldg(a.index + ts - 1) == r_in;
  const bool more = te < a.nnz && __ldg(a.index + te) == r_out;
  // (a tile inside one segment does not own it, and needs no search)
  if (tid >= 32 && tid < 64 && more && !(has_head && r_in == r_out)) {
    // last tile whose first id is still r_out: among the next 32, else by a
    // 32-way search (ids ascend), so that a segment of any length takes a few
    // steps: the first tile with another id is in [lo, hi].  (One segment of
    // 30 M elements, N = 64: 10.7 ms with 32 tiles a step all the way and four
    // heads in flight in fix_kernel, 3.3 ms now.)
    int lo = tile + 1, hi = a.tiles, step = 1;
    while (lo < hi) {
      const long long j = lo + (long long)wl * step;
      const unsigned m = __ballot_sync(0xffffffffu, j >= hi || __ldg(a.index + j * TILE) != r_out);
      const int f = m ? __ffs(m) - 1 : 32;
      if (f < 32) hi = (int)min((long long)hi, lo + (long long)f * step);
      if (f > 0) lo = (int)min((long long)hi, lo + (long long)(f - 1) * step + 1);
      step = (hi - lo + 31) / 32;
    }
    if (wl == 0) s_last = lo - 1;
  }
  __syncthreads();
  const int m = min(max(n - g * S, 0), S);
  const T *src = (const T *)a.src + (int64_t)(ts + g * S) * a.N;
  const int32_t *info = s_info + g * (S + 4);
  float *shead = s_head + g * COLS + lane * V, *stail = s_tail + g * COLS + lane * V;
  int hr = 0;
  const bool is_max = a.reduce == SS_MAX;
  auto walk = [&](auto op, auto mean) {
    return seg_walk<T, G, V, NV, decltype(op)::value, decltype(mean)::value, ADDC>(a, src, m, info, s_bits, g * S, shead,
                                                                                   stail, lane, col0, act, strm);
  };
  // (accumulating is defined for sums only)
  if (ADDC && !act[0]) hr = 0;
  else if (ADDC || a.reduce == SS_SUM) hr = a.kahan ? walk(Op<SEG_KADD>(), Op<0>()) : walk(Op<SEG_ADD>(), Op<0>());
  else if constexpr (!ADDC) {
    if (is_max) hr = walk(Op<SEG_MAXV>(), Op<0>());
    else hr = a.kahan ? walk(Op<SEG_KADD>(), Op<1>()) : walk(Op<SEG_ADD>(), Op<1>());
  }
  if (lane == 0) {
    if (a.reduce == SS_MEAN) {
      // elements up to the first segment end, and after the last one
      const int last = prev_bit(s_bits, g * S, g * S + m);
      int first = g * S;
      while (first <= last && !(s_bits[first >> 5] >> (first & 31) & 1u)) first++;
      s_hn[g] = first + 1 - g * S;
      s_tn[g] = g * S + m - 1 - last;
    }
    if (hr) atomicOr(s_ends + (g >> 5), 1u << (g & 31));
  }
  __syncthreads();
  auto prev_end = [&](int x) {  // the last group before x with a segment end, or -1
    int w = x >> 5;
    uint32_t b = w < EW ? s_ends[w] & ((1u << (x & 31)) - 1u) : 0u;
    while (b == 0 && w > 0) b = s_ends[--w];
    return b ? w * 32 + 31 - __clz(b) : -1;
  };
  // a segment's pieces in order: tails of groups [s, x), then the head of x
  auto chain = [&](int s, int x, bool head, float (&acc)[NV][V], int &count) {
    count = head ? s_hn[x] : 0;
    for (int k = max(s, 0); k < x; k++) count += s_tn[k];
    #pragma unroll
    for (int j = 0; j < NV; j++) {
      const int c = lane * V + j * G * V, k0 = max(s, 0), k1 = x + (head ? 1 : 0);
      auto at = [&](int k) { return (k < x ? s_tail + k * COLS : s_head + x * COLS) + c; };
      if (is_max) {
        #pragma unroll
        for (int i = 0; i < V; i++) acc[j][i] = -INFINITY;
        for (int k = k0; k < k1; k++)
          #pragma unroll
          for (int i = 0; i < V; i++) acc[j][i] = fmaxf(acc[j][i], at(k)[i]);
      } else {
        sum_pieces<V>(k0, k1, at, acc[j]);
      }
    }
  };
  auto to_slot = [&](float *slots, int *counts, float (&acc)[NV][V], int count) {
    float *d = slots + (int64_t)tile * a.N + col0;
    #pragma unroll
    for (int j = 0; j < NV; j++)
      if (act[j]) store_vec<float, V>(d + j * G * V, acc[j], strm);
    if (lane == 0 && a.reduce == SS_MEAN) counts[tile] = count;  // every phase writes the same
  };
  float acc[NV][V];
  int count;
  if (hr) {
    const int s = prev_end(g);
    chain(s, g, true, acc, count);
    if (s < 0 && has_head) {  // the segment that entered the tile ends
      to_slot(a.heads, a.hcnt, acc, count);
    } else if (hr > 0) {
      seg_store<G, V, NV, ADDC>(a, hr - 1, acc, count, col0, act, strm);
    }
  }
  if (g == 0) {
    int2 span = make_int2(-1, 0);
    if (more) {  // the last segment goes on
      const int s = prev_end(NG);
      chain(s, NG, false, acc, count);
      const bool whole = s < 0 && has_head;  // the tile lies inside one segment
      to_slot(whole ? a.heads : a.tails, whole ? a.hcnt : a.tcnt, acc, count);
      if (!whole) span = make_int2(r_out, s_last);
    }
    if (lane == 0) a.span[tile] = span;  // every phase writes the same
  }
}

template <typename T>
inline void *seg_tile_ptr(int G, int V, int NV, bool addc) {
#define SS_SEGT(g, v, nv)           \
  if (G == g && V == v && NV == nv) \
    return addc ? (void *)seg_tile_kernel<T, g, v, nv, true> : (void *)seg_tile_kernel<T, g, v, nv, false>;
#define SS_SEGT_G(v) SS_SEGT(1, v, 1) SS_SEGT(2, v, 1) SS_SEGT(4, v, 1) SS_SEGT(8, v, 1) SS_SEGT(16, v, 1)
  SS_SEGT_G(1) SS_SEGT(16, 1, 2) SS_SEGT(16, 1, 3) SS_SEGT(16, 1, 4)
  SS_SEGT_G(2) SS_SEGT(16, 2, 2)
  SS_SEGT_G(4) SS_SEGT(32, 4, 1)
  if constexpr (sizeof(T) == 2) { SS_SEGT_G(8) SS_SEGT(32, 8, 1) }
#undef SS_SEGT_G
#undef SS_SEGT
  return nullptr;
}

void *seg_tile_kernel_f32(int G, int V, int NV, bool addc);
void *seg_tile_kernel_bf16(int G, int V, int NV, bool addc);
void *seg_tile_kernel_f16(int G, int V, int NV, bool addc);

}  // namespace ss
