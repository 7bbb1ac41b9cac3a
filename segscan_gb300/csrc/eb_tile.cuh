// Element-balanced SpMM over block tiles: the ebsr walk of one matrix and of
// the batched launch.
//
// Reference counterpart: csrspmm_rowcaching_nnzbalance_cg_kernel
// (test-cg/include/spmm/spmm_cg.cuh:376-551).
//
// A block takes a tile of consecutive nonzeros, cut into equal pieces, one
// per group of G lanes laid along N (E = V * NV columns a
// lane), and
//  * the tile's columns and values go to shared memory with plain 16-byte
//    loads, each piece padded by four words so that the groups of a warp
//    read their streams without bank conflicts;
//  * the rows that start in the tile (row_start, or a warp search) mark their
//    last nonzero with row + 1 and write the empty rows; no nonzero is
//    searched or labelled one by one;
//  * a group walks its piece four nonzeros at a time: four B rows gathered
//    together, four multiply-adds, and at a marked nonzero the finished row
//    is stored by a predicated store, so groups of one warp do not diverge
//    at their row ends;
//  * a group's first row end may belong to a row that an earlier group
//    started: it goes to shared memory with every group's last partial, and
//    the pieces of a row are added in order after the walk;
//  * rows that straddle tiles leave their parts in one head and one tail slot
//    per tile; a small kernel, launched to overlap the walk's end, adds them
//    up (fix_kernel in eb_tile.cu).  Counting the tiles in with atomics and
//    letting the last one add cost every block 5 to 12 K of its 60 K cycles,
//    with nothing else of the block in flight.
// Nonzeros of rows longer than kahan_threshold are summed with compensation:
// warps that hold any take a second instantiation of the walk, which also
// skips columns outside [0, K).
//
// What bounds it (power-law 1e6 x 1e6, 4.6 M nonzeros): at N = 64 FP32 the
// gathered rows, 1.16 GB of DRAM traffic at 5.96 TB/s (195 us); with BF16
// storage 0.59 GB at 4.2 TB/s and 65 instructions per 32 gathered vectors
// (142 us, issue 48 % busy), at N = 4 the latency of a tile's steps (61 us,
// issue 35 % busy, 40 % of the warp slots in use).
#pragma once

#include "eb_common.cuh"
#include "internal.h"

namespace ss {

constexpr int TW_T = 256;  // threads per block

// One matrix of a launch (16-byte multiple: copied by 16-byte words).
struct __align__(16) TileProb {
  const int32_t *indptr, *cols;
  const void *vals;  // null = ones
  const void *B;
  void *C;
  const int32_t *perm;       // value of nonzero q is vals[perm[q]] in type perm_dtype, or null: vals[q]
  const int32_t *row_start;  // [tiles + 1] first row starting at or after each tile, or null: searched
  int2 *span;                // [tiles] row that starts in the tile and goes on (or -1), its last tile
  float *heads, *tails;      // [tiles * N] partials of a tile's first / last row
  int M, K, nnz;
  int piece;       // nonzeros per group, a multiple of eight
  uint32_t inv_piece;
  int item_begin;  // first block of this matrix (batched)
  int wide;        // columns and values may be loaded 16 bytes at a time
  int index;       // host: the matrix's place in its batch
  int perm_dtype;
};

struct TileArgs {
  TileProb p;              // the matrix (single launch)
  const TileProb *probs;   // batched: the matrices ...
  const int32_t *item_prob;  // ... and the matrix of each block; null = single
  int items, phases;       // blocks per column phase
  int N, accumulate, kahan;
  float keep_frac;
};

// Shared memory of a block, in words after the TileProb.
struct TileSmem {
  int col, val, info, head, tail, kb, ends, total;
};
__host__ __device__ inline TileSmem tile_smem(int G, int E, int piece) {
  const int NG = TW_T / G, words = NG * (piece + 4);
  TileSmem s;
  int o = (int)sizeof(TileProb) / 4;
  s.col = o; o += words;
  s.val = o; o += words;
  s.info = o; o += words;
  s.head = o; o += TW_T * E;
  s.tail = o; o += TW_T * E;
  s.kb = o; o += (NG * piece + 31) / 32;
  s.ends = o; o += (NG + 31) / 32;
  s.total = o;
  return s;
}

// e / piece for e below 2^16 and inv = ceil(2^32 / piece)
__device__ __forceinline__ int piece_of(int e, uint32_t inv) { return (int)__umulhi((uint32_t)e, inv); }
inline uint32_t inverse_of(int piece) { return (uint32_t)(((1ull << 32) + piece - 1) / piece); }

// Waits for the kernels that this one was launched to overlap (programmatic
// stream serialization); nothing to wait for in an ordinary launch.
__device__ __forceinline__ void grid_dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// The next kernel of the stream, if launched so, may start its blocks.
__device__ __forceinline__ void grid_dependents_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <int V>
__device__ __forceinline__ void store_smem(float *p, const float (&v)[V]) {
  if constexpr (V % 4 == 0) {
    #pragma unroll
    for (int i = 0; i < V; i += 4)
      *reinterpret_cast<float4 *>(p + i) = make_float4(v[i], v[i + 1], v[i + 2], v[i + 3]);
  } else if constexpr (V == 2) {
    *reinterpret_cast<float2 *>(p) = make_float2(v[0], v[1]);
  } else {
    p[0] = v[0];
  }
}

template <int V>
__device__ __forceinline__ void load_smem(const float *p, float (&v)[V]) {
  if constexpr (V % 4 == 0) {
    #pragma unroll
    for (int i = 0; i < V; i += 4) {
      const float4 x = *reinterpret_cast<const float4 *>(p + i);
      v[i] = x.x; v[i + 1] = x.y; v[i + 2] = x.z; v[i + 3] = x.w;
    }
  } else if constexpr (V == 2) {
    const float2 x = *reinterpret_cast<const float2 *>(p);
    v[0] = x.x; v[1] = x.y;
  } else {
    v[0] = p[0];
  }
}

// V elements of the output, widened (plain loads: the row is rewritten here).
template <typename TC, int V>
__device__ __forceinline__ void load_old(const TC *p, float (&out)[V]) {
  if constexpr (V * sizeof(TC) > 16) {
    constexpr int H = V / 2;
    float lo[H], hi[H];
    load_old<TC, H>(p, lo);
    load_old<TC, H>(p + H, hi);
    #pragma unroll
    for (int i = 0; i < H; i++) { out[i] = lo[i]; out[H + i] = hi[i]; }
  } else {
    RawVec<TC, V> r;
    if constexpr (V * sizeof(TC) == 16) {
      const uint4 x = *reinterpret_cast<const uint4 *>(p);
      r.w[0] = x.x; r.w[1] = x.y; r.w[2] = x.z; r.w[3] = x.w;
    } else if constexpr (V * sizeof(TC) == 8) {
      const uint2 x = *reinterpret_cast<const uint2 *>(p);
      r.w[0] = x.x; r.w[1] = x.y;
    } else if constexpr (V * sizeof(TC) == 4) {
      r.w[0] = *reinterpret_cast<const uint32_t *>(p);
    } else {
      r.w[0] = *reinterpret_cast<const uint16_t *>(p);
    }
    unpack_raw<TC, V>(r, out);
  }
}

// One predicated instruction each (where on > 0), so that groups of one warp
// do not branch apart where only some of them end a row.
__device__ __forceinline__ void st_if(void *p, const uint32_t (&w)[4], uint64_t pol, int on) {
  asm volatile("{\n .reg .pred p;\n setp.gt.s32 p, %6, 0;\n"
               " @p st.global.L2::cache_hint.v4.u32 [%0], {%1, %2, %3, %4}, %5;\n}" ::"l"(p), "r"(w[0]), "r"(w[1]),
               "r"(w[2]), "r"(w[3]), "l"(pol), "r"(on) : "memory");
}
__device__ __forceinline__ void st_if(void *p, const uint32_t (&w)[2], uint64_t pol, int on) {
  asm volatile("{\n .reg .pred p;\n setp.gt.s32 p, %4, 0;\n"
               " @p st.global.L2::cache_hint.v2.u32 [%0], {%1, %2}, %3;\n}" ::"l"(p), "r"(w[0]), "r"(w[1]), "l"(pol),
               "r"(on) : "memory");
}
__device__ __forceinline__ void st_if(void *p, const uint32_t (&w)[1], uint64_t pol, int on) {
  asm volatile("{\n .reg .pred p;\n setp.gt.s32 p, %3, 0;\n @p st.global.L2::cache_hint.u32 [%0], %1, %2;\n}" ::
               "l"(p), "r"(w[0]), "l"(pol), "r"(on) : "memory");
}
__device__ __forceinline__ void st16_if(void *p, uint16_t w, uint64_t pol, int on) {
  asm volatile("{\n .reg .pred p;\n setp.gt.s32 p, %3, 0;\n @p st.global.L2::cache_hint.u16 [%0], %1, %2;\n}" ::
               "l"(p), "h"(w), "l"(pol), "r"(on) : "memory");
}
__device__ __forceinline__ void ld_if(const void *p, uint32_t (&w)[4], int on) {
  asm volatile("{\n .reg .pred p;\n setp.gt.s32 p, %5, 0;\n @p ld.global.v4.u32 {%0, %1, %2, %3}, [%4];\n}"
               : "+r"(w[0]), "+r"(w[1]), "+r"(w[2]), "+r"(w[3]) : "l"(p), "r"(on) : "memory");
}
__device__ __forceinline__ void ld_if(const void *p, uint32_t (&w)[2], int on) {
  asm volatile("{\n .reg .pred p;\n setp.gt.s32 p, %3, 0;\n @p ld.global.v2.u32 {%0, %1}, [%2];\n}"
               : "+r"(w[0]), "+r"(w[1]) : "l"(p), "r"(on) : "memory");
}
__device__ __forceinline__ void ld_if(const void *p, uint32_t (&w)[1], int on) {
  asm volatile("{\n .reg .pred p;\n setp.gt.s32 p, %2, 0;\n @p ld.global.u32 %0, [%1];\n}"
               : "+r"(w[0]) : "l"(p), "r"(on) : "memory");
}
__device__ __forceinline__ void ld16_if(const void *p, uint32_t &w, int on) {
  uint16_t h = 0;
  asm volatile("{\n .reg .pred p;\n setp.gt.s32 p, %2, 0;\n @p ld.global.u16 %0, [%1];\n}"
               : "+h"(h) : "l"(p), "r"(on) : "memory");
  w = h;
}
template <typename T, int V>
__device__ __forceinline__ void store_vec_if(T *p, const float (&v)[V], uint64_t pol, int on) {
  if constexpr (V * sizeof(T) > 16) {
    constexpr int H = V / 2;
    float lo[H], hi[H];
    #pragma unroll
    for (int i = 0; i < H; i++) { lo[i] = v[i]; hi[i] = v[H + i]; }
    store_vec_if<T, H>(p, lo, pol, on);
    store_vec_if<T, H>(p + H, hi, pol, on);
  } else if constexpr (V * sizeof(T) == 2) {
    const T h = Elem<T>::from_f(v[0]);
    st16_if(p, *reinterpret_cast<const uint16_t *>(&h), pol, on);
  } else {
    uint32_t w[V * sizeof(T) / 4];
    #pragma unroll
    for (int i = 0; i < (int)(V * sizeof(T) / 4); i++) {
      if constexpr (sizeof(T) == 4) w[i] = __float_as_uint(v[i]);
      else w[i] = pack2(v[2 * i], v[2 * i + 1], (T *)nullptr);
    }
    st_if(p, w, pol, on);
  }
}
// V elements of the output as words, kept packed until they are added.
template <typename T, int V>
struct OldVec {
  static constexpr int B = V * (int)sizeof(T), W = B > 16 ? 4 : (B + 3) / 4, P = (B + 15) / 16;
  uint32_t w[P][W];
};
template <typename T, int V>
__device__ __forceinline__ void load_old_if(const T *p, OldVec<T, V> &o, int on) {
  #pragma unroll
  for (int k = 0; k < OldVec<T, V>::P; k++) {
    const char *q = (const char *)p + 16 * k;
    if constexpr (OldVec<T, V>::B == 2) ld16_if(q, o.w[k][0], on);
    else ld_if(q, o.w[k], on);
  }
}
template <typename T, int V>
__device__ __forceinline__ void unpack_old(const OldVec<T, V> &o, float (&out)[V]) {
  constexpr int VP = V / OldVec<T, V>::P;
  #pragma unroll
  for (int k = 0; k < OldVec<T, V>::P; k++) {
    RawVec<T, VP> r;
    float x[VP];
    #pragma unroll
    for (int i = 0; i < OldVec<T, V>::W; i++) r.w[i] = o.w[k][i];
    unpack_raw<T, VP>(r, x);
    #pragma unroll
    for (int i = 0; i < VP; i++) out[k * VP + i] = x[i];
  }
}

template <int V, int NV>
__device__ __forceinline__ void clear(float (&x)[NV][V]) {
  #pragma unroll
  for (int j = 0; j < NV; j++)
    #pragma unroll
    for (int i = 0; i < V; i++) x[j][i] = 0.f;
}

// acc = pieces k0 .. k1 - 1 (at(k): V partials in shared memory) added in order
// with compensation.  A sum that is not finite is added up again without, which
// gives its Inf or NaN: checking every step instead costs 5 % at N = 4, where
// the chain of a few pieces is a row's longest (1e6 power-law 63.5 -> 67.2 us).
template <int V, typename At>
__device__ __forceinline__ void sum_pieces(int k0, int k1, At at, float (&acc)[V]) {
  float comp[V], x[V];
  #pragma unroll
  for (int i = 0; i < V; i++) acc[i] = comp[i] = 0.f;
  for (int k = k0; k < k1; k++) {
    load_smem<V>(at(k), x);
    #pragma unroll
    for (int i = 0; i < V; i++) kahan_step(acc[i], comp[i], __fsub_rn(x[i], comp[i]));
  }
  bool finite = true;
  #pragma unroll
  for (int i = 0; i < V; i++) finite &= fabsf(acc[i]) < INFINITY;
  if (finite) return;
  #pragma unroll
  for (int i = 0; i < V; i++) comp[i] = 0.f;
  for (int k = k0; k < k1; k++) {
    load_smem<V>(at(k), x);
    #pragma unroll
    for (int i = 0; i < V; i++) comp[i] += x[i];
  }
  #pragma unroll
  for (int i = 0; i < V; i++) acc[i] = fabsf(acc[i]) < INFINITY ? acc[i] : comp[i];
}

// Row `row` of C = acc (+ the old row in accumulate mode), this lane's columns.
template <typename TC, int G, int V, int NV, bool ADDC>
__device__ __forceinline__ void tile_store(const TileProb &p, int N, int row, const float (&acc)[NV][V],
                                           int col0, const bool (&act)[NV], uint64_t pol) {
  if ((unsigned)row >= (unsigned)p.M) return;
  TC *dst = (TC *)p.C + (int64_t)row * N + col0;
  #pragma unroll
  for (int j = 0; j < NV; j++) {
    if (!act[j]) continue;
    TC *d = dst + j * G * V;
    float x[V];
    #pragma unroll
    for (int i = 0; i < V; i++) x[i] = acc[j][i];
    if (ADDC) {
      float prev[V];
      load_old<TC, V>(d, prev);
      #pragma unroll
      for (int i = 0; i < V; i++) x[i] += prev[i];
    }
    store_vec<TC, V>(d, x, pol);
  }
}

// One group's piece: S nonzeros from its staged columns, values and row-end
// marks.  The first row end goes to shead (its row + 1 is returned, 0 when
// the piece has none), what follows the last one to stail, the others to C.
template <typename T, typename TC, int G, int V, int NV, bool SLOW, bool ADDC>
__device__ __forceinline__ int tile_walk(const TileProb &p, int N, int S, const int32_t *scol,
                                         const float *sval, const int32_t *sinfo, const uint32_t *kb, int p0,
                                         float *shead, float *stail, int lane, int col0, const bool (&act)[NV],
                                         uint64_t keep, uint64_t strm) {
  const char *Bj[NV];
  char *Cj[NV];
  const uint32_t ldb = (uint32_t)N * (uint32_t)sizeof(T), ldc = (uint32_t)N * (uint32_t)sizeof(TC);
  #pragma unroll
  for (int j = 0; j < NV; j++) {
    // a lane past the last column repeats a column that it (or lane 0)
    // computes too and stores the same value to the same place: no predicate
    // per load and store (accumulating, such lanes leave the walk to the
    // others: they could read a row after another lane's store)
    const int cj = act[j] ? col0 + j * G * V : act[0] ? col0 : col0 - lane * V;
    Bj[j] = (const char *)((const T *)p.B + cj);
    Cj[j] = (char *)((TC *)p.C + cj) - ldc;  // marks hold row + 1
  }
  float acc[NV][V], comp[NV][V];
  clear<V, NV>(acc);
  clear<V, NV>(comp);
  int hr = 0;
  RawVec<T, V> raw[4][NV];
  // accumulating: the rows of C that end among the four nonzeros, loaded with
  // their B rows so that a row end does not wait for memory
  OldVec<TC, V> old[ADDC ? 4 : 1][NV];
  auto fetch = [&](int u, int c) {
    #pragma unroll
    for (int j = 0; j < NV; j++) {
      if (!SLOW || c >= 0) load_raw<T, V>((const T *)(Bj[j] + (uint64_t)(uint32_t)c * ldb), raw[u][j], keep);
      else zero_raw<T, V>(raw[u][j]);
    }
  };
  auto consume = [&](int u, float v, int end, bool kah) {
    #pragma unroll
    for (int j = 0; j < NV; j++) {
      float b[V];
      unpack_raw<T, V>(raw[u][j], b);
      if (SLOW && kah) {
        kahan_fma<V>(acc[j], comp[j], v, b);
      } else {
        #pragma unroll
        for (int i = 0; i < V; i++) acc[j][i] = fmaf(v, b[i], acc[j][i]);
      }
    }
    const bool first = end != 0 && hr == 0; const int out = end != 0 && hr != 0;
    #pragma unroll
    for (int j = 0; j < NV; j++) {
      if (first) store_smem<V>(shead + j * G * V, acc[j]);
      TC *d = (TC *)(Cj[j] + (uint64_t)(uint32_t)end * ldc);
      if (ADDC) {
        float x[V];
        unpack_old<TC, V>(old[u][j], x);
        #pragma unroll
        for (int i = 0; i < V; i++) x[i] += acc[j][i];
        store_vec_if<TC, V>(d, x, strm, out);
      } else {
        store_vec_if<TC, V>(d, acc[j], strm, out);
      }
      #pragma unroll
      for (int i = 0; i < V; i++) {
        acc[j][i] = end ? 0.f : acc[j][i];
        if (SLOW) comp[j][i] = end ? 0.f : comp[j][i];
      }
    }
    hr = first ? end : hr;
  };
  #pragma unroll 1
  for (int q = 0; q < S; q += 4) {
    const int4 c4 = *reinterpret_cast<const int4 *>(scol + q);
    fetch(0, c4.x); fetch(1, c4.y); fetch(2, c4.z); fetch(3, c4.w);
    const float4 v4 = *reinterpret_cast<const float4 *>(sval + q);
    const int4 i4 = *reinterpret_cast<const int4 *>(sinfo + q);
    if constexpr (ADDC) {
      const int is[4] = {i4.x, i4.y, i4.z, i4.w};
      #pragma unroll
      for (int u = 0; u < 4; u++)
        #pragma unroll
        for (int j = 0; j < NV; j++)
          load_old_if<TC, V>((const TC *)(Cj[j] + (uint64_t)(uint32_t)is[u] * ldc), old[u][j], is[u]);
    }
    const uint32_t k4 = SLOW ? kb[(p0 + q) >> 5] >> ((p0 + q) & 31) : 0u;
    consume(0, v4.x, i4.x, k4 & 1u);
    consume(1, v4.y, i4.y, k4 & 2u);
    consume(2, v4.z, i4.z, k4 & 4u);
    consume(3, v4.w, i4.w, k4 & 8u);
  }
  #pragma unroll
  for (int j = 0; j < NV; j++) store_smem<V>(stail + j * G * V, acc[j]);
  return hr;
}

// Blocks per SM the registers are bounded for.  Five (48 registers) where a
// lane holds one FP32 vector and the gathered rows are long (N = 64: 208 us
// against 214 at four); at small N and with wider lanes the bound costs more
// in spills than the fifth block gives (N = 4: 61 us at four, 74 at five;
// BF16 N = 64: 157 and 225).  Accumulating needs four old rows beside the
// gathered ones.
template <typename T, int G, int V, int NV, bool ADDC>
constexpr int tile_min_blocks() {
  return ADDC ? (V * NV > 4 ? 2 : 3) : sizeof(T) == 4 && V == 4 && G >= 8 ? 5 : 4;
}

template <typename T, typename TC, int G, int V, int NV, bool ADDC>
__global__ void __launch_bounds__(TW_T, (tile_min_blocks<T, G, V, NV, ADDC>())) eb_tile_kernel(TileArgs a) {
  constexpr int NG = TW_T / G, E = V * NV, COLS = G * E, EW = (NG + 31) / 32;
  extern __shared__ __align__(16) int32_t smem[];
  const int tid = threadIdx.x, wl = tid & 31;
  const int phase = blockIdx.x / a.items;
  const int item = blockIdx.x - phase * a.items;
  if (tid < (int)sizeof(TileProb) / 16) {
    const TileProb *src = a.item_prob ? a.probs + __ldg(a.item_prob + item) : &a.p;
    reinterpret_cast<int4 *>(smem)[tid] = reinterpret_cast<const int4 *>(src)[tid];
  }
  __syncthreads();
  const TileProb &p = *reinterpret_cast<const TileProb *>(smem);
  grid_dependents_launch();  // fix_kernel, which waits for this grid
  const int S = p.piece, TILE = NG * S;
  const TileSmem L = tile_smem(G, E, S);
  int32_t *s_col = smem + L.col, *s_info = smem + L.info;
  float *s_val = (float *)(smem + L.val), *s_head = (float *)(smem + L.head), *s_tail = (float *)(smem + L.tail);
  uint32_t *s_kb = (uint32_t *)(smem + L.kb), *s_ends = (uint32_t *)(smem + L.ends);
  __shared__ int s_rows[2];
  const int tile = item - p.item_begin;
  const uint64_t keep = policy_keep(a.keep_frac), strm = policy_stream();
  const int lane = tid & (G - 1), g = tid / G;
  const int col0 = phase * COLS + lane * V;
  bool act[NV];
  #pragma unroll
  for (int j = 0; j < NV; j++) act[j] = col0 + j * G * V < a.N;

  const int ts = tile * TILE;
  const int n = min(TILE, p.nnz - ts), te = ts + n;
  // the tile's columns and values, on their way while the tile's rows are
  // found (and, in a single launch, while the kernel that finds them runs)
  constexpr int LOADS = 2;  // a tile is at most 2048 nonzeros
  int c[LOADS][4];
  float v[LOADS][4];
  #pragma unroll
  for (int k = 0; k < LOADS; k++) {
    const int e = (tid + k * TW_T) * 4;
    #pragma unroll
    for (int i = 0; i < 4; i++) { c[k][i] = -1; v[k][i] = 1.f; }
    if (e >= n) continue;
    if (sizeof(T) == 4 && p.perm) {  // values in another order and type
      #pragma unroll
      for (int i = 0; i < 4; i++) {
        if (e + i >= n) continue;
        c[k][i] = ld_idx(p.cols + ts + e + i, strm);
        const int q = ld_idx(p.perm + ts + e + i, strm);
        v[k][i] = (unsigned)q >= (unsigned)p.nnz ? 0.f
                  : p.perm_dtype == SS_F32       ? load_val<float>((const float *)p.vals, q, keep)
                  : p.perm_dtype == SS_BF16      ? load_val<__nv_bfloat16>((const __nv_bfloat16 *)p.vals, q, keep)
                                                 : load_val<__half>((const __half *)p.vals, q, keep);
      }
    } else if (p.wide && e + 4 <= n) {
      const uint4 x = ld_u128(p.cols + ts + e, strm);
      c[k][0] = x.x; c[k][1] = x.y; c[k][2] = x.z; c[k][3] = x.w;
      if (p.vals) load_vec<T, 4>((const T *)p.vals + ts + e, v[k], strm);
    } else {
      #pragma unroll
      for (int i = 0; i < 4; i++) {
        if (e + i >= n) continue;
        c[k][i] = ld_idx(p.cols + ts + e + i, strm);
        v[k][i] = load_val<T>((const T *)p.vals, (int64_t)ts + e + i, strm);
      }
    }
  }
  // rows that start in the tile: [rlo, rhi)
  int rlo, rhi;
  if (p.row_start) {
    grid_dependency_wait();  // tile_rows_kernel has finished
    rlo = __ldcg(p.row_start + tile);
    rhi = __ldcg(p.row_start + tile + 1);
  } else if (tid < 64) {
    const int key = tid < 32 ? ts : te;
    const int r = tid < 32 ? (ts == 0 ? 0 : group_lower_bound(p.indptr, p.M, key, wl, 32, 0xffffffffu))
                           : (te >= p.nnz ? p.M : group_lower_bound(p.indptr, p.M, key, wl, 32, 0xffffffffu));
    if (wl == 0) s_rows[tid >> 5] = r;
  }
  bool slow = false;
  #pragma unroll
  for (int k = 0; k < LOADS; k++) {
    const int e = (tid + k * TW_T) * 4;
    if (e >= TILE) continue;
    #pragma unroll
    for (int i = 0; i < 4; i++)
      if ((unsigned)c[k][i] >= (unsigned)p.K) {
        c[k][i] = -1;
        v[k][i] = 0.f;  // (Inf and NaN times the zero row would not vanish)
        slow = true;
      }
    const int w = e + 4 * piece_of(e, p.inv_piece);
    *reinterpret_cast<int4 *>(s_col + w) = make_int4(c[k][0], c[k][1], c[k][2], c[k][3]);
    *reinterpret_cast<float4 *>(s_val + w) = make_float4(v[k][0], v[k][1], v[k][2], v[k][3]);
    *reinterpret_cast<int4 *>(s_info + w) = make_int4(0, 0, 0, 0);
  }
  for (int i = tid; i < (TILE + 31) / 32; i += TW_T) s_kb[i] = 0;
  if (tid < EW) s_ends[tid] = 0;
  if (!p.row_start) {
    __syncthreads();
    rlo = s_rows[0];
    rhi = s_rows[1];
  }
  rlo = min(max(rlo, 0), p.M);
  rhi = min(max(rhi, 0), p.M);
  const bool has_head = rlo > 0 && __ldg(p.indptr + rlo) > ts;
  const int rb = rlo - (has_head ? 1 : 0);
  int rs = 0, re = 0;
  if (rb + tid < rhi) {
    rs = __ldg(p.indptr + rb + tid);
    re = __ldg(p.indptr + rb + tid + 1);
  }
  __syncthreads();
  // each row that ends in the tile marks its last nonzero; rows above the
  // threshold mark all of theirs; empty rows are written here
  for (int r0 = rb; r0 < rhi; r0 += TW_T) {
    const int r = r0 + tid;
    bool empty = false;
    if (r < rhi) {
      const int s = rs, e = re;
      if (r + TW_T < rhi) {
        rs = __ldg(p.indptr + r + TW_T);
        re = __ldg(p.indptr + r + TW_T + 1);
      }
      empty = s == e;
      const unsigned pos = (unsigned)(e - 1 - ts);
      if (!empty && pos < (unsigned)n) s_info[pos + 4 * piece_of(pos, p.inv_piece)] = r + 1;
      if (e - s > a.kahan) {
        const int k0 = max(s - ts, 0), k1 = min(e - ts, n) - 1;
        for (int w = k0 >> 5; w <= k1 >> 5; w++) {
          uint32_t m = 0xffffffffu;
          if (w == (k0 >> 5)) m &= 0xffffffffu << (k0 & 31);
          if (w == (k1 >> 5)) m &= 0xffffffffu >> (31 - (k1 & 31));
          atomicOr(s_kb + w, m);
        }
      }
    }
    if (!ADDC) {
      unsigned todo = __ballot_sync(0xffffffffu, empty);
      while (todo) {
        const int src = __ffs(todo) - 1;
        todo &= todo - 1;
        if (wl < G) {
          float z[NV][V];
          clear<V, NV>(z);
          tile_store<TC, G, V, NV, false>(p, a.N, r0 + (tid & ~31) + src, z, col0, act, strm);
        }
      }
    }
  }
  slow = __syncthreads_or(slow);
  {
    const int WN = (32 / G) * S, w0 = (tid >> 5) * WN;  // the warp's nonzeros
    for (int w = w0 >> 5; w <= (w0 + WN - 1) >> 5; w++) slow |= s_kb[w] != 0;
  }
  const int gb = g * (S + 4);
  float *shead = s_head + g * COLS + lane * V, *stail = s_tail + g * COLS + lane * V;
  // accumulating into 16 bits is rare: one instantiation, the one that fits all
  constexpr bool FAST = !(ADDC && sizeof(TC) == 2);
  int hr;
  if (ADDC && !act[0])
    hr = 0;
  else if (FAST && !slow)
    hr = tile_walk<T, TC, G, V, NV, !FAST, ADDC>(p, a.N, S, s_col + gb, s_val + gb, s_info + gb, s_kb, g * S, shead,
                                           stail, lane, col0, act, keep, strm);
  else
    hr = tile_walk<T, TC, G, V, NV, true, ADDC>(p, a.N, S, s_col + gb, s_val + gb, s_info + gb, s_kb, g * S, shead,
                                          stail, lane, col0, act, keep, strm);
  if (lane == 0 && hr) atomicOr(s_ends + (g >> 5), 1u << (g & 31));
  __syncthreads();
  // the last group before x with a row end, or -1
  auto prev_end = [&](int x) {
    int w = x >> 5;
    uint32_t m = w < EW ? s_ends[w] & ((1u << (x & 31)) - 1u) : 0u;
    while (m == 0 && w > 0) m = s_ends[--w];
    return m ? w * 32 + 31 - __clz(m) : -1;
  };
  // a row's pieces in order: tails of groups [s, x), then the head of group x
  auto chain = [&](int s, int x, bool head, float (&acc)[NV][V]) {
    #pragma unroll
    for (int j = 0; j < NV; j++) {
      const int c = lane * V + j * G * V;
      sum_pieces<V>(max(s, 0), x + (head ? 1 : 0),
                    [&](int k) { return (k < x ? s_tail + k * COLS : s_head + x * COLS) + c; }, acc[j]);
    }
  };
  auto to_slot = [&](float *slots, float (&acc)[NV][V]) {
    float *d = slots + (int64_t)tile * a.N + col0;
    #pragma unroll
    for (int j = 0; j < NV; j++)
      if (act[j]) store_vec<float, V>(d + j * G * V, acc[j], strm);
  };
  float acc[NV][V];
  if (hr) {
    const int s = prev_end(g);
    chain(s, g, true, acc);
    if (s < 0 && has_head) {  // the row that entered the tile ends
      to_slot(p.heads, acc);
    } else {
      tile_store<TC, G, V, NV, ADDC>(p, a.N, hr - 1, acc, col0, act, strm);
    }
  }
  if (g == 0) {
    const int next = te < p.nnz ? __ldg(p.indptr + rhi) : te;  // where the tile's last row ends
    int2 span = make_int2(-1, 0);
    if (next > te) {  // it goes on
      const int s = prev_end(NG);
      chain(s, NG, false, acc);
      const bool whole = s < 0 && has_head;  // the tile lies inside one row
      to_slot(whole ? p.heads : p.tails, acc);
      if (!whole) span = make_int2(rhi - 1, (next - 1) / TILE);
    }
    if (lane == 0) p.span[tile] = span;  // every phase writes the same
  }
}

template <typename T, typename TC>
inline void *tile_ptr(int G, int V, int NV, bool addc) {
#define SS_TILE(g, v, nv)           \
  if (G == g && V == v && NV == nv) \
    return addc ? (void *)eb_tile_kernel<T, TC, g, v, nv, true> : (void *)eb_tile_kernel<T, TC, g, v, nv, false>;
#define SS_TILE_G(v) SS_TILE(1, v, 1) SS_TILE(2, v, 1) SS_TILE(4, v, 1) SS_TILE(8, v, 1) SS_TILE(16, v, 1)
  SS_TILE_G(1) SS_TILE(16, 1, 2) SS_TILE(16, 1, 3) SS_TILE(16, 1, 4)
  SS_TILE_G(2) SS_TILE(16, 2, 2)
  SS_TILE_G(4) SS_TILE(32, 4, 1)
  if constexpr (sizeof(T) == 2) { SS_TILE_G(8) SS_TILE(32, 8, 1) }
#undef SS_TILE_G
#undef SS_TILE
  return nullptr;
}

// Kernel tables, one translation unit per pair of types.
void *tile_kernel_f32(int G, int V, int NV, bool addc);
void *tile_kernel_f32_bf16(int G, int V, int NV, bool addc);
void *tile_kernel_f32_f16(int G, int V, int NV, bool addc);
void *tile_kernel_bf16(int G, int V, int NV, bool addc);
void *tile_kernel_bf16_f32(int G, int V, int NV, bool addc);
void *tile_kernel_f16(int G, int V, int NV, bool addc);
void *tile_kernel_f16_f32(int G, int V, int NV, bool addc);

// Geometry of the walk over one matrix at width N.
struct TileGeom {
  int G, V, NV, phases;  // lanes, elements per vector, vectors per lane, column phases
  int piece, tile;       // nonzeros of a piece and of a tile
  int tiles;
  size_t smem;
};
// vmax: elements per vector that the alignment of B and C allows; seg: the
// segment walk, whose rows stream instead of being gathered
TileGeom tile_geom(int N, int nnz, int dtype, int vmax, bool seg = false);
// What fix_kernel needs of one matrix (or segment reduction).
struct TileFix {
  const int2 *span;
  const float *heads, *tails;
  const int *hcnt, *tcnt;  // segment means
  void *C;
  int M, tiles, item_begin, tile_nz;
};
struct FixArgs {
  TileFix f;               // single launch
  const TileFix *fixes;    // batched: the matrices and the matrix of each tile
  const int32_t *item_prob;
  int items, N, accumulate, reduce;
};
// Launched right after the walk.
ss_status run_fix(int c_dtype, FixArgs &a, int vmax, cudaStream_t s);
// Launches the walk of `a` (a.items * a.phases blocks, `smem` bytes each).
// after_rows: right after tile_rows_kernel on the stream, which it overlaps.
ss_status run_tile(int val_dtype, int c_dtype, const TileGeom &g, size_t smem, TileArgs &a, bool after_rows,
                   cudaStream_t s);

}  // namespace ss
