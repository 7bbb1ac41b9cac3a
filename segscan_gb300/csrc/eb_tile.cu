// Geometry and launch of the tile walk (kernel in eb_tile.cuh).
#include <algorithm>
#include <cstring>

#include "seg_tile.cuh"

namespace ss {

// row_start[t] = first row that starts at or after nonzero t * tile_nz
// (row_start[tiles] = M; also M where indptr[M] ends before the tile does, as
// in matrices whose dropped entries follow the last row), four rows a thread.  2 us on a million rows, against
// 2.5 us of search latency in every wave of the walk (N = 64: 207 -> 203 us).
__global__ void __launch_bounds__(256) tile_rows_kernel(const int32_t *__restrict__ indptr, int M, int tile,
                                                        uint32_t inv_tile, int tiles, int32_t *__restrict__ row_start) {
  grid_dependents_launch();  // the walk may load its tiles; it waits for the rows
  const long long stride = (long long)gridDim.x * 256, i0 = blockIdx.x * 256ll + threadIdx.x;
  // p / tile: the product with floor(2^32 / tile) is at most one short
  auto tile_of = [&](int p) {
    const int q = (int)__umulhi((uint32_t)p, inv_tile);
    return p < 0 ? -1 : p - q * tile >= tile ? q + 1 : q;
  };
  for (long long r0 = i0 * 4; r0 <= M; r0 += stride * 4) {
    int x[5];
    x[0] = r0 > 0 ? tile_of(__ldg(indptr + r0 - 1)) : -1;
    #pragma unroll
    for (int i = 0; i < 4; i++)
      x[i + 1] = r0 + i < M ? tile_of(__ldg(indptr + r0 + i)) : r0 + i == M ? tiles : INT_MIN;
    #pragma unroll
    for (int i = 0; i < 4; i++)
      for (int t = max(x[i] + 1, 0); t <= min(x[i + 1], tiles - 1); t++) row_start[t] = (int)r0 + i;
  }
  if (i0 == 0) row_start[tiles] = M;
}

TileGeom tile_geom(int N, int nnz, int dtype, int vmax, bool seg) {
  TileGeom g;
  int V = std::min(16 / dtype_size(dtype), std::max(1, vmax));
  while (N % V) V >>= 1;
  const int nv = ceil_div(N, V);
  g.V = V;
  g.NV = 1;
  g.G = std::min(16, ceil_pow2(nv));
  // 17 to 32 wide vectors: one phase of 32 lanes instead of two of 16, unless
  // two full phases gather a matrix's rows as fast (N = 128: 420 against 428
  // us).  A part empty second phase costs more (N = 100 FP32 is 25 vectors),
  // and streamed rows are better read in one piece.
  if (V >= 4 && nv > 16 && nv <= 32 && (seg || nv < 32)) g.G = 32;
  // widths that no wide vector divides: several vectors per lane, as many as
  // leave the fewest idle columns (N = 47: 16 lanes of three, 108 us, against
  // three phases of one, 252 us)
  const int most = V == 1 ? 4 : V == 2 ? 2 : 1;
  if (nv > 16)
    for (int m = 2; m <= most; m++)
      if (ceil_div(nv, 16 * m) * m <= ceil_div(nv, 16 * g.NV) * g.NV) g.NV = m;
  g.phases = ceil_div(N, g.G * V * g.NV);
  // Pieces as long as shared memory allows without costing resident blocks
  // (2048 nonzeros a tile, 1024 with 16 or 32 lanes): a block's set-up is
  // about a quarter of its time there.  Shorter where two blocks per SM would
  // not be filled (more, shorter blocks than that are slower: 320 K nonzeros
  // BF16 N = 64 18 us at 313 blocks, 20 at 625, 25 at 1250), and cut so that
  // a few waves of blocks are whole ones.
  const int NG = TW_T / g.G;
  const int most_piece = g.G >= 32 ? 128 : g.G >= 16 ? 64 : 8 * g.G;
  const long long work = (long long)nnz * g.phases;             // nonzeros over the column phases
  const long long wave = 4LL * sm_count() * NG, half = wave / 2;  // groups of a resident wave
  long long piece = most_piece;
  if (work <= half * most_piece) piece = ceil_div(work, half);
  else if (work > wave * most_piece && work <= 6 * wave * most_piece)
    piece = ceil_div(work, wave * ceil_div(work, wave * most_piece));
  g.piece = (int)std::max(8LL, (piece + 7) / 8 * 8);  // odd strides of four words: no bank conflicts
  g.tile = NG * g.piece;
  g.tiles = std::max(1, ceil_div(nnz, g.tile));
  g.smem = (size_t)tile_smem(g.G, V * g.NV, g.piece).total * 4;
  return g;
}

// The tile walk's scratch grows with the matrix (two partial rows a tile), the
// group walk's does not: past 2^18 tiles (256 M nonzeros at 16 lanes, 128 MB
// at N = 64) the group walk keeps it.  It also takes what a block index or a
// 32-bit row stride cannot hold.
bool tile_fits(int N, int nnz, int dtype) {
  if (N >= (1 << 29)) return false;
  for (int v = 1; v <= 16 / dtype_size(dtype); v <<= 1) {
    const TileGeom g = tile_geom(N, nnz, dtype, v);
    if (g.tiles > 1 << 18 || (long long)g.tiles * g.phases >= (1LL << 31)) return false;
  }
  return true;
}

static size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

static size_t tile_ws(const TileGeom &g, int N) {
  return align256((size_t)g.tiles * 8) + align256((size_t)(g.tiles + 1) * 4) +
         2 * (size_t)g.tiles * (size_t)N * sizeof(float);
}

size_t tile_workspace_bytes(int N, int nnz, int dtype) {
  // the alignment of B and C, and so the vector, is not known to the query
  size_t most = 0;
  for (int v = 1; v <= 16 / dtype_size(dtype); v <<= 1) most = std::max(most, tile_ws(tile_geom(N, nnz, dtype, v), N));
  return most;
}

int tile_vmax(const void *B, int b_bytes, const void *C, int c_bytes) {
  int v = 16 / b_bytes;
  while (v > 1 && (((uintptr_t)B % (size_t)(b_bytes * v)) || ((uintptr_t)C % (size_t)std::min(16, c_bytes * v)))) v >>= 1;
  return v;
}

static void *tile_kernel(int val_dtype, int c_dtype, int G, int V, int NV, bool addc) {
  if (val_dtype == SS_F32)
    return c_dtype == SS_F32    ? tile_kernel_f32(G, V, NV, addc)
           : c_dtype == SS_BF16 ? tile_kernel_f32_bf16(G, V, NV, addc)
                                : tile_kernel_f32_f16(G, V, NV, addc);
  if (val_dtype == SS_BF16) return c_dtype == SS_F32 ? tile_kernel_bf16_f32(G, V, NV, addc) : tile_kernel_bf16(G, V, NV, addc);
  return c_dtype == SS_F32 ? tile_kernel_f16_f32(G, V, NV, addc) : tile_kernel_f16(G, V, NV, addc);
}

// A launch whose blocks may start before the stream's last kernel has ended
// (overlap): they wait for it where they need its results.
static ss_status launch_overlapping(void *fn, void *arg, int blocks, size_t smem, bool overlap, cudaStream_t s,
                                    const char *what) {
  void *args[] = {arg};
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)blocks, 1, 1);
  cfg.blockDim = dim3(TW_T, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = &attr;
  cfg.numAttrs = overlap ? 1 : 0;
  cudaError_t e = cudaLaunchKernelExC(&cfg, fn, args);
  return e == cudaSuccess ? SS_OK : cuda_fail(e, what);
}

// Rows that straddle tiles, a warp per tile: the row that starts in tile o
// and goes on (span) is tail(o) + heads(o+1..last) in tile order with
// compensation (or the maximum), plus the old row in accumulate mode, divided
// by the segment's length for a mean; stored once.
template <typename TC, int V>
__global__ void __launch_bounds__(TW_T) fix_kernel(FixArgs a) {
  grid_dependency_wait();  // the walk has finished
  const int item = blockIdx.x * (TW_T / 32) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (item >= a.items) return;
  const TileFix f = a.item_prob ? a.fixes[__ldg(a.item_prob + item)] : a.f;
  const int o = item - f.item_begin;
  const int2 span = __ldcg(f.span + o);
  const int r = span.x, l = span.y;
  if ((unsigned)r >= (unsigned)f.M || l <= o || l >= f.tiles) return;
  const bool is_max = a.reduce == SS_MAX, mean = a.reduce == SS_MEAN;
  float len = 1.f;
  if (mean) len = (float)(__ldcg(f.tcnt + o) + (l - o - 1) * f.tile_nz + __ldcg(f.hcnt + l));
  const uint64_t strm = policy_stream();
  for (int col = lane * V; col < a.N; col += 32 * V) {
    float acc[V], comp[V];
    load_slot<V>(f.tails + (int64_t)o * a.N + col, acc);
    #pragma unroll
    for (int i = 0; i < V; i++) comp[i] = 0.f;
    auto add = [&](const float (&x)[V]) {
      #pragma unroll
      for (int i = 0; i < V; i++) {
        if (is_max) acc[i] = fmaxf(acc[i], x[i]);
        else kahan_add(acc[i], comp[i], x[i]);
      }
    };
    auto head = [&](int k, float (&x)[V]) { load_slot<V>(f.heads + (int64_t)k * a.N + col, x); };
    int k = o + 1;
    // A row over many tiles is one chain of loads: eight heads in flight (one
    // row of 4.6 M nonzeros, N = 64: 767 us with four, 510 with eight; sixteen
    // take 92 registers, and the batch of 64 matrices 86 -> 89 us).
    #pragma unroll 1
    for (; k + 8 <= l + 1; k += 8) {
      float x[8][V];
      #pragma unroll
      for (int u = 0; u < 8; u++) head(k + u, x[u]);
      #pragma unroll
      for (int u = 0; u < 8; u++) add(x[u]);
    }
    #pragma unroll 1
    for (; k <= l; k += 4) {
      float x[4][V];
      #pragma unroll
      for (int u = 0; u < 4; u++) head(min(k + u, l), x[u]);
      #pragma unroll
      for (int u = 0; u < 4; u++) {
        if (k + u > l) break;
        add(x[u]);
      }
    }
    TC *d = (TC *)f.C + (int64_t)r * a.N + col;
    if (a.accumulate) {
      float old[V];
      load_old<TC, V>(d, old);
      #pragma unroll
      for (int i = 0; i < V; i++) acc[i] += old[i];
    }
    if (mean) {
      #pragma unroll
      for (int i = 0; i < V; i++) acc[i] = acc[i] / len;
    }
    store_vec<TC, V>(d, acc, strm);
  }
}

template <typename TC>
static void *fix_ptr(int V) {
  return V >= 4 ? (void *)fix_kernel<TC, 4> : V == 2 ? (void *)fix_kernel<TC, 2> : (void *)fix_kernel<TC, 1>;
}

ss_status run_fix(int c_dtype, FixArgs &a, int V, cudaStream_t s) {
  void *fn = c_dtype == SS_F32 ? fix_ptr<float>(V) : c_dtype == SS_BF16 ? fix_ptr<__nv_bfloat16>(V) : fix_ptr<__half>(V);
  return launch_overlapping(fn, &a, ceil_div(a.items, TW_T / 32), 0, true, s, "straddling rows launch");
}

ss_status run_tile(int val_dtype, int c_dtype, const TileGeom &g, size_t smem, TileArgs &a, bool after_rows,
                   cudaStream_t s) {
  void *fn = tile_kernel(val_dtype, c_dtype, g.G, g.V, g.NV, a.accumulate != 0);
  if (!fn) return fail(SS_ERR_UNSUPPORTED_KNOBS, "no tile walk for G=%d V=%d NV=%d", g.G, g.V, g.NV);
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return cuda_fail(e, "tile walk shared memory");
  }
  return launch_overlapping(fn, &a, a.items * a.phases, smem, after_rows, s, "tile walk launch");
}

ss_status launch_ebsr_tile(const SpmmCall &c, void *ws, cudaStream_t s) {
  const TileGeom g = tile_geom(c.N, c.nnz, c.val_dtype,
                               tile_vmax(c.B, dtype_size(c.val_dtype), c.C, dtype_size(c.c_dtype)));
  TileArgs a;
  memset(&a, 0, sizeof(a));
  TileProb &p = a.p;
  p.indptr = c.indptr; p.cols = c.indices; p.vals = c.vals; p.B = c.B; p.C = c.C;
  p.M = c.M; p.K = c.K; p.nnz = c.nnz;
  p.perm = c.perm; p.perm_dtype = c.perm_dtype;
  p.piece = g.piece; p.inv_piece = inverse_of(g.piece);
  p.wide = (((uintptr_t)c.indices | (uintptr_t)c.vals) & 15u) == 0;
  char *w = (char *)ws;
  p.span = (int2 *)w; w += align256((size_t)g.tiles * 8);
  int32_t *row_start = (int32_t *)w; w += align256((size_t)(g.tiles + 1) * 4);
  // No more blocks than are resident at once: each searches its own rows and
  // the launch is saved (Poisson 12 a row, N = 64: 1 K rows at N = 16 6.97 ->
  // 6.06 us, 40 K rows 23.5 -> 20.4 us).  With more waves every one pays for
  // the search (80 K rows 29.1 -> 30.0 us, 1 M rows at N = 16 110 -> 116 us).
  const bool searched = (long long)g.tiles * g.phases <= 4LL * sm_count();
  p.row_start = searched ? nullptr : row_start;
  p.heads = (float *)w;
  p.tails = p.heads + (size_t)g.tiles * c.N;
  a.items = g.tiles; a.phases = g.phases;
  a.N = c.N; a.accumulate = c.accumulate; a.kahan = c.kahan_threshold;
  a.keep_frac = l2_keep_fraction((size_t)c.K * c.N * dtype_size(c.val_dtype));
  if (!searched) {
    const long long want = ((long long)c.M + 1024) / 1024;
    tile_rows_kernel<<<(unsigned)std::min(want, (long long)sm_count() * 16), 256, 0, s>>>(
        c.indptr, c.M, g.tile, (uint32_t)((1ull << 32) / g.tile), g.tiles, row_start);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_fail(e, "tile rows launch");
  }
  ss_status st = run_tile(c.val_dtype, c.c_dtype, g, g.smem, a, !searched, s);
  if (st || g.tiles == 1) return st;  // one tile: no row straddles
  FixArgs f;
  memset(&f, 0, sizeof(f));
  f.f.span = p.span; f.f.heads = p.heads; f.f.tails = p.tails; f.f.C = c.C;
  f.f.M = c.M; f.f.tiles = g.tiles; f.f.tile_nz = g.tile;
  f.items = g.tiles; f.N = c.N; f.accumulate = c.accumulate; f.reduce = SS_SUM;
  return run_fix(c.c_dtype, f, g.V, s);
}

// ---------------------------------------------------------------------
// segment_coo
// ---------------------------------------------------------------------
static size_t seg_tile_ws(const TileGeom &g, int N) {
  return align256((size_t)g.tiles * 8) + align256((size_t)2 * g.tiles * 4) +
         2 * (size_t)g.tiles * (size_t)N * sizeof(float);
}

bool seg_tile_fits(int N, int nnz) {
  if (N >= (1 << 29)) return false;
  for (int dt : {SS_F32, SS_BF16})
    for (int v = 1; v <= 16 / dtype_size(dt); v <<= 1) {
      const TileGeom g = tile_geom(N, nnz, dt, v, true);
      if (g.tiles > 1 << 18 || (long long)g.tiles * g.phases >= (1LL << 31)) return false;
    }
  return true;
}

size_t seg_tile_workspace_bytes(int N, int nnz) {
  size_t most = 0;  // over the source types and the alignments of src and dst
  for (int dt : {SS_F32, SS_BF16})
    for (int v = 1; v <= 16 / dtype_size(dt); v <<= 1)
      most = std::max(most, seg_tile_ws(tile_geom(N, nnz, dt, v, true), N));
  return most;
}

ss_status launch_seg_tile(const SegCall &c, bool kahan, void *ws, cudaStream_t s) {
  const TileGeom g = tile_geom(c.N, c.nnz, c.src_dtype, tile_vmax(c.src, dtype_size(c.src_dtype), c.dst, 4), true);
  SegTileArgs a;
  memset(&a, 0, sizeof(a));
  a.src = c.src; a.index = c.index; a.dst = c.dst;
  a.M = c.dst_len; a.nnz = c.nnz; a.N = c.N; a.piece = g.piece; a.inv_piece = inverse_of(g.piece); a.tiles = g.tiles; a.phases = g.phases;
  a.reduce = c.reduce; a.kahan = kahan;
  char *w = (char *)ws;
  a.span = (int2 *)w; w += align256((size_t)g.tiles * 8);
  a.hcnt = (int *)w;
  a.tcnt = a.hcnt + g.tiles; w += align256((size_t)2 * g.tiles * 4);
  a.heads = (float *)w;
  a.tails = a.heads + (size_t)g.tiles * c.N;
  void *fn = c.src_dtype == SS_F32    ? seg_tile_kernel_f32(g.G, g.V, g.NV, c.accumulate != 0)
             : c.src_dtype == SS_BF16 ? seg_tile_kernel_bf16(g.G, g.V, g.NV, c.accumulate != 0)
                                      : seg_tile_kernel_f16(g.G, g.V, g.NV, c.accumulate != 0);
  if (!fn) return fail(SS_ERR_UNSUPPORTED_KNOBS, "no segment tile walk for G=%d V=%d NV=%d", g.G, g.V, g.NV);
  const int NG = TW_T / g.G;
  const size_t smem = ((size_t)NG * (g.piece + 4) + 2 * (size_t)TW_T * g.V * g.NV + ceil_div(g.tile, 32)) * 4;
  void *args[] = {&a};
  cudaError_t e = cudaLaunchKernel(fn, dim3((unsigned)(g.tiles * g.phases), 1, 1), dim3(TW_T, 1, 1), args, smem, s);
  if (e != cudaSuccess) return cuda_fail(e, "segment tile walk launch");
  if (g.tiles == 1) return SS_OK;
  FixArgs f;
  memset(&f, 0, sizeof(f));
  f.f.span = a.span; f.f.heads = a.heads; f.f.tails = a.tails; f.f.hcnt = a.hcnt; f.f.tcnt = a.tcnt;
  f.f.C = c.dst; f.f.M = c.dst_len; f.f.tiles = g.tiles; f.f.tile_nz = g.tile;
  f.items = g.tiles; f.N = c.N; f.accumulate = c.accumulate; f.reduce = c.reduce;
  return run_fix(SS_F32, f, g.V, s);
}

}  // namespace ss
