// Batched SpMM host side: plan building and the launch (kernels in
// batched.cuh, instantiated per storage type in batched_*.cu).
#include <algorithm>
#include <cstring>
#include <vector>

#include "batched.cuh"

namespace ss {

static size_t a256(size_t x) { return (x + 255) & ~(size_t)255; }

// Fills h (everything but the offsets' final sizes) and per-matrix chunk
// sizes; returns the number of items.
// strategies: per matrix SS_EBSR (element-balanced chunks) or SS_RBSR
// (blocks of whole rows), null = all SS_EBSR.  vmax: elements per vector the
// alignment of every B and C allows (the tile walk's vector).
static ss_status batch_layout(int count, const ss_csr *mats, int N, const ss_knobs *per_mat, const int *strategies,
                              int vmax, BatchHeader &h, std::vector<BatchMat> *out, std::vector<TileProb> *tout) {
  if (count < 1 || !mats || N < 1) return fail(SS_ERR_INVALID_ARG, "batch needs count >= 1, N >= 1 and matrices");
  const int dt = mats[0].value_dtype;
  ss_knobs k0;
  if (per_mat) k0 = per_mat[0];
  else ss_default_knobs(SS_EBSR, N, &k0);
  EbGeom g;
  ss_status st = geom_sr(1, 1, N, dt, dtype_size(dt), k0, g);
  if (st) return st;
  if (g.cs.NV != 1) return fail(SS_ERR_UNSUPPORTED_KNOBS, "batched walk needs one vector per lane (coarsen <= 16 B)");
  memset(&h, 0, sizeof(h));
  h.count = count;
  h.N = N;
  h.val_dtype = dt;
  h.V = g.cs.V;
  h.NV = g.cs.NV;
  h.G = g.team_lanes;
  h.log2G = ilog2(g.team_lanes);
  h.stage = g.stage;
  h.col_tile = g.cs.col_tile;
  h.tiles = g.cs.tiles;
  h.workers_per_block = g.workers_per_block;
  h.block = g.block;
  h.smem = g.smem;
  h.kahan = k0.kahan_threshold > 0 ? k0.kahan_threshold : 1024;
  const TileGeom tg0 = tile_geom(N, 0, dt, vmax);
  h.tG = tg0.G;
  h.tV = tg0.V;
  h.tNV = tg0.NV;
  h.tphases = tg0.phases;
  // A row-balanced item is one group's serial walk: items of a whole chunk left
  // a few such matrices with one long wave (nine of 512 matrices, N = 64 BF16:
  // 555 us a step against 482), so they shrink where the row-balanced nonzeros
  // do not fill eight items a group slot.
  long long rb_nnz = 0;
  for (int m = 0; m < count; m++)
    if (strategies && strategies[m] == SS_RBSR) rb_nnz += std::max(0, mats[m].nnz);
  const long long rb_item = std::max(32LL, rb_nnz / ((long long)sm_count() * std::max(1, h.workers_per_block) * 8));
  long long items = 0, titems = 0;
  for (int m = 0; m < count; m++) {
    const ss_csr &A = mats[m];
    if (A.nrow < 0 || A.ncol < 0 || A.nnz < 0 || (A.nrow > 0 && !A.indptr) || (A.nnz > 0 && !A.indices))
      return fail(SS_ERR_INVALID_ARG, "matrix %d: bad descriptor", m);
    if (A.value_dtype != dt) return fail(SS_ERR_INVALID_ARG, "matrix %d: all matrices share one value dtype", m);
    const int tnz = per_mat ? per_mat[m].thread_nz : k0.thread_nz;
    if (tnz < 1 || tnz > 4096) return fail(SS_ERR_UNSUPPORTED_KNOBS, "matrix %d: thread_nz %d", m, tnz);
    BatchMat bm;
    memset(&bm, 0, sizeof(bm));
    bm.indptr = A.indptr;
    bm.indices = A.indices;
    bm.vals = A.values;
    bm.M = A.nrow;
    bm.K = A.ncol;
    bm.nnz = A.nnz;
    bm.chunk = tnz * h.G;
    bm.num_chunks = A.nnz > 0 ? ceil_div(A.nnz, bm.chunk) : 0;
    const int strategy = strategies ? strategies[m] : SS_EBSR;
    if (strategy != SS_EBSR && strategy != SS_RBSR)
      return fail(SS_ERR_UNSUPPORTED_KNOBS, "matrix %d: batched strategy %d is neither SS_EBSR nor SS_RBSR", m,
                  strategy);
    if (strategy == SS_RBSR && A.nnz > 0) {
      // whole rows per item, about rb_item and at most one chunk of nonzeros
      // at the mean row length
      const long long rows = (std::min((long long)bm.chunk, rb_item) * A.nrow + A.nnz - 1) / A.nnz;
      bm.rows_per_item = (int)std::min<long long>(std::max(1LL, rows), (long long)A.nrow);
      bm.num_chunks = ceil_div(A.nrow, bm.rows_per_item);
    }
    if (A.nrow > 0 && (A.nnz == 0 || (strategy == SS_EBSR && tile_tuple(h.log2G, tnz) && tile_fits(N, A.nnz, dt)))) {
      const TileGeom g = tile_geom(N, A.nnz, dt, vmax);
      TileProb p;
      memset(&p, 0, sizeof(p));
      p.indptr = A.indptr; p.cols = A.indices; p.vals = A.values;
      p.M = A.nrow; p.K = A.ncol; p.nnz = A.nnz;
      p.piece = g.piece; p.inv_piece = inverse_of(g.piece);
      p.item_begin = (int)titems;
      p.wide = (((uintptr_t)A.indices | (uintptr_t)A.values) & 15u) == 0;
      p.index = m;
      titems += g.tiles;
      h.tsmem = std::max(h.tsmem, g.smem);
      h.tile_count++;
      if (tout) tout->push_back(p);
      bm.num_chunks = 0;
    }
    bm.item_begin = (int)items;
    bm.use_tma = (((uintptr_t)A.indices & 15u) == 0) && (A.values == nullptr || ((uintptr_t)A.values & 15u) == 0) &&
                 (bm.chunk % 8) == 0;
    items += bm.num_chunks;
    if (items > 0x7fffffffLL || titems * h.tphases > 0x7fffffffLL) return fail(SS_ERR_CAPACITY, "too many work items");
    if (out) out->push_back(bm);
  }
  h.total_items = (int)items;
  h.tile_items = (int)titems;
  size_t o = 0;
  h.mats_off = o; o += a256(sizeof(BatchMat) * (size_t)count);
  h.item_mat_off = o; o += a256(4 * (size_t)items);
  h.tprobs_off = o; o += a256(sizeof(TileProb) * (size_t)h.tile_count);
  h.tfix_off = o; o += a256(sizeof(TileFix) * (size_t)h.tile_count);
  h.titem_off = o; o += a256(4 * (size_t)titems);
  h.tspan_off = o; o += a256(8 * (size_t)titems);
  // arrival counts per (item, column tile), then the work counters: one
  // memset per step clears both
  h.rows_off = o; o += 4 * (size_t)items * (size_t)(h.tiles > 0 ? h.tiles : 1);
  h.counter_off = o; o = a256(o + 4 * (size_t)(h.tiles > 0 ? h.tiles : 1));
  h.heads_off = o; o += a256(4 * (size_t)items * N);
  h.tails_off = o; o += a256(4 * (size_t)items * N);
  h.theads_off = o; o += a256(4 * (size_t)titems * N);
  h.ttails_off = o; o += a256(4 * (size_t)titems * N);
  h.dev_bytes = o;
  // the walk stores head/tail partials as vectors of up to 32 bytes
  if ((h.heads_off | h.tails_off | h.mats_off | h.item_mat_off | h.rows_off) & 255)
    return fail(SS_ERR_INVALID_ARG, "internal: misaligned batch plan layout");
  return SS_OK;
}

static size_t host_bytes_for(const BatchHeader &h) {
  return a256(sizeof(BatchHeader)) + a256(sizeof(BatchMat) * (size_t)h.count) + a256(4 * (size_t)h.total_items) +
         a256(sizeof(TileProb) * (size_t)h.tile_count) + a256(sizeof(TileFix) * (size_t)h.tile_count) +
         a256(4 * (size_t)h.tile_items);
}

// The sizes a plan may need, whatever the alignment of its operands.
static ss_status batch_most(int count, const ss_csr *mats, int N, const ss_knobs *per_mat, const int *strategies,
                            size_t *host, size_t *dev) {
  *host = *dev = 0;
  for (int v = 1; v <= 8; v <<= 1) {
    BatchHeader h;
    ss_status st = batch_layout(count, mats, N, per_mat, strategies, v, h, nullptr, nullptr);
    if (st) return st;
    *host = std::max(*host, host_bytes_for(h));
    *dev = std::max(*dev, h.dev_bytes);
  }
  return SS_OK;
}

}  // namespace ss

using namespace ss;

extern "C" {

ss_status ss_batch_plan_size_ex(int count, const ss_csr *mats, int N, const ss_knobs *per_mat,
                                const int *per_mat_strategy, size_t *host_bytes, size_t *dev_bytes) {
  if (!host_bytes || !dev_bytes) return fail(SS_ERR_INVALID_ARG, "null size pointer");
  return batch_most(count, mats, N, per_mat, per_mat_strategy, host_bytes, dev_bytes);
}

ss_status ss_batch_plan_ex(int count, const ss_csr *mats, int N, const void *const *B, void *const *C,
                           int c_dtype, const ss_knobs *per_mat, const int *per_mat_strategy, void *host_buf,
                           size_t host_bytes, void *dev_buf, size_t dev_bytes, void *stream) {
  if (!B || !C || !host_buf || !dev_buf) return fail(SS_ERR_INVALID_ARG, "null pointer");
  BatchHeader h;
  std::vector<BatchMat> bm;
  std::vector<TileProb> tp;
  if (count < 1 || !mats || N < 1) return fail(SS_ERR_INVALID_ARG, "batch needs count >= 1, N >= 1 and matrices");
  if (mats[0].value_dtype < SS_F32 || mats[0].value_dtype > SS_F16 || c_dtype < SS_F32 || c_dtype > SS_F16)
    return fail(SS_ERR_INVALID_ARG, "unknown dtype");
  int vmax = 16 / dtype_size(mats[0].value_dtype);
  for (int m = 0; m < count; m++)
    vmax = std::min(vmax, tile_vmax(B[m], dtype_size(mats[0].value_dtype), C[m], dtype_size(c_dtype)));
  ss_status st = batch_layout(count, mats, N, per_mat, per_mat_strategy, vmax, h, &bm, &tp);
  if (st) return st;
  if (c_dtype != SS_F32 && c_dtype != h.val_dtype) return fail(SS_ERR_INVALID_ARG, "c_dtype must be F32 or the value dtype");
  h.c_dtype = c_dtype;
  if (host_bytes < host_bytes_for(h) || dev_bytes < h.dev_bytes || ((uintptr_t)dev_buf % 256))
    return fail(SS_ERR_WORKSPACE, "plan needs %zu host bytes and %zu device bytes (256-byte aligned)",
                host_bytes_for(h), h.dev_bytes);
  const int es = dtype_size(h.val_dtype), cs = dtype_size(c_dtype);
  for (int m = 0; m < count; m++) {
    if ((mats[m].nnz > 0 && !B[m]) || (mats[m].nrow > 0 && !C[m]))
      return fail(SS_ERR_INVALID_ARG, "matrix %d: null B or C", m);
    if (((uintptr_t)B[m] % (size_t)(es * h.V)) || ((uintptr_t)C[m] % (size_t)(cs * h.V)))
      return fail(SS_ERR_ALIGNMENT, "matrix %d: B/C not aligned to the %d-element vector", m, h.V);
    bm[m].B = B[m];
    bm[m].C = C[m];
  }
  char *hb = (char *)host_buf;
  memcpy(hb, &h, sizeof(h));
  BatchMat *hm = (BatchMat *)(hb + a256(sizeof(BatchHeader)));
  memcpy(hm, bm.data(), sizeof(BatchMat) * (size_t)count);
  int32_t *him = (int32_t *)((char *)hm + a256(sizeof(BatchMat) * (size_t)count));
  for (int m = 0; m < count; m++)
    for (int c = 0; c < bm[m].num_chunks; c++) him[bm[m].item_begin + c] = m;
  TileProb *ht = (TileProb *)((char *)him + a256(4 * (size_t)h.total_items));
  TileFix *hf = (TileFix *)((char *)ht + a256(sizeof(TileProb) * (size_t)h.tile_count));
  int32_t *hti = (int32_t *)((char *)hf + a256(sizeof(TileFix) * (size_t)h.tile_count));
  std::vector<TileFix> tf((size_t)h.tile_count);
  char *db = (char *)dev_buf;
  for (int i = 0; i < h.tile_count; i++) {
    TileProb &p = tp[i];
    const int m = p.index;
    p.B = B[m];
    p.C = C[m];
    p.span = (int2 *)(db + h.tspan_off) + p.item_begin;
    p.heads = (float *)(db + h.theads_off) + (size_t)p.item_begin * N;
    p.tails = (float *)(db + h.ttails_off) + (size_t)p.item_begin * N;
    const int end = i + 1 < h.tile_count ? tp[i + 1].item_begin : h.tile_items;
    for (int c = p.item_begin; c < end; c++) hti[c] = i;
    TileFix &f = tf[(size_t)i];
    memset(&f, 0, sizeof(f));
    f.span = p.span; f.heads = p.heads; f.tails = p.tails; f.C = p.C;
    f.M = p.M; f.tiles = end - p.item_begin; f.item_begin = p.item_begin;
  }
  if (h.tile_count > 0) memcpy(hf, tf.data(), sizeof(TileFix) * (size_t)h.tile_count);
  if (h.tile_count > 0) memcpy(ht, tp.data(), sizeof(TileProb) * (size_t)h.tile_count);
  cudaStream_t s = (cudaStream_t)stream;
  cudaError_t e = cudaMemcpyAsync((char *)dev_buf + h.mats_off, hm, sizeof(BatchMat) * (size_t)count,
                                  cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess && h.total_items > 0)
    e = cudaMemcpyAsync((char *)dev_buf + h.item_mat_off, him, 4 * (size_t)h.total_items, cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess && h.tile_count > 0)
    e = cudaMemcpyAsync(db + h.tprobs_off, ht, sizeof(TileProb) * (size_t)h.tile_count, cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess && h.tile_count > 0)
    e = cudaMemcpyAsync(db + h.tfix_off, hf, sizeof(TileFix) * (size_t)h.tile_count, cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess && h.tile_items > 0)
    e = cudaMemcpyAsync(db + h.titem_off, hti, 4 * (size_t)h.tile_items, cudaMemcpyHostToDevice, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);  // the host buffer may be reused after return
  return e == cudaSuccess ? SS_OK : cuda_fail(e, "batch plan upload");
}

ss_status ss_batch_plan_size(int count, const ss_csr *mats, int N, const ss_knobs *per_mat, size_t *host_bytes,
                             size_t *dev_bytes) {
  return ss_batch_plan_size_ex(count, mats, N, per_mat, nullptr, host_bytes, dev_bytes);
}

ss_status ss_batch_plan(int count, const ss_csr *mats, int N, const void *const *B, void *const *C, int c_dtype,
                        const ss_knobs *per_mat, void *host_buf, size_t host_bytes, void *dev_buf, size_t dev_bytes,
                        void *stream) {
  return ss_batch_plan_ex(count, mats, N, B, C, c_dtype, per_mat, nullptr, host_buf, host_bytes, dev_buf, dev_bytes,
                          stream);
}

ss_status ss_spmm_batched(const void *host_plan, void *dev_plan, void *stream) {
  ss::NvtxRange nvtx_range("ss_spmm_batched");
  if (!host_plan || !dev_plan) return fail(SS_ERR_INVALID_ARG, "null plan");
  BatchHeader h;
  memcpy(&h, host_plan, sizeof(h));
  if (h.total_items == 0 && h.tile_items == 0) return SS_OK;
  cudaStream_t s = (cudaStream_t)stream;
  char *plan = (char *)dev_plan;
  cudaError_t e;
  if (h.tile_items > 0) {
    TileArgs a;
    memset(&a, 0, sizeof(a));
    a.probs = (const TileProb *)(plan + h.tprobs_off);
    a.item_prob = (const int32_t *)(plan + h.titem_off);
    a.items = h.tile_items;
    a.phases = h.tphases;
    a.N = h.N;
    a.kahan = h.kahan;
    a.keep_frac = 1.0f;
    TileGeom g;
    memset(&g, 0, sizeof(g));
    g.G = h.tG;
    g.V = h.tV;
    g.NV = h.tNV;
    ss_status st = run_tile(h.val_dtype, h.c_dtype, g, h.tsmem, a, false, s);
    if (st == SS_OK && h.tile_items > h.tile_count) {  // some matrix has two tiles
      FixArgs f;
      memset(&f, 0, sizeof(f));
      f.fixes = (const TileFix *)(plan + h.tfix_off);
      f.item_prob = a.item_prob;
      f.items = h.tile_items;
      f.N = h.N;
      f.reduce = SS_SUM;
      st = run_fix(h.c_dtype, f, h.tV, s);
    }
    if (st || h.total_items == 0) return st;
  }
  // arrival counts and work counters (adjacent in the plan)
  e = cudaMemsetAsync(plan + h.rows_off, 0, h.heads_off - h.rows_off, s);
  if (e != cudaSuccess) return cuda_fail(e, "batched counter reset");
  void *fn;
  if (h.val_dtype == SS_F32) fn = batched_kernel_f32(h.V, h.NV);
  else if (h.val_dtype == SS_BF16) fn = batched_kernel_bf16(h.V, h.NV, h.c_dtype == SS_F32);
  else fn = batched_kernel_f16(h.V, h.NV, h.c_dtype == SS_F32);
  if (!fn) return fail(SS_ERR_UNSUPPORTED_KNOBS, "no batched kernel for V=%d NV=%d", h.V, h.NV);
  if (h.smem > 48 * 1024) {
    const ss_status st = allow_smem(fn, SR_SMEM_MAX, "batched smem attribute");
    if (st) return st;
  }
  int per_sm = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, h.block, h.smem);
  if (e != cudaSuccess || per_sm < 1) return fail(SS_ERR_UNSUPPORTED_KNOBS, "batched block does not fit an SM");
  long long grid = (long long)per_sm * sm_count();
  const long long need = ((long long)h.total_items + h.workers_per_block - 1) / h.workers_per_block;
  if (grid > need) grid = need;
  int *err_ptr = walk_error_ptr();
  void *args[] = {&plan, &h, &err_ptr};
  e = cudaLaunchKernel(fn, dim3((unsigned)grid, (unsigned)h.tiles, 1), dim3(h.block, 1, 1), args, h.smem, s);
  return e == cudaSuccess ? SS_OK : cuda_fail(e, "batched launch");
}

}  // extern "C"
