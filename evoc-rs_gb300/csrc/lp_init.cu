// lp_init.cu — label_propagation_init (src/graph/label_prop.rs:403-564,
// evoc-rs 0.2.7) on the GPU: the recursive coarsening initialisation that
// evoc() runs before the embedding.
//
// One level (label_prop_init_inner, label_prop.rs:403-535) of an n-node graph:
//   1. partition by label propagation (label_prop.cu);
//   2. per part P: node count c_P, inv_P = 1 / sqrt(c_P) (the L2 column
//      norm of the partition matrix, sparse.rs:427-458), the L1 row scale of
//      its transpose (serial sum of c_P copies of inv_P, sparse.rs:468-492);
//   3. coarse graph clip(N^T G B) (sparse.rs:307-365): the products
//      inv_P * w_ij of every entry are ordered (P, j, i) by two stable radix
//      sorts and summed serially per (P, j) (the sparse accumulator's order:
//      rows of P ascending), then re-ordered (P, Q = part(j), j) and summed
//      serially per (P, Q); clipped to [0, 1] (sparse.rs:501-510);
//   4. coarse data (sparse.rs:545-568): per part, its nodes in order,
//      acc += scale * x;
//   5. recursion on the coarse graph and data (base case: PCA of the data,
//      or a random unit-row init, below 64 nodes);
//   6. a short embedding of the coarse graph (the library's own plan path);
//   7. expansion: the graph's symmetric part G o G^T times N, L1 row
//      normalised, times the coarse layout (per (i, Q) serial sums after the
//      same sort), averaged with the direct term N_l1 x layout, centred by
//      serial column sums, scaled.
// Summation orders are the reference's (restated in the oracle), so the
// initial embedding equals the oracle's bit for bit. Random draws are Philox
// (the documented deviation); the PCA base case is a Jacobi eigen-solve of
// the small Gram matrix in double on the host, with a fixed sign convention.
#include "evoc_device.cuh"
#include "evoc_internal.h"
#include "row_groups.cuh"


#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

namespace evoc {
namespace {

inline unsigned grid_of(int64_t n, int t = 256) { return (unsigned)((n + t - 1) / t); }

// ---------------------------------------------------------------------------
// Per-part constants.
// ---------------------------------------------------------------------------
__global__ void k_part_count(const uint32_t* __restrict__ part, int64_t n,
                             int32_t* __restrict__ cnt) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) atomicAdd(&cnt[part[i]], 1);
}

// inv = 1 / sqrt(c) (c is exact: c products 1 * 1 summed); rv = inv * (1 / s)
// with s the serial sum of c copies of inv; u = inv * (1 / inv).
__global__ void k_part_consts(const int32_t* __restrict__ cnt, int64_t np,
                              float* __restrict__ inv, float* __restrict__ rv,
                              float* __restrict__ u) {
  const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= np) return;
  const int32_t c = cnt[p];
  const float nrm = fsqrt((float)c);
  const float iv = nrm > 0.0f ? fdiv(1.0f, nrm) : 1.0f;
  float s = 0.0f;
  for (int32_t k = 0; k < c; ++k) s = fadd(s, fabsf(iv));
  rv[p] = s > 0.0f ? fmul(iv, fdiv(1.0f, s)) : iv;
  const float a = fabsf(iv);
  u[p] = a > 0.0f ? fmul(iv, fdiv(1.0f, a)) : iv;
  inv[p] = iv;
}

// ---------------------------------------------------------------------------
// Sort-and-sum machinery. An entry list in a given order is sorted stably by
// (major, minor) with two radix passes (minor first), then equal (major,
// minor) runs are summed serially in list order (first value, then +).
// Keys are u32; values are uint2 (other key, float bits).
// ---------------------------------------------------------------------------
// Coarse-graph products in row-major order: key j, value (P, inv_P * w_ij).
__global__ void k_gen_products(const int64_t* __restrict__ indptr,
                               const uint32_t* __restrict__ indices,
                               const float* __restrict__ w, int64_t n,
                               const uint32_t* __restrict__ part,
                               const float* __restrict__ inv, uint32_t* __restrict__ keys,
                               uint2* __restrict__ vals) {
  const int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (i >= n) return;
  const uint32_t P = part[i];
  const float iv = inv[P];
  for (int64_t e = indptr[i] + lane; e < indptr[i + 1]; e += 32) {
    keys[e] = indices[e];
    vals[e] = make_uint2(P, __float_as_uint(fmul(iv, w[e])));
  }
}

// vals[i] = (i, 0)
__global__ void k_iota_pairs(uint2* __restrict__ vals, int64_t n) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) vals[i] = make_uint2((uint32_t)i, 0u);
}

// Entries of G in row-major order as (key column j, value (row i, w bits)):
// the input of the stable transpose (sparse.rs:256-296).
__global__ void k_transpose_gen(const int64_t* __restrict__ indptr,
                                const uint32_t* __restrict__ indices,
                                const float* __restrict__ w, int64_t n,
                                uint32_t* __restrict__ keys, uint2* __restrict__ vals) {
  const int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (i >= n) return;
  for (int64_t e = indptr[i] + lane; e < indptr[i + 1]; e += 32) {
    keys[e] = indices[e];
    vals[e] = make_uint2((uint32_t)i, __float_as_uint(w[e]));
  }
}

__global__ void k_unpack_pairs(const uint2* __restrict__ vals, int64_t m,
                               uint32_t* __restrict__ idx, float* __restrict__ w) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= m) return;
  idx[e] = vals[e].x;
  w[e] = __uint_as_float(vals[e].y);
}

// keys <- vals.x, vals <- (old key, vals.y)
__global__ void k_swap_keys(uint32_t* __restrict__ keys, uint2* __restrict__ vals, int64_t m) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= m) return;
  const uint32_t k = keys[e];
  const uint2 v = vals[e];
  keys[e] = v.x;
  vals[e] = make_uint2(k, v.y);
}

// keys <- map[vals.x], vals unchanged
__global__ void k_map_keys(uint32_t* __restrict__ keys, const uint2* __restrict__ vals,
                           int64_t m, const uint32_t* __restrict__ map) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e < m) keys[e] = map[vals[e].x];
}

// head[e] = 1 where (keys, vals.x) starts a new run
__global__ void k_run_heads(const uint32_t* __restrict__ keys, const uint2* __restrict__ vals,
                            int64_t m, int32_t* __restrict__ head) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= m) return;
  head[e] = (e == 0 || keys[e] != keys[e - 1] || vals[e].x != vals[e - 1].x) ? 1 : 0;
}

// First entry of each run: start[rid[e]] = e for heads; start[runs] = m.
__global__ void k_run_starts(const int32_t* __restrict__ head, const int64_t* __restrict__ rid,
                             int64_t m, int64_t* __restrict__ start) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= m) return;
  if (head[e]) start[rid[e]] = e;
  if (e == m - 1) start[rid[m]] = m;
}

// Serial sum of each run: (key, (vals.x, sum bits)). A thread per run, the next
// eight values loaded before the eight in hand are added: runs are a few entries
// or, for a part's own weight in the coarse graph, thousands, and one dependent
// load per addition made those the kernel's length.
__global__ void k_run_sums(const uint32_t* __restrict__ keys, const uint2* __restrict__ vals,
                           const int64_t* __restrict__ start, int64_t runs,
                           uint32_t* __restrict__ okeys, uint2* __restrict__ ovals) {
  constexpr int U = 8;
  const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= runs) return;
  const int64_t a = start[r], b = start[r + 1];
  const uint2 v0 = vals[a];
  float s = __uint_as_float(v0.y);
  int64_t f = a + 1;
  if (f + U <= b) {
    float t[U];
#pragma unroll
    for (int u = 0; u < U; ++u) t[u] = __uint_as_float(vals[f + u].y);
    for (f += U; f + U <= b; f += U) {
      float x[U];
#pragma unroll
      for (int u = 0; u < U; ++u) x[u] = __uint_as_float(vals[f + u].y);
#pragma unroll
      for (int u = 0; u < U; ++u) s = fadd(s, t[u]);
#pragma unroll
      for (int u = 0; u < U; ++u) t[u] = x[u];
    }
#pragma unroll
    for (int u = 0; u < U; ++u) s = fadd(s, t[u]);
  }
  for (; f < b; ++f) s = fadd(s, __uint_as_float(vals[f].y));
  okeys[r] = keys[a];
  ovals[r] = make_uint2(v0.x, __float_as_uint(s));
}

// Sums the equal-(keys, vals.x) runs of a sorted list serially into (ok, ov);
// returns their count.
int64_t sum_runs(evoc_ctx* ctx, const uint32_t* keys, const uint2* vals, int64_t m,
                 DevBuf<uint32_t>& ok, DevBuf<uint2>& ov) {
  cudaStream_t s = ctx->stream;
  DevBuf<int32_t> head(m, s);
  DevBuf<int64_t> rid(m + 1, s);
  k_run_heads<<<grid_of(m), 256, 0, s>>>(keys, vals, m, head.get());
  EVOC_CHECK_LAUNCH();
  exclusive_scan_i32_to_i64(ctx, head.get(), rid.get(), m);
  int64_t runs = 0;
  EVOC_CUDA(cudaMemcpyAsync(&runs, rid.get() + m, sizeof(int64_t), cudaMemcpyDeviceToHost, s));
  EVOC_CUDA(cudaStreamSynchronize(s));
  DevBuf<int64_t> start(runs + 1, s);
  k_run_starts<<<grid_of(m), 256, 0, s>>>(head.get(), rid.get(), m, start.get());
  EVOC_CHECK_LAUNCH();
  ok.alloc(runs, s);
  ov.alloc(runs, s);
  k_run_sums<<<grid_of(runs, 128), 128, 0, s>>>(keys, vals, start.get(), runs, ok.get(),
                                                ov.get());
  EVOC_CHECK_LAUNCH();
  return runs;
}

// Sorts (keys, vals) by (keys major, vals.x minor), stably, then sums the
// equal-(key, minor) runs serially. Returns the run count; the runs replace
// the list.
int64_t sort_and_sum(evoc_ctx* ctx, DevBuf<uint32_t>& keys, DevBuf<uint2>& vals, int64_t m,
                     int major_bits, int minor_bits) {
  cudaStream_t s = ctx->stream;
  if (m == 0) return 0;
  // minor first (keys <- vals.x), then major
  k_swap_keys<<<grid_of(m), 256, 0, s>>>(keys.get(), vals.get(), m);
  EVOC_CHECK_LAUNCH();
  radix_sort_pairs(ctx, keys, vals, m, minor_bits);
  k_swap_keys<<<grid_of(m), 256, 0, s>>>(keys.get(), vals.get(), m);
  EVOC_CHECK_LAUNCH();
  radix_sort_pairs(ctx, keys, vals, m, major_bits);
  DevBuf<uint32_t> ok;
  DevBuf<uint2> ov;
  const int64_t runs = sum_runs(ctx, keys.get(), vals.get(), m, ok, ov);
  keys = std::move(ok);
  vals = std::move(ov);
  return runs;
}

// Row counts of a (row, (col, value)) run list sorted by row.
__global__ void k_row_hist(const uint32_t* __restrict__ keys, int64_t m,
                           int32_t* __restrict__ cnt) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e < m) atomicAdd(&cnt[keys[e]], 1);
}

// CSR columns and clipped values from the sorted runs.
__global__ void k_runs_to_csr(const uint2* __restrict__ vals, int64_t m, float lo, float hi,
                              uint32_t* __restrict__ idx, float* __restrict__ w) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= m) return;
  float v = __uint_as_float(vals[e].y);
  if (v < lo)
    v = lo;
  else if (v > hi)
    v = hi;
  idx[e] = vals[e].x;
  w[e] = v;
}

// ---------------------------------------------------------------------------
// Canonical graphs (symmetric, sorted rows, equal weights both ways): row j of G
// lists column j's entries too, so both products of a level are sums over one
// row, grouped by the part of the neighbour (row_groups.cuh), and no entry has
// to be sorted across rows. Needs at most RG_LABELS parts.
// The coarse graphs of a canonical one have sorted rows and entries both ways, with
// weights that need not be equal: there (TWIN) an entry's other weight is searched
// for in its column's row. Levels of 644 and 11,274 nodes spend 0.20 and 0.54 ms on both
// products so, 0.43 and 1.09 with a transpose and sorts of all entries.
// ---------------------------------------------------------------------------
struct RowGraph {
  const int64_t* indptr;
  const uint32_t* indices;
  const float* w;
  const uint32_t* part;
  const float* inv;
};

// The weight of (j, i): a binary search of row j for column i, which is there.
__device__ __forceinline__ float twin_weight(const RowGraph& g, uint32_t j, uint32_t i) {
  int64_t a = g.indptr[j], b = g.indptr[j + 1] - 1;
  while (a < b) {
    const int64_t m = (a + b) >> 1;
    if (g.indices[m] < i)
      a = m + 1;
    else
      b = m;
  }
  return g.w[a];
}

// Entry q = (i, j)'s label and product: inv_P * w_ji of the coarse graph, or (SYM) the
// expansion's (w_ij * w_ji) * inv_Q (the symmetric part).
template <bool SYM, bool TWIN>
__device__ __forceinline__ uint32_t row_entry(const RowGraph& g, uint32_t i, int64_t q, float* v) {
  const uint32_t j = g.indices[q], l = g.part[j];
  const float w = g.w[q], t = TWIN ? twin_weight(g, j, i) : w;
  *v = SYM ? fmul(fmul(w, t), g.inv[l]) : fmul(g.inv[l], t);
  return l;
}

template <bool SYM, bool TWIN, int CAP>
__device__ __forceinline__ int row_groups(const RowGraph& g, RgWarp<CAP>& sm, int64_t i, int64_t b,
                                          int len, int lane) {
  for (int p = lane; p < len; p += 32) {
    float v;
    const uint32_t l = row_entry<SYM, TWIN>(g, (uint32_t)i, b + p, &v);
    sm.key[p] = (l << RG_POS_BITS) | (uint32_t)p;
    sm.val[p] = v;
  }
  return rg_group(sm, len, lane);
}

template <bool SYM, bool TWIN>
__device__ __forceinline__ int long_row_groups(const RowGraph& g, RgLong& sm, uint32_t i) {
  const int64_t b = g.indptr[i], e = g.indptr[i + 1];
  rg_long_clear(sm);
  for (int64_t c = b; c < e; c += RG_CHUNK) {
    for (int q = threadIdx.x; q < RG_CHUNK; q += RG_LONG_THREADS) {
      uint32_t key = 0xffffffffu;
      float v = 0.0f;
      if (c + q < e) key = (row_entry<SYM, TWIN>(g, i, c + q, &v) << 10) | (uint32_t)q;
      sm.key[q] = key;
      sm.val[q] = v;
    }
    rg_long_chunk(sm, nullptr, 0u);
  }
  return rg_long_list(sm);
}

// Coarse graph, first product: row j's (P, sum of inv_P w_ij over i in P), P
// ascending, at the head of the row's CSR range in tmp; cnt[j] of them.
template <bool TWIN, int CAP>
__device__ __forceinline__ void coarse_row(const RowGraph& g, RgWarp<CAP>& sm, int64_t j, int64_t b,
                                           int len, int lane, uint2* __restrict__ tmp,
                                           int32_t* __restrict__ cnt) {
  const int runs = row_groups<false, TWIN>(g, sm, j, b, len, lane);
  for (int r = lane; r < runs; r += 32)
    tmp[b + r] = make_uint2(sm.key[sm.start[r]] >> RG_POS_BITS, __float_as_uint(sm.sum[r]));
  if (lane == 0) cnt[j] = runs;
}

template <bool TWIN>
__global__ void __launch_bounds__(32 * RG_WARPS, RG_BLOCKS) k_coarse_rows(RowGraph g, int64_t n,
                                                               uint2* __restrict__ tmp,
                                                               int32_t* __restrict__ cnt,
                                                               RgLists lists) {
  __shared__ RgWarp<RG_CAP> sm_all[RG_WARPS];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int64_t j = (int64_t)blockIdx.x * RG_WARPS + wid;
  if (j >= n) return;
  const int64_t b = g.indptr[j], len = g.indptr[j + 1] - b;
  if (rg_defer(lists, j, len, lane)) return;
  coarse_row<TWIN>(g, sm_all[wid], j, b, (int)len, lane, tmp, cnt);
}

template <bool TWIN>
__global__ void __launch_bounds__(32 * RG_MID_WARPS) k_coarse_rows_mid(RowGraph g,
                                                                       uint2* __restrict__ tmp,
                                                                       int32_t* __restrict__ cnt,
                                                                       RgLists lists) {
  extern __shared__ __align__(16) unsigned char rg_raw[];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  RgWarp<RG_MID>& sm = reinterpret_cast<RgWarp<RG_MID>*>(rg_raw)[wid];
  for (int64_t j; (j = rg_next_mid(lists, lane)) >= 0;) {
    __syncwarp();  // the previous row's readers are done
    coarse_row<TWIN>(g, sm, j, g.indptr[j], (int)(g.indptr[j + 1] - g.indptr[j]), lane, tmp, cnt);
  }
}

template <bool TWIN>
__global__ void __launch_bounds__(RG_LONG_THREADS) k_coarse_rows_long(
    RowGraph g, uint2* __restrict__ tmp, int32_t* __restrict__ cnt, RgLists lists) {
  extern __shared__ __align__(16) unsigned char rg_raw[];
  RgLong& sm = *reinterpret_cast<RgLong*>(rg_raw);
  const int nl = lists.count[1];
  for (int item = blockIdx.x; item < nl; item += gridDim.x) {
    const uint32_t j = lists.longs[item];
    const int64_t b = g.indptr[j];
    const int runs = long_row_groups<false, TWIN>(g, sm, j);
    for (int r = threadIdx.x; r < runs; r += RG_LONG_THREADS) {
      const uint32_t l = sm.list[r];
      tmp[b + r] = make_uint2(l, __float_as_uint(sm.acc[l]));
    }
    if (threadIdx.x == 0) cnt[j] = runs;
  }
}

// cnt of the nodes in part order.
__global__ void k_perm_counts(const uint2* __restrict__ nodes, int64_t n,
                              const int32_t* __restrict__ cnt, int32_t* __restrict__ out) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t < n) out[t] = cnt[nodes[t].x];
}

// The rows' sums in (Q = part(j), j) order: key P, value (Q, sum). Eight lanes
// per row (a row has about ten parts).
__global__ void k_coarse_gather(const uint2* __restrict__ nodes, int64_t n,
                                const int64_t* __restrict__ indptr,
                                const uint32_t* __restrict__ part, const uint2* __restrict__ tmp,
                                const int64_t* __restrict__ off, uint32_t* __restrict__ keys,
                                uint2* __restrict__ vals) {
  const int64_t t = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 3;
  if (t >= n) return;
  const uint32_t j = nodes[t].x, Q = part[j];
  const uint2* src = tmp + indptr[j];
  const int64_t o = off[t];
  const int c = (int)(off[t + 1] - o);
  for (int r = threadIdx.x & 7; r < c; r += 8) {
    const uint2 v = src[r];
    keys[o + r] = v.x;
    vals[o + r] = make_uint2(Q, v.y);
  }
}

// Expansion: row i's (Q, e) groups, L1-normalised (serial over Q), times the
// coarse layout (serial over Q, a lane per dimension), plus the direct term,
// halved: res[i][k]. Label and sum of run r come from the two accessors.
template <class Label, class Sum>
__device__ __forceinline__ void expand_row(int64_t i, int runs, int lane, int32_t dim,
                                           const float* __restrict__ layout,
                                           const uint32_t* __restrict__ part,
                                           const float* __restrict__ u, float* __restrict__ res,
                                           Label label, Sum sum) {
  float nrm = 0.0f;
  for (int r = 0; r < runs; ++r) nrm = fadd(nrm, fabsf(sum(r)));
  const bool scale = nrm > 0.0f;
  const float sc = scale ? fdiv(1.0f, nrm) : 1.0f;
  if (lane >= dim) return;
  float acc = 0.0f;
#pragma unroll 4
  for (int r = 0; r < runs; ++r) {
    const float e = sum(r);
    const float v = scale ? fmul(e, sc) : e;
    acc = fadd(acc, fmul(v, layout[(int64_t)label(r) * dim + lane]));
  }
  const uint32_t P = part[i];
  const float direct = fadd(0.0f, fmul(u[P], layout[(int64_t)P * dim + lane]));
  res[i * dim + lane] = fmul(fadd(acc, direct), 0.5f);
}

template <bool TWIN, int CAP>
__device__ __forceinline__ void expand_warp_row(const RowGraph& g, RgWarp<CAP>& sm, int64_t i,
                                                int64_t b, int len, int lane, int32_t dim,
                                                const float* __restrict__ layout,
                                                const float* __restrict__ u,
                                                float* __restrict__ res) {
  const int runs = row_groups<true, TWIN>(g, sm, i, b, len, lane);
  expand_row(
      i, runs, lane, dim, layout, g.part, u, res,
      [&](int r) { return sm.key[sm.start[r]] >> RG_POS_BITS; }, [&](int r) { return sm.sum[r]; });
}

template <bool TWIN>
__global__ void __launch_bounds__(32 * RG_WARPS, RG_BLOCKS) k_expand_groups(
    RowGraph g, int64_t n, int32_t dim, const float* __restrict__ layout,
    const float* __restrict__ u, float* __restrict__ res, RgLists lists) {
  __shared__ RgWarp<RG_CAP> sm_all[RG_WARPS];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int64_t i = (int64_t)blockIdx.x * RG_WARPS + wid;
  if (i >= n) return;
  const int64_t b = g.indptr[i], len = g.indptr[i + 1] - b;
  if (rg_defer(lists, i, len, lane)) return;
  expand_warp_row<TWIN>(g, sm_all[wid], i, b, (int)len, lane, dim, layout, u, res);
}

template <bool TWIN>
__global__ void __launch_bounds__(32 * RG_MID_WARPS) k_expand_groups_mid(
    RowGraph g, int32_t dim, const float* __restrict__ layout, const float* __restrict__ u,
    float* __restrict__ res, RgLists lists) {
  extern __shared__ __align__(16) unsigned char rg_raw[];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  RgWarp<RG_MID>& sm = reinterpret_cast<RgWarp<RG_MID>*>(rg_raw)[wid];
  for (int64_t i; (i = rg_next_mid(lists, lane)) >= 0;) {
    __syncwarp();  // the previous row's readers are done
    expand_warp_row<TWIN>(g, sm, i, g.indptr[i], (int)(g.indptr[i + 1] - g.indptr[i]), lane, dim, layout,
                    u, res);
  }
}

template <bool TWIN>
__global__ void __launch_bounds__(RG_LONG_THREADS) k_expand_groups_long(
    RowGraph g, int32_t dim, const float* __restrict__ layout, const float* __restrict__ u,
    float* __restrict__ res, RgLists lists) {
  extern __shared__ __align__(16) unsigned char rg_raw[];
  RgLong& sm = *reinterpret_cast<RgLong*>(rg_raw);
  const int nl = lists.count[1];
  for (int item = blockIdx.x; item < nl; item += gridDim.x) {
    const uint32_t i = lists.longs[item];
    const int runs = long_row_groups<true, TWIN>(g, sm, i);
    if (threadIdx.x < 32)
      expand_row(
          (int64_t)i, runs, (int)threadIdx.x, dim, layout, g.part, u, res,
          [&](int r) { return (uint32_t)sm.list[r]; }, [&](int r) { return sm.acc[sm.list[r]]; });
  }
}

// ---------------------------------------------------------------------------
// Data reduction: block per part, thread per feature column.
// ---------------------------------------------------------------------------
// Block (part, 128 feature columns); thread per column. The sum over the
// part's nodes stays serial in node order. Node ids come through shared
// memory 128 at a time, and each thread issues the loads of the next 16
// nodes before their adds, so a large part is not one long chain of
// dependent loads.
constexpr int RD_THREADS = 128;
__global__ void __launch_bounds__(RD_THREADS) k_reduce_data(
    const float* __restrict__ x, int64_t d, const int64_t* __restrict__ poff,
    const uint2* __restrict__ nodes, const float* __restrict__ rv, float* __restrict__ out) {
  constexpr int U = 16;
  __shared__ uint32_t ids[RD_THREADS];
  const int64_t P = blockIdx.x;
  const int64_t k = (int64_t)blockIdx.y * RD_THREADS + threadIdx.x;
  const bool on = k < d;
  const float v = rv[P];
  const int64_t a = poff[P], b = poff[P + 1];
  float acc = 0.0f;
  for (int64_t c = a; c < b; c += RD_THREADS) {
    const int cnt = (int)min((int64_t)RD_THREADS, b - c);
    __syncthreads();  // the previous chunk's ids are read
    if ((int)threadIdx.x < cnt) ids[threadIdx.x] = nodes[c + threadIdx.x].x;
    __syncthreads();
    if (on) {
      int q = 0;
      for (; q + U <= cnt; q += U) {
        float xv[U];
#pragma unroll
        for (int u = 0; u < U; ++u) xv[u] = __ldg(x + (int64_t)ids[q + u] * d + k);
#pragma unroll
        for (int u = 0; u < U; ++u) acc = fadd(acc, fmul(v, xv[u]));
      }
      for (; q < cnt; ++q) acc = fadd(acc, fmul(v, __ldg(x + (int64_t)ids[q] * d + k)));
    }
  }
  if (on) out[P * d + k] = acc;
}

// ---------------------------------------------------------------------------
// Expansion.
// ---------------------------------------------------------------------------
// Products of the symmetric part G o G^T (rows merged with the transpose's,
// both sorted) times N: key Q = part(j), value (i, s_ij * inv_Q), in
// row-major order (canonical graphs pass themselves as the transpose).
__global__ void k_sym_count(const int64_t* __restrict__ ap, const uint32_t* __restrict__ ai,
                            const int64_t* __restrict__ bp, const uint32_t* __restrict__ bi,
                            int64_t n, int32_t* __restrict__ cnt) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  int64_t p = ap[i], q = bp[i];
  const int64_t ep = ap[i + 1], eq = bp[i + 1];
  int32_t c = 0;
  while (p < ep && q < eq) {
    if (ai[p] == bi[q]) {
      ++c;
      ++p;
      ++q;
    } else if (ai[p] < bi[q]) {
      ++p;
    } else {
      ++q;
    }
  }
  cnt[i] = c;
}

__global__ void k_sym_products(const int64_t* __restrict__ ap, const uint32_t* __restrict__ ai,
                               const float* __restrict__ aw, const int64_t* __restrict__ bp,
                               const uint32_t* __restrict__ bi, const float* __restrict__ bw,
                               int64_t n, const int64_t* __restrict__ off,
                               const uint32_t* __restrict__ part, const float* __restrict__ inv,
                               uint32_t* __restrict__ keys, uint2* __restrict__ vals) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  int64_t p = ap[i], q = bp[i], o = off[i];
  const int64_t ep = ap[i + 1], eq = bp[i + 1];
  while (p < ep && q < eq) {
    if (ai[p] == bi[q]) {
      const uint32_t j = ai[p];
      const float sv = fmul(aw[p], bw[q]);  // sparse.rs:378-417
      const uint32_t Q = part[j];
      keys[o] = Q;
      vals[o] = make_uint2((uint32_t)i, __float_as_uint(fmul(sv, inv[Q])));
      ++o;
      ++p;
      ++q;
    } else if (ai[p] < bi[q]) {
      ++p;
    } else {
      ++q;
    }
  }
}

// Row i of the expander (runs (i, Q, e) sorted by (i, Q)), L1-normalised, times
// the coarse layout, plus the direct term, halved: res[i][k].
__global__ void k_expand_rows(const int64_t* __restrict__ eptr, const uint2* __restrict__ ev,
                              int64_t n, int32_t dim, const float* __restrict__ layout,
                              const uint32_t* __restrict__ part, const float* __restrict__ u,
                              float* __restrict__ res) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int64_t a = eptr[i], b = eptr[i + 1];
  float nrm = 0.0f;
  for (int64_t e = a; e < b; ++e) nrm = fadd(nrm, fabsf(__uint_as_float(ev[e].y)));
  const float sc = nrm > 0.0f ? fdiv(1.0f, nrm) : 1.0f;
  const bool scale = nrm > 0.0f;
  const uint32_t P = part[i];
  const float dv = u[P];
  for (int32_t k = 0; k < dim; ++k) {
    float acc = 0.0f;
    for (int64_t e = a; e < b; ++e) {
      const float v = scale ? fmul(__uint_as_float(ev[e].y), sc) : __uint_as_float(ev[e].y);
      acc = fadd(acc, fmul(v, layout[(int64_t)ev[e].x * dim + k]));
    }
    const float direct = fadd(0.0f, fmul(dv, layout[(int64_t)P * dim + k]));
    res[i * dim + k] = fmul(fadd(acc, direct), 0.5f);
  }
}

// Column centring: serial column sums over all rows, then scaling.
//
// The sum s + x0 + x1 + ... rounds after each addition, so added one by one it is a
// chain of n additions (5.8 cycles each fed from shared memory: 6.0 ms for 2 M rows).
// But while the sum stays inside one binade its values are integers m of one unit
// u, 2^23 < m < 2^24, and an addition is m += rint(x / u), where only a tie looks
// at the sum: it goes to the even neighbour, so its step depends on m's parity. A
// run of additions is then a pair of integers, its total step from an even and from
// an odd m, and two runs compose: (a b)_p = a_p + b_((p + a_p) & 1). One block per
// column takes CM_CHUNK values at a time: a thread composes CM_K of them, a block
// scan gives each thread the m that its run begins with, and the thread checks that
// its run keeps inside the binade. From the first run that does not (or whose
// values are not finite, or above a quarter of the sum), warp 0 adds one by one;
// twice as many each time that a chunk ends early, so that sums which never settle
// cost little more than the chain. The result is the chain's, bit for bit.
// 2 M rows of 8 columns, by the chain 6.0 ms whatever they hold: 0.42 ms with a mean
// of three deviations, 0.74 ms of 0.01, 2.9 ms for pure noise (a sum that crosses
// binades all the time), 5.9 ms for x, -x, x, -x (never in chunks).
constexpr int CM_THREADS = 512;
constexpr int CM_K = 16;
constexpr int CM_CHUNK = CM_THREADS * CM_K;
constexpr int CM_RUN = 256;        // additions of one serial unit
constexpr int CM_MAX_UNITS = 64;
constexpr float CM_ROUND = 12582912.0f;  // 1.5 * 2^23: adding it rounds to an integer
constexpr int CM_WORTH = 512;      // values in steps that pay for a chunk's work
// The first values are always added one by one: a young sum soon leaves its binade
// (8192 values of noise 24 us so, 45 us in chunks).
constexpr int64_t CM_HEAD = CM_CHUNK;
// Above this many rows the columns are first copied out (k_columns): value i of a
// column then lies in plane (i / 4) % 4, at float 4 (i / 16) + i % 4, so that the 16
// values of each thread are four coalesced loads of a warp rather than 16 scattered.
constexpr int64_t CM_DIRECT = CM_HEAD;
__device__ __forceinline__ int64_t cm_index(int64_t i, int64_t groups) {
  return ((i >> 2) & 3) * 4 * groups + 4 * (i >> 4) + (i & 3);
}

struct SumStep {
  int even, odd;  // total step from an even and from an odd sum
};
// (Sums wrap where a run is already known to leave the binade.)
__device__ __forceinline__ int wrap_add(int a, int b) { return (int)((unsigned)a + (unsigned)b); }
__device__ __forceinline__ SumStep then(SumStep a, SumStep b) {
  return {wrap_add(a.even, (a.even & 1) ? b.odd : b.even),
          wrap_add(a.odd, (a.odd & 1) ? b.even : b.odd)};
}
// Lane l: the composition of lanes 0..l.
__device__ __forceinline__ SumStep warp_steps(SumStep x, int lane) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    SumStep y;
    y.even = __shfl_up_sync(0xffffffffu, x.even, o);
    y.odd = __shfl_up_sync(0xffffffffu, x.odd, o);
    if (lane >= o) x = then(y, x);
  }
  return x;
}

// COLS: column j is x[16 j ld ..], ld groups of CM_K values in cm_index order with
// zeros from n up; else value i of column j is x[i * ld + j].
template <bool COLS>
__global__ void __launch_bounds__(CM_THREADS) k_col_mean(const float* __restrict__ x, int64_t n,
                                                        int64_t ld, float inv_n,
                                                        float* __restrict__ mean) {
  constexpr unsigned FULL = 0xffffffffu;
  constexpr int WARPS = CM_THREADS / 32;
  __shared__ SumStep agg[WARPS];
  __shared__ int first_sh, m_sh;
  __shared__ float s_sh;
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  __shared__ __align__(16) float run[CM_RUN];
  const float* col = COLS ? x + blockIdx.x * CM_K * ld : x + blockIdx.x;
  auto at = [&](int64_t i) {
    return i < n ? col[COLS ? cm_index(i, ld) : i * ld] : 0.0f;
  };
  auto load = [&](int64_t p, float (&v)[CM_K]) {  // values p .. p + CM_K - 1
    if constexpr (COLS) {
      const float4* c4 = reinterpret_cast<const float4*>(col) + p / CM_K;
#pragma unroll
      for (int q = 0; q < CM_K / 4; ++q) {
        const float4 t = p < n ? __ldg(c4 + q * ld) : make_float4(0.f, 0.f, 0.f, 0.f);
        v[4 * q] = t.x, v[4 * q + 1] = t.y, v[4 * q + 2] = t.z, v[4 * q + 3] = t.w;
      }
    } else {
#pragma unroll
      for (int k = 0; k < CM_K; ++k) v[k] = at(p + k);
    }
  };
  float s = 0.0f;  // the sum of the values below pos, in every thread
  int64_t pos = 0;  // a multiple of CM_K
  int units = 1;
  float v[CM_K];
  int64_t held = -1;  // the chunk that v belongs to
  while (pos < n) {
    const int bits = __float_as_int(s), ex = (bits >> 23) & 255;
    int first = 0;
    if (ex >= 27 && ex <= 227) {  // a normal sum, and so are its unit and the inverse
      const bool neg = bits < 0;
      const float inv = __int_as_float((277 - ex) << 23 | (bits & 0x80000000));  // +-1 / u
      const int m = (bits & 0x7fffff) | 0x800000;
      if (held != pos) {
        load(pos + tid * CM_K, v);
        held = pos;
      }
      SumStep d = {0, 0};
      int lo = 0, hi = 0;
      bool near = true, tie = false;
#pragma unroll
      for (int k = 0; k < CM_K; ++k) {
        const float t = fmul(v[k], inv);  // exact, or far below half a unit
        near = near && fabsf(t) < 4194304.0f;  // no for NaN
        const float y = fadd(t, CM_ROUND);
        tie = tie || fabsf(fsub(t, fsub(y, CM_ROUND))) == 0.5f;
        d.even = wrap_add(d.even, __float_as_int(y) - __float_as_int(CM_ROUND));
        lo = min(lo, d.even);
        hi = max(hi, d.even);
      }
      if (!near) d.even = lo = hi = 0;
      d.odd = d.even;
      if (near && tie) {
        d = {0, 0};
        lo = hi = 0;
#pragma unroll
        for (int k = 0; k < CM_K; ++k) {
          const float t = fmul(v[k], inv), y = fadd(t, CM_ROUND);
          const float rem = fsub(t, fsub(y, CM_ROUND));
          const int i = __float_as_int(y) - __float_as_int(CM_ROUND);
          const int w = fabsf(rem) == 0.5f ? (rem > 0.0f ? 1 : -1) : 0;  // from an odd sum
          d.even += i + ((d.even & 1) ? w : 0);
          d.odd += i + ((d.odd & 1) ? 0 : w);
          lo = min(lo, d.even);
          hi = max(hi, d.even);
        }
      }
      const int64_t ahead = pos + CM_CHUNK;
      if (ahead < n) {
        load(ahead + tid * CM_K, v);
        held = ahead;
      }
      const SumStep inc = warp_steps(d, lane);
      SumStep before;
      before.even = __shfl_up_sync(FULL, inc.even, 1);
      before.odd = __shfl_up_sync(FULL, inc.odd, 1);
      if (lane == 0) before = {0, 0};
      if (lane == 31) agg[wid] = inc;
      if (tid == 0) first_sh = CM_THREADS;
      __syncthreads();
      const SumStep all = warp_steps(lane < WARPS ? agg[lane] : SumStep{0, 0}, lane);
      SumStep base;
      base.even = __shfl_sync(FULL, all.even, max(wid - 1, 0));
      base.odd = __shfl_sync(FULL, all.odd, max(wid - 1, 0));
      if (wid > 0) before = then(base, before);
      const int mt = wrap_add(m, (m & 1) ? before.odd : before.even);
      // a run's values from an odd sum are within 2 of lo and hi
      const bool leaves =
          !near || wrap_add(mt, lo - 2) <= (1 << 23) || wrap_add(mt, hi + 2) >= (1 << 24);
      const unsigned out = __ballot_sync(FULL, leaves);
      if (lane == 0 && out) atomicMin(&first_sh, wid * 32 + __ffs(out) - 1);
      __syncthreads();
      first = first_sh;
      if (first < CM_THREADS) {
        if (tid == first) m_sh = mt;
      } else if (tid == CM_THREADS - 1) {
        m_sh = mt + ((mt & 1) ? d.odd : d.even);
      }
      __syncthreads();
      // m_sh * u with the sign of s: exact, m_sh stays below 2^24
      const float mag = fmul((float)m_sh, __int_as_float((ex - 23) << 23));
      s = neg ? -mag : mag;
      pos = min(n, pos + (int64_t)first * CM_K);
    }
    if (first < CM_THREADS && pos < n) {
      if (first * CM_K >= CM_WORTH) units = 1;
      const int64_t end = min(n, pos == 0 ? CM_HEAD : pos + (int64_t)CM_RUN * units);
      if (wid == 0) {
        float a = s, c[CM_RUN / 32];
#pragma unroll
        for (int q = 0; q < CM_RUN / 32; ++q) c[q] = at(pos + 32 * q + lane);
        for (int64_t p = pos; p < end; p += CM_RUN) {
          float nx[CM_RUN / 32];
#pragma unroll
          for (int q = 0; q < CM_RUN / 32; ++q) nx[q] = at(p + CM_RUN + 32 * q + lane);
#pragma unroll
          for (int q = 0; q < CM_RUN / 32; ++q) run[32 * q + lane] = c[q];
          __syncwarp();
#pragma unroll 16
          for (int q = 0; q < CM_RUN / 4; ++q) {  // past the end: + 0, the sum is never -0
            const float4 t = reinterpret_cast<const float4*>(run)[q];
            a = fadd(fadd(fadd(fadd(a, t.x), t.y), t.z), t.w);
          }
          __syncwarp();
#pragma unroll
          for (int q = 0; q < CM_RUN / 32; ++q) c[q] = nx[q];
        }
        if (lane == 0) s_sh = a;
      }
      __syncthreads();
      s = s_sh;
      __syncthreads();
      pos = end;
      units = end == CM_HEAD ? 1 : min(2 * units, CM_MAX_UNITS);
    } else {
      units = 1;
    }
  }
  if (tid == 0) mean[blockIdx.x] = fmul(s, inv_n);
}

// Rows (n x dim, dim <= 16) to columns of ld groups of CM_K floats in cm_index order,
// zeros from n up.
__global__ void __launch_bounds__(256) k_columns(const float* __restrict__ x, int64_t n,
                                                int32_t dim, int64_t ld,
                                                float* __restrict__ cols) {
  __shared__ float tile[16][256 + 1];
  const int64_t r0 = (int64_t)blockIdx.x * 256;
  const int tid = threadIdx.x;
  const int rows = (int)min((int64_t)256, n - r0);
  for (int q = tid; q < rows * dim; q += 256) {
    const int r = q / dim;
    tile[q - r * dim][r] = __ldg(x + r0 * dim + q);
  }
  __syncthreads();
  if (r0 + tid < ld * CM_K) {
    cols += cm_index(r0 + tid, ld);
    for (int j = 0; j < dim; ++j) cols[j * ld * CM_K] = tid < rows ? tile[j][tid] : 0.0f;
  }
}

// mean[j] = inv_n * (the serial sum of column j of x).
void column_means(const float* x, int64_t n, int32_t dim, float inv_n, float* mean,
                  cudaStream_t s) {
  DevBuf<float> cols;
  const int64_t ld = (n + CM_K - 1) / CM_K;
  bool by_cols = n > CM_DIRECT;
  if (by_cols) {
    try {
      cols.alloc(ld * CM_K * dim, s);
    } catch (const Error&) {  // no room for the copy: the strided form needs none
      by_cols = false;
    }
  }
  if (by_cols) {
    k_columns<<<grid_of(ld * CM_K), 256, 0, s>>>(x, n, dim, ld, cols.get());
    EVOC_CHECK_LAUNCH();
    k_col_mean<true><<<dim, CM_THREADS, 0, s>>>(cols.get(), n, ld, inv_n, mean);
  } else {
    k_col_mean<false><<<dim, CM_THREADS, 0, s>>>(x, n, dim, inv_n, mean);
  }
  EVOC_CHECK_LAUNCH();
}

__global__ void k_center_scale(float* __restrict__ res, int64_t n, int32_t dim,
                               const float* __restrict__ mean, float scale) {
  const int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= n * dim) return;
  const int32_t j = (int32_t)(q % dim);
  res[q] = fmul(scale, fsub(res[q], mean[j]));
}

// Random init of the base case (label_prop.rs:338-360): uniform in [-1, 1],
// rows L2-normalised in double. Philox counter (q_lo, q_hi, "LP", "RINI").
__global__ void k_lp_random_init(float* __restrict__ out, int64_t n, int32_t dim, uint64_t seed) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float r[32];
  double nrm = 0.0;
  for (int32_t j = 0; j < dim; ++j) {
    const uint64_t q = (uint64_t)i * dim + j;
    const uint4 o = philox4x32_10(make_uint4((uint32_t)q, (uint32_t)(q >> 32), 0x4C50u, 0x52494E49u),
                                  make_uint2((uint32_t)seed, (uint32_t)(seed >> 32)));
    const double uu = (double)((((uint64_t)o.y << 32) | o.x) >> 11) * (1.0 / 9007199254740992.0);
    r[j] = (float)__dsub_rn(__dmul_rn(uu, 2.0), 1.0);
    nrm = __dadd_rn(nrm, __dmul_rn((double)r[j], (double)r[j]));
  }
  nrm = __dsqrt_rn(nrm);
  for (int32_t j = 0; j < dim; ++j)
    out[i * dim + j] = nrm > 0.0 ? (float)__ddiv_rn((double)r[j], nrm) : r[j];
}

// ---------------------------------------------------------------------------
// Host: the PCA base case (double, Jacobi eigen-solve of the Gram matrix).
// ---------------------------------------------------------------------------
void host_unit_range(std::vector<float>& m, int64_t n, int64_t d) {
  for (int64_t j = 0; j < d; ++j) {
    float lo = INFINITY, hi = -INFINITY;
    for (int64_t i = 0; i < n; ++i) {
      const float v = m[i * d + j];
      if (v < lo) lo = v;
      if (v > hi) hi = v;
    }
    const float range = hi - lo;
    if (range > 0.0f) {
      const float mid = (hi + lo) / 2.0f, half = range / 2.0f;
      for (int64_t i = 0; i < n; ++i) m[i * d + j] = (m[i * d + j] - mid) / half;
    }
  }
}

void host_jacobi(std::vector<double>& a, int64_t k, std::vector<double>& w,
                 std::vector<double>& v) {
  v.assign((size_t)(k * k), 0.0);
  for (int64_t i = 0; i < k; ++i) v[i * k + i] = 1.0;
  for (int sweep = 0; sweep < 100; ++sweep) {
    double off = 0.0;
    for (int64_t p = 0; p < k; ++p)
      for (int64_t q = p + 1; q < k; ++q) off += a[p * k + q] * a[p * k + q];
    if (off < 1e-30) break;
    for (int64_t p = 0; p < k; ++p)
      for (int64_t q = p + 1; q < k; ++q) {
        const double apq = a[p * k + q];
        if (std::fabs(apq) < 1e-300) continue;
        const double theta = (a[q * k + q] - a[p * k + p]) / (2.0 * apq);
        const double t =
            (theta >= 0 ? 1.0 : -1.0) / (std::fabs(theta) + std::sqrt(theta * theta + 1.0));
        const double c = 1.0 / std::sqrt(t * t + 1.0), sn = t * c;
        for (int64_t r = 0; r < k; ++r) {
          const double ap = a[r * k + p], aq = a[r * k + q];
          a[r * k + p] = c * ap - sn * aq;
          a[r * k + q] = sn * ap + c * aq;
        }
        for (int64_t r = 0; r < k; ++r) {
          const double ap = a[p * k + r], aq = a[q * k + r];
          a[p * k + r] = c * ap - sn * aq;
          a[q * k + r] = sn * ap + c * aq;
        }
        for (int64_t r = 0; r < k; ++r) {
          const double vp = v[r * k + p], vq = v[r * k + q];
          v[r * k + p] = c * vp - sn * vq;
          v[r * k + q] = sn * vp + c * vq;
        }
      }
  }
  w.resize((size_t)k);
  for (int64_t i = 0; i < k; ++i) w[i] = a[i * k + i];
}

// Principal components of n points in d dims (n small): the top k = min(dim,
// n, d) eigenvectors of the centred Gram matrix, scaled by sqrt(eigenvalue),
// each signed so its largest-magnitude entry is positive, then unit-range
// normalised per column; columns beyond k are zero.
std::vector<float> host_pca_init(const std::vector<float>& data, int64_t n, int64_t d,
                                 int64_t dim) {
  const int64_t k = std::min(std::min(dim, n), d);
  std::vector<double> mean((size_t)d, 0.0);
  for (int64_t i = 0; i < n; ++i)
    for (int64_t j = 0; j < d; ++j) mean[j] += (double)data[i * d + j];
  const double inv_n = 1.0 / (double)n;
  for (double& m : mean) m *= inv_n;
  std::vector<double> x((size_t)(n * d));
  for (int64_t i = 0; i < n; ++i)
    for (int64_t j = 0; j < d; ++j) x[i * d + j] = (double)data[i * d + j] - mean[j];
  std::vector<double> g((size_t)(n * n), 0.0);
  for (int64_t a = 0; a < n; ++a)
    for (int64_t b = 0; b < n; ++b) {
      double acc = 0.0;
      for (int64_t j = 0; j < d; ++j) acc += x[a * d + j] * x[b * d + j];
      g[a * n + b] = acc;
    }
  std::vector<double> w, v;
  host_jacobi(g, n, w, v);
  std::vector<int64_t> order((size_t)n);
  for (int64_t i = 0; i < n; ++i) order[i] = i;
  std::sort(order.begin(), order.end(), [&](int64_t a, int64_t b) { return w[a] > w[b]; });
  std::vector<float> pc((size_t)(n * k));
  for (int64_t c = 0; c < k; ++c) {
    const int64_t e = order[c];
    const double sig = std::sqrt(std::max(w[e], 0.0));
    int64_t big = 0;
    for (int64_t i = 1; i < n; ++i)
      if (std::fabs(v[i * n + e]) > std::fabs(v[big * n + e])) big = i;
    const double sgn = v[big * n + e] < 0 ? -1.0 : 1.0;
    for (int64_t i = 0; i < n; ++i) pc[i * k + c] = (float)(sgn * v[i * n + e] * sig);
  }
  host_unit_range(pc, n, k);
  std::vector<float> out((size_t)(n * dim), 0.0f);
  for (int64_t i = 0; i < n; ++i)
    for (int64_t c = 0; c < k; ++c) out[i * dim + c] = pc[i * k + c];
  return out;
}

struct LpParams {
  int32_t n_lp_iter = 20;
  int64_t base_thr = 64;
  double scaling = 0.1;
};

// One level of label_prop_init_inner on graph g (device), data (device n x d
// or null): writes the n x dim initial embedding into d_out (device). twin: g has
// sorted rows and every entry's (j, i) too.
void lp_init_inner(evoc_ctx* ctx, const evoc_graph* g, int32_t dim, const float* d_data,
                   int64_t d, int32_t n_emb_epochs, int64_t approx_parts, uint64_t seed,
                   const LpParams& lp, float* d_out, bool twin = false) {
  cudaStream_t s = ctx->stream;
  const int64_t n = g->n;
  if (n < lp.base_thr) {  // label_prop.rs:440-445
    if (d_data && dim <= d) {
      std::vector<float> x((size_t)(n * d));
      EVOC_CUDA(cudaMemcpyAsync(x.data(), d_data, x.size() * sizeof(float),
                                cudaMemcpyDeviceToHost, s));
      EVOC_CUDA(cudaStreamSynchronize(s));
      const std::vector<float> pc = host_pca_init(x, n, d, dim);
      EVOC_CUDA(cudaMemcpyAsync(d_out, pc.data(), pc.size() * sizeof(float),
                                cudaMemcpyHostToDevice, s));
      EVOC_CUDA(cudaStreamSynchronize(s));
    } else if (n > 0) {
      k_lp_random_init<<<grid_of(n), 128, 0, s>>>(d_out, n, dim, seed);
      EVOC_CHECK_LAUNCH();
    }
    return;
  }
  // stage trace (EVOC_TRACE=1): one block per level, innermost level first
  StageTrace tr(s);
  const std::string lvl = "lp n=" + std::to_string(n) + ": ";
  auto mark = [&](const char* what) {
    if (tr.on) tr.mark((lvl + what).c_str());
  };
  // 1. partition (label_prop.rs:448)
  DevBuf<uint32_t> part(n, s);
  const int64_t np = label_prop_partition(ctx, g, approx_parts, lp.n_lp_iter, seed, part.get());
  mark("partition");
  if (np <= 0) throw Error(EVOC_ERR_INTERNAL, "label propagation produced no parts");
  // 2. per-part constants and node lists
  DevBuf<int32_t> cnt(np, s);
  EVOC_CUDA(cudaMemsetAsync(cnt.get(), 0, np * sizeof(int32_t), s));
  k_part_count<<<grid_of(n), 256, 0, s>>>(part.get(), n, cnt.get());
  EVOC_CHECK_LAUNCH();
  DevBuf<float> inv(np, s), rv(np, s), u(np, s);
  k_part_consts<<<grid_of(np, 128), 128, 0, s>>>(cnt.get(), np, inv.get(), rv.get(), u.get());
  EVOC_CHECK_LAUNCH();
  const int pbits = bits_for((uint64_t)std::max<int64_t>(np - 1, 1));
  const int nbits = bits_for((uint64_t)std::max<int64_t>(n - 1, 1));
  // the nodes in part order (stable sort of node ids by part)
  DevBuf<uint2> nodes(n, s);
  {
    DevBuf<uint32_t> pk(n, s);
    EVOC_CUDA(cudaMemcpyAsync(pk.get(), part.get(), n * sizeof(uint32_t),
                              cudaMemcpyDeviceToDevice, s));
    k_iota_pairs<<<grid_of(n), 256, 0, s>>>(nodes.get(), n);
    EVOC_CHECK_LAUNCH();
    radix_sort_pairs(ctx, pk, nodes, n, pbits);
  }
  // canonical graphs and those made from them sum within their rows; others by
  // sorting all entries
  const bool by_rows = (g->canonical || twin) && np <= RG_LABELS && g->nnz > 0;
  const RowGraph rg{g->indptr.get(), g->indices.get(), g->weights.get(), part.get(), inv.get()};
  DevBuf<uint32_t> row_lists;  // rows above RG_CAP: middle, long
  DevBuf<int32_t> row_counts;  // their counters: coarse graph, expansion
  RgLists lists{}, lists2{};
  const unsigned rgrid = (unsigned)((n + RG_WARPS - 1) / RG_WARPS);
  // no row is above RG_CAP (RG_MID) when the graph has no more entries than that
  const unsigned mgrid = g->nnz <= RG_CAP ? 0u : (unsigned)std::min<int64_t>(
      4 * (int64_t)ctx->num_sms, (g->nnz / RG_CAP + RG_MID_WARPS - 1) / RG_MID_WARPS);
  const unsigned lgrid = (unsigned)std::min<int64_t>(2 * (int64_t)ctx->num_sms, g->nnz / RG_MID);
  const size_t msmem = RG_MID_WARPS * sizeof(RgWarp<RG_MID>);
  auto* coarse_short = twin ? k_coarse_rows<true> : k_coarse_rows<false>;
  auto* coarse_mid = twin ? k_coarse_rows_mid<true> : k_coarse_rows_mid<false>;
  auto* coarse_long = twin ? k_coarse_rows_long<true> : k_coarse_rows_long<false>;
  auto* expand_short = twin ? k_expand_groups<true> : k_expand_groups<false>;
  auto* expand_mid = twin ? k_expand_groups_mid<true> : k_expand_groups_mid<false>;
  auto* expand_long = twin ? k_expand_groups_long<true> : k_expand_groups_long<false>;
  if (by_rows) {
    row_lists.alloc(2 * n, s);
    row_counts.alloc(6, s);
    EVOC_CUDA(cudaMemsetAsync(row_counts.get(), 0, row_counts.bytes(), s));
    lists = RgLists{row_lists.get(), row_lists.get() + n, row_counts.get()};
    lists2 = RgLists{row_lists.get(), row_lists.get() + n, row_counts.get() + 3};
    for (const void* f : {(const void*)coarse_long, (const void*)expand_long})
      EVOC_CUDA(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)sizeof(RgLong)));
    for (const void* f : {(const void*)coarse_mid, (const void*)expand_mid})
      EVOC_CUDA(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)msmem));
  }
  // 3. coarse graph clip(N^T G B)
  evoc_graph coarse;
  coarse.ctx = ctx;
  coarse.n = np;
  coarse.canonical = false;
  coarse.indptr.alloc(np + 1, s);
  {
    const int64_t m = g->nnz;
    DevBuf<uint32_t> keys, ok;
    DevBuf<uint2> vals, ov;
    int64_t runs = 0;
    if (by_rows) {
      // (P, a) per row j, gathered in (Q, j) order and sorted by P: (P, Q, j)
      DevBuf<uint2> tmp(m, s);
      DevBuf<int32_t> rcnt(n, s), pcnt(n, s);
      coarse_short<<<rgrid, 32 * RG_WARPS, 0, s>>>(rg, n, tmp.get(), rcnt.get(), lists);
      EVOC_CHECK_LAUNCH();
      if (lgrid) {
        coarse_long<<<lgrid, RG_LONG_THREADS, sizeof(RgLong), s>>>(rg, tmp.get(),
                                                                          rcnt.get(), lists);
        EVOC_CHECK_LAUNCH();
      }
      if (mgrid) {
        coarse_mid<<<mgrid, 32 * RG_MID_WARPS, msmem, s>>>(rg, tmp.get(), rcnt.get(),
                                                                  lists);
        EVOC_CHECK_LAUNCH();
      }
      k_perm_counts<<<grid_of(n), 256, 0, s>>>(nodes.get(), n, rcnt.get(), pcnt.get());
      EVOC_CHECK_LAUNCH();
      DevBuf<int64_t> off(n + 1, s);
      exclusive_scan_i32_to_i64(ctx, pcnt.get(), off.get(), n);
      EVOC_CUDA(cudaMemcpyAsync(&runs, off.get() + n, sizeof(int64_t), cudaMemcpyDeviceToHost, s));
      EVOC_CUDA(cudaStreamSynchronize(s));
      keys.alloc(runs, s);
      vals.alloc(runs, s);
      k_coarse_gather<<<grid_of(n * 8), 256, 0, s>>>(nodes.get(), n, g->indptr.get(), part.get(),
                                                     tmp.get(), off.get(), keys.get(),
                                                     vals.get());
      EVOC_CHECK_LAUNCH();
      radix_sort_pairs(ctx, keys, vals, runs, pbits);
    } else if (m > 0) {
      keys.alloc(m, s);
      vals.alloc(m, s);
      k_gen_products<<<grid_of(n * 32), 256, 0, s>>>(g->indptr.get(), g->indices.get(),
                                                     g->weights.get(), n, part.get(), inv.get(),
                                                     keys.get(), vals.get());
      EVOC_CHECK_LAUNCH();
      // keys j, vals (P, prod): order (P, j, i) -> runs (P, (j, A_Pj))
      k_swap_keys<<<grid_of(m), 256, 0, s>>>(keys.get(), vals.get(), m);  // keys P, vals (j, .)
      EVOC_CHECK_LAUNCH();
      runs = sort_and_sum(ctx, keys, vals, m, pbits, nbits);
      // (P, (j, a)) -> (P, Q = part(j), j order kept): stable sort by Q, then by P
      DevBuf<uint32_t> q(runs, s);
      k_map_keys<<<grid_of(runs), 256, 0, s>>>(q.get(), vals.get(), runs, part.get());
      EVOC_CHECK_LAUNCH();
      k_swap_keys<<<grid_of(runs), 256, 0, s>>>(keys.get(), vals.get(), runs);  // keys j, vals (P, a)
      EVOC_CHECK_LAUNCH();
      std::swap(keys, q);  // keys Q
      radix_sort_pairs(ctx, keys, vals, runs, pbits);
      k_swap_keys<<<grid_of(runs), 256, 0, s>>>(keys.get(), vals.get(), runs);  // keys P, vals (Q, a)
      EVOC_CHECK_LAUNCH();
      radix_sort_pairs(ctx, keys, vals, runs, pbits);
    }
    if (m > 0) {
      runs = sum_runs(ctx, keys.get(), vals.get(), runs, ok, ov);
      DevBuf<int32_t> rc(np, s);
      EVOC_CUDA(cudaMemsetAsync(rc.get(), 0, np * sizeof(int32_t), s));
      k_row_hist<<<grid_of(runs), 256, 0, s>>>(ok.get(), runs, rc.get());
      EVOC_CHECK_LAUNCH();
      exclusive_scan_i32_to_i64(ctx, rc.get(), coarse.indptr.get(), np);
      coarse.nnz = runs;
      coarse.indices.alloc(std::max<int64_t>(runs, 1), s);
      coarse.weights.alloc(std::max<int64_t>(runs, 1), s);
      k_runs_to_csr<<<grid_of(runs), 256, 0, s>>>(ov.get(), runs, 0.0f, 1.0f,
                                                  coarse.indices.get(), coarse.weights.get());
      EVOC_CHECK_LAUNCH();
    } else {
      EVOC_CUDA(cudaMemsetAsync(coarse.indptr.get(), 0, (np + 1) * sizeof(int64_t), s));
      coarse.nnz = 0;
    }
  }
  mark("coarse graph");
  // 4. coarse data: per part, its nodes in order
  DevBuf<float> cdata;
  if (d_data) {
    DevBuf<int64_t> poff(np + 1, s);
    exclusive_scan_i32_to_i64(ctx, cnt.get(), poff.get(), np);
    cdata.alloc(np * d, s);
    k_reduce_data<<<dim3((unsigned)np, (unsigned)((d + RD_THREADS - 1) / RD_THREADS)),
                    RD_THREADS, 0, s>>>(d_data, d, poff.get(), nodes.get(), rv.get(),
                                        cdata.get());
    EVOC_CHECK_LAUNCH();
  }
  mark("coarse data");
  // 5. recursion
  const int32_t e = std::min(n_emb_epochs, 255);
  DevBuf<float> cinit(np * dim, s), layout(np * dim, s);
  lp_init_inner(ctx, &coarse, dim, d_data ? cdata.get() : nullptr, d, e, approx_parts / 4,
                seed + 3000, lp, cinit.get(), g->canonical || twin);
  mark("coarser levels");
  // 6. short embedding of the coarse graph (label_prop.rs:486-498)
  {
    evoc_embed_params_t ep;
    evoc_embed_params_default(&ep);
    ep.n_epochs = e;
    ep.initial_alpha = (float)(0.001 * (double)e);
    std::vector<ProblemDesc> probs{ProblemDesc{&coarse, seed + 4000}};
    evoc_plan* pl = plan_create(ctx, probs, dim, ep);
    try {
      plan_run_device(pl, cinit.get(), layout.get());
    } catch (...) {
      plan_free(pl);
      throw;
    }
    EVOC_CUDA(cudaStreamSynchronize(s));
    plan_free(pl);
  }
  mark("coarse embedding");
  // 7. expansion (label_prop.rs:500-534)
  {
    if (by_rows) {
      expand_short<<<rgrid, 32 * RG_WARPS, 0, s>>>(rg, n, dim, layout.get(), u.get(), d_out,
                                                      lists2);
      EVOC_CHECK_LAUNCH();
      if (lgrid) {
        expand_long<<<lgrid, RG_LONG_THREADS, sizeof(RgLong), s>>>(
            rg, dim, layout.get(), u.get(), d_out, lists2);
        EVOC_CHECK_LAUNCH();
      }
      if (mgrid) {
        expand_mid<<<mgrid, 32 * RG_MID_WARPS, msmem, s>>>(rg, dim, layout.get(),
                                                                    u.get(), d_out, lists2);
        EVOC_CHECK_LAUNCH();
      }
    } else {
      // the transpose of g (rows of G^T, entries in row order)
      DevBuf<int64_t> tptr;
      DevBuf<uint32_t> tidx;
      DevBuf<float> tw;
      const int64_t *bp = g->indptr.get();
      const uint32_t* bi = g->indices.get();
      const float* bw = g->weights.get();
      if (!g->canonical && g->nnz > 0) {
        const int64_t m = g->nnz;
        DevBuf<uint32_t> tk(m, s);
        DevBuf<uint2> tv(m, s);
        k_transpose_gen<<<grid_of(n * 32), 256, 0, s>>>(g->indptr.get(), g->indices.get(),
                                                        g->weights.get(), n, tk.get(), tv.get());
        EVOC_CHECK_LAUNCH();
        radix_sort_pairs(ctx, tk, tv, m, nbits);
        DevBuf<int32_t> tc(n, s);
        EVOC_CUDA(cudaMemsetAsync(tc.get(), 0, n * sizeof(int32_t), s));
        k_row_hist<<<grid_of(m), 256, 0, s>>>(tk.get(), m, tc.get());
        EVOC_CHECK_LAUNCH();
        tptr.alloc(n + 1, s);
        exclusive_scan_i32_to_i64(ctx, tc.get(), tptr.get(), n);
        tidx.alloc(m, s);
        tw.alloc(m, s);
        k_unpack_pairs<<<grid_of(m), 256, 0, s>>>(tv.get(), m, tidx.get(), tw.get());
        EVOC_CHECK_LAUNCH();
        bp = tptr.get();
        bi = tidx.get();
        bw = tw.get();
      }
      mark("expansion: transpose");
      DevBuf<int32_t> sc(n, s);
      DevBuf<int64_t> soff(n + 1, s);
      k_sym_count<<<grid_of(n), 256, 0, s>>>(g->indptr.get(), g->indices.get(), bp, bi, n,
                                             sc.get());
      EVOC_CHECK_LAUNCH();
      exclusive_scan_i32_to_i64(ctx, sc.get(), soff.get(), n);
      int64_t ms = 0;
      EVOC_CUDA(cudaMemcpyAsync(&ms, soff.get() + n, sizeof(int64_t), cudaMemcpyDeviceToHost, s));
      EVOC_CUDA(cudaStreamSynchronize(s));
      DevBuf<uint32_t> keys(std::max<int64_t>(ms, 1), s);
      DevBuf<uint2> vals(std::max<int64_t>(ms, 1), s);
      DevBuf<int64_t> eptr(n + 1, s);
      int64_t runs = 0;
      if (ms > 0) {
        k_sym_products<<<grid_of(n), 256, 0, s>>>(g->indptr.get(), g->indices.get(),
                                                  g->weights.get(), bp, bi, bw, n, soff.get(),
                                                  part.get(), inv.get(), keys.get(), vals.get());
        EVOC_CHECK_LAUNCH();
        // keys Q, vals (i, prod): order (i, Q, j) -> runs (i, (Q, e))
        k_swap_keys<<<grid_of(ms), 256, 0, s>>>(keys.get(), vals.get(), ms);  // keys i, vals (Q, .)
        EVOC_CHECK_LAUNCH();
        mark("expansion: symmetric products");
        runs = sort_and_sum(ctx, keys, vals, ms, nbits, pbits);
      }
      mark("expansion: sort and sum");
      DevBuf<int32_t> rc(n, s);
      EVOC_CUDA(cudaMemsetAsync(rc.get(), 0, n * sizeof(int32_t), s));
      if (runs > 0) {
        k_row_hist<<<grid_of(runs), 256, 0, s>>>(keys.get(), runs, rc.get());
        EVOC_CHECK_LAUNCH();
      }
      exclusive_scan_i32_to_i64(ctx, rc.get(), eptr.get(), n);
      k_expand_rows<<<grid_of(n, 128), 128, 0, s>>>(eptr.get(), vals.get(), n, dim, layout.get(),
                                                    part.get(), u.get(), d_out);
      EVOC_CHECK_LAUNCH();
    }
    mark("expansion: rows");
    DevBuf<float> mean(dim, s);
    const float inv_n = (float)(1.0 / (double)n);
    column_means(d_out, n, dim, inv_n, mean.get(), s);
    k_center_scale<<<grid_of(n * dim), 256, 0, s>>>(d_out, n, dim, mean.get(),
                                                    (float)lp.scaling);
    EVOC_CHECK_LAUNCH();
    EVOC_CUDA(cudaStreamSynchronize(s));
  }
  mark("expansion: centring");
}

}  // namespace

void label_propagation_init_device(evoc_ctx* ctx, const evoc_graph* g, int32_t dim,
                                   const float* d_data, int64_t d, uint64_t seed, float* d_out) {
  if (dim < 1 || dim > 16) throw Error(EVOC_ERR_UNSUPPORTED, "dim must be in 1..16");
  const int64_t n = g->n;
  if (n <= 0) throw Error(EVOC_ERR_INVALID_ARGUMENT, "empty graph");
  if (d_data && d <= 0) throw Error(EVOC_ERR_INVALID_ARGUMENT, "data dimension must be > 0");
  // label_prop.rs:555-560: approx parts = clamp(8 sqrt(n), 256, 16384), at most n
  const int64_t parts = std::min<int64_t>(
      std::min<int64_t>(std::max<int64_t>((int64_t)(8.0 * std::sqrt((double)n)), 256), 16384), n);
  LpParams lp;
  lp_init_inner(ctx, g, dim, d_data, d, 50, parts, seed, lp, d_out);
}

}  // namespace evoc
