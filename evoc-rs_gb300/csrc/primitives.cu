// primitives.cu — device-wide exclusive scan and stable LSD radix sort.
//
// Both are deterministic (no floating point, fixed traversal order) and are
// used to build CSR offsets and the stable column-major transposes of the
// fuzzy union and of the embedding's per-node incidence lists.
//
// Both read their input once per pass: a block takes its tile by a counter,
// publishes the tile's sum and adds up the sums of the tiles before it (the
// decoupled look-back of Merrill and Garland, "Single-pass parallel prefix scan
// with decoupled look-back", 2016, and of the onesweep radix sort of Adinets and
// Merrill, 2022). Tiles are taken in order, so every tile that a block waits for
// is running or done. No wait is relied on all the same: after LOOKBACK_POLLS
// looks the reader sums the missing tile's input itself (the "decoupled
// fallback" of Smith, Levien and Owens, 2025), so every launch ends with the
// same result whatever is scheduled when.
#include "evoc_device.cuh"
#include "evoc_internal.h"

#include <algorithm>
#include <string>

namespace evoc {

[[noreturn]] void throw_cuda(cudaError_t e, const char* what, const char* file,
                             int line) {
  (void)cudaGetLastError();
  int code = (e == cudaErrorMemoryAllocation) ? EVOC_ERR_OUT_OF_MEMORY
                                              : EVOC_ERR_CUDA;
  throw Error(code, std::string(what) + " failed: " + cudaGetErrorString(e) +
                        " (" + file + ":" + std::to_string(line) + ")");
}

int bits_for(uint64_t max_value) {
  int b = 0;
  while (b < 64 && (max_value >> b) != 0) ++b;
  return b;
}

void check_status(evoc_ctx* ctx, const char* where) {
  int32_t st = 0;
  EVOC_CUDA(cudaMemcpyAsync(&st, ctx->status.get(), sizeof(int32_t),
                            cudaMemcpyDeviceToHost, ctx->stream));
  EVOC_CUDA(cudaStreamSynchronize(ctx->stream));
  if (st == 0) return;
  EVOC_CUDA(cudaMemsetAsync(ctx->status.get(), 0, sizeof(int32_t), ctx->stream));
  std::string w(where);
  if (st & ST_BAD_INDEX)
    throw Error(EVOC_ERR_INVALID_INPUT, w + ": an index is >= n");
  if (st & ST_BAD_VALUE)
    throw Error(EVOC_ERR_INVALID_INPUT, w + ": a distance or weight is NaN, or a coordinate "
                                            "is not finite");
  if (st & ST_EMPTY_ROW)
    throw Error(EVOC_ERR_INVALID_INPUT,
                w + ": empty kNN row with local_connectivity > 0");
  if (st & ST_CROSS_BLOCK)
    throw Error(EVOC_ERR_INVALID_INPUT, w + ": an edge joins two problems (graph not block-diagonal)");
  if (st & ST_WAIT_TIMEOUT)
    throw Error(EVOC_ERR_INTERNAL, w + ": a tensor-core wait timed out (results discarded)");
  if (st & ST_TOO_MANY_NEG)
    throw Error(EVOC_ERR_UNSUPPORTED,
                w + ": more than 2^20 negative samples per edge and epoch "
                    "(negative_sample_rate too large)");
  throw Error(EVOC_ERR_INTERNAL, w + ": device self-check failed");
}

namespace {

constexpr unsigned long long LB_SUM = 1ull << 62;     // the tile's own sum
constexpr unsigned long long LB_PREFIX = 2ull << 62;  // the sum up to and with the tile
constexpr unsigned long long LB_VALUE = (1ull << 62) - 1ull;
constexpr int LOOKBACK_POLLS = 1 << 14;  // about 10 ms; a tile takes microseconds

__device__ __forceinline__ void lb_store(unsigned long long* p, unsigned long long v) {
  *reinterpret_cast<volatile unsigned long long*>(p) = v;
}
// The published word of one tile, or 0 when it did not come in time.
__device__ __forceinline__ unsigned long long lb_wait(const unsigned long long* p) {
  const volatile unsigned long long* vp = p;
  unsigned long long v = *vp;
  for (int k = 0; (v & ~LB_VALUE) == 0ull && k < LOOKBACK_POLLS; ++k) v = *vp;
  return (v & ~LB_VALUE) ? v : 0ull;
}

// ---------------------------------------------------------------------------
// Scan: tiles of 4096 elements (512 threads x 8), one launch. Up to
// SCAN_ONE_BLOCK elements a single block walks the tiles and nothing is waited
// for. The bound is memory (4 or 8 bytes in, 8 out per element).
// ---------------------------------------------------------------------------
constexpr int SCAN_THREADS = 512;
constexpr int SCAN_ITEMS = 8;
constexpr int SCAN_TILE = SCAN_THREADS * SCAN_ITEMS;
// one block takes about 1 us per tile; the look-back needs a clearing launch
// first, which costs about as much as four tiles
constexpr int64_t SCAN_ONE_BLOCK = 4 * SCAN_TILE;

// A thread's eight values are consecutive: one slot of padding after each eight keeps
// the threads of a warp on different banks (a scan of 2,000 values 5.5 -> 3.7 us).
__device__ __forceinline__ int scan_slot(int i) { return i + (i >> 3); }
static_assert(SCAN_ITEMS == 8, "scan_slot");

struct ScanSmem {
  int64_t v[SCAN_TILE + SCAN_TILE / SCAN_ITEMS];
  int64_t warp_tot[SCAN_THREADS / 32];
  int64_t carry;
  int64_t tile;
};

// Exclusive scan of the tile in sm.v in place (without carry); returns its sum.
__device__ __forceinline__ int64_t scan_tile(ScanSmem& sm) {
  __syncthreads();
  int64_t local[SCAN_ITEMS];
  int64_t run = 0;
#pragma unroll
  for (int j = 0; j < SCAN_ITEMS; ++j) {
    local[j] = run;
    run += sm.v[scan_slot(threadIdx.x * SCAN_ITEMS + j)];
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int64_t incl = run;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int64_t y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  if (lane == 31) sm.warp_tot[warp] = incl;
  __syncthreads();
  int64_t before = 0, total = 0;
#pragma unroll
  for (int w = 0; w < SCAN_THREADS / 32; ++w) {
    const int64_t x = sm.warp_tot[w];
    if (w < warp) before += x;
    total += x;
  }
  const int64_t off = before + incl - run;
#pragma unroll
  for (int j = 0; j < SCAN_ITEMS; ++j) sm.v[scan_slot(threadIdx.x * SCAN_ITEMS + j)] = off + local[j];
  __syncthreads();
  return total;
}

template <typename Tin>
__device__ __forceinline__ void scan_load(ScanSmem& sm, const Tin* __restrict__ in, int64_t n,
                                          int64_t base) {
#pragma unroll
  for (int j = 0; j < SCAN_ITEMS; ++j) {
    const int i = j * SCAN_THREADS + threadIdx.x;
    sm.v[scan_slot(i)] = base + i < n ? (int64_t)in[base + i] : 0;
  }
}

__device__ __forceinline__ void scan_store(const ScanSmem& sm, int64_t* __restrict__ out, int64_t n,
                                           int64_t base, int64_t carry, int64_t total) {
#pragma unroll
  for (int j = 0; j < SCAN_ITEMS; ++j) {
    const int i = j * SCAN_THREADS + threadIdx.x;
    if (base + i < n) out[base + i] = carry + sm.v[scan_slot(i)];
  }
  if (threadIdx.x == 0 && n <= base + SCAN_TILE) out[n] = carry + total;
}

template <typename Tin>
__global__ void __launch_bounds__(SCAN_THREADS) k_scan_one(const Tin* __restrict__ in, int64_t n,
                                                           int64_t* __restrict__ out) {
  __shared__ ScanSmem sm;
  int64_t carry = 0;
  for (int64_t base = 0; base == 0 || base < n; base += SCAN_TILE) {
    __syncthreads();  // the previous tile is stored
    scan_load(sm, in, n, base);
    const int64_t total = scan_tile(sm);
    scan_store(sm, out, n, base, carry, total);
    carry += total;
  }
}

// state[0]: the tile counter; state[1 + t]: tile t's word (all zero at launch).
template <typename Tin>
__global__ void __launch_bounds__(SCAN_THREADS) k_scan_lookback(
    const Tin* __restrict__ in, int64_t n, unsigned long long* __restrict__ state,
    int64_t* __restrict__ out) {
  __shared__ ScanSmem sm;
  if (threadIdx.x == 0) sm.tile = (int64_t)atomicAdd(state, 1ull);
  __syncthreads();
  const int64_t tile = sm.tile, base = tile * SCAN_TILE;
  unsigned long long* word = state + 1;
  scan_load(sm, in, n, base);
  const int64_t total = scan_tile(sm);
  if (threadIdx.x < 32) {  // warp 0: 32 earlier tiles at a time
    const int lane = threadIdx.x;
    if (lane == 0)
      lb_store(word + tile, (tile == 0 ? LB_PREFIX : LB_SUM) | (unsigned long long)total);
    int64_t carry = 0;
    for (int64_t t = tile - 1 - lane; __any_sync(0xffffffffu, t >= 0); t -= 32) {
      unsigned long long v = t >= 0 ? lb_wait(word + t) : LB_PREFIX;
      if (v == 0ull) {  // not published in time: sum it here
        int64_t x = 0;
        for (int64_t g = t * SCAN_TILE; g < (t + 1) * SCAN_TILE; ++g) x += (int64_t)in[g];
        v = LB_SUM | (unsigned long long)x;
      }
      const uint32_t pre = __ballot_sync(0xffffffffu, (v & ~LB_VALUE) == LB_PREFIX);
      int64_t x = (pre == 0 || lane <= __ffs(pre) - 1) ? (int64_t)(v & LB_VALUE) : 0;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
      carry += x;
      if (pre) break;
    }
    if (lane == 0) {
      if (tile > 0) lb_store(word + tile, LB_PREFIX | (unsigned long long)(carry + total));
      sm.carry = carry;
    }
  }
  __syncthreads();
  scan_store(sm, out, n, base, sm.carry, total);
}

template <typename Tin>
void scan_impl(evoc_ctx* ctx, const Tin* in, int64_t* out, int64_t n) {
  cudaStream_t s = ctx->stream;
  if (n <= SCAN_ONE_BLOCK) {
    k_scan_one<Tin><<<1, SCAN_THREADS, 0, s>>>(in, n, out);
    EVOC_CHECK_LAUNCH();
    return;
  }
  const int64_t tiles = (n + SCAN_TILE - 1) / SCAN_TILE;
  DevBuf<unsigned long long> state(tiles + 1, s);
  EVOC_CUDA(cudaMemsetAsync(state.get(), 0, state.bytes(), s));
  k_scan_lookback<Tin><<<(unsigned)tiles, SCAN_THREADS, 0, s>>>(in, n, state.get(), out);
  EVOC_CHECK_LAUNCH();
}

// ---------------------------------------------------------------------------
// Radix sort: 8-bit digits, tiles of 4096 elements (256 threads x 16). One
// launch counts the digits of every pass, then one launch per pass: a warp
// ranks its own 512 consecutive elements (peers by __match_any_sync, counts in
// shared memory, no block barrier), the tile is put in digit order in shared
// memory, each digit's offset comes from the look-back, and each digit's run
// leaves contiguously. Bound by memory: 24 bytes per element and pass.
// ---------------------------------------------------------------------------
constexpr int RS_THREADS = 256;
constexpr int RS_ITEMS = 16;
constexpr int RS_TILE = RS_THREADS * RS_ITEMS;
constexpr int RS_WARPS = RS_THREADS / 32;
constexpr int RS_MAX_PASSES = 4;

__global__ void __launch_bounds__(RS_THREADS) k_radix_hist(const uint32_t* __restrict__ keys,
                                                           int64_t n, int passes,
                                                           unsigned long long* __restrict__ hist) {
  __shared__ int32_t h[RS_MAX_PASSES][256];
  for (int p = 0; p < passes; ++p) h[p][threadIdx.x] = 0;
  __syncthreads();
  for (int64_t g = (int64_t)blockIdx.x * RS_THREADS + threadIdx.x; g < n;
       g += (int64_t)gridDim.x * RS_THREADS) {
    const uint32_t k = keys[g];
    for (int p = 0; p < passes; ++p) atomicAdd(&h[p][(k >> (8 * p)) & 255u], 1);
  }
  __syncthreads();
  for (int p = 0; p < passes; ++p) {
    const int32_t c = h[p][threadIdx.x];
    if (c) atomicAdd(&hist[p * 256 + threadIdx.x], (unsigned long long)c);
  }
}

// Stable rank of each of the thread's RS_ITEMS elements among the earlier ones
// of its warp with the same digit; cnt (zeroed) gets the warp's digit counts.
__device__ __forceinline__ void radix_rank(const uint32_t (&key)[RS_ITEMS], int shift, int valid_n,
                                           int lane, int32_t* __restrict__ cnt,
                                           uint16_t (&rank)[RS_ITEMS]) {
  const unsigned FULL = 0xffffffffu;
  const uint32_t lt = (1u << lane) - 1u;
#pragma unroll
  for (int r = 0; r < RS_ITEMS; ++r) {
    const bool valid = r * 32 + lane < valid_n;
    const uint32_t d = valid ? (key[r] >> shift) & 255u : 256u;
    const uint32_t peers = __match_any_sync(FULL, d);
    const int before = valid ? cnt[d] : 0;
    __syncwarp();
    if (valid && (peers & lt) == 0) cnt[d] = before + __popc(peers);
    __syncwarp();
    rank[r] = (uint16_t)(before + __popc(peers & lt));
  }
}

struct RadixSmem {
  uint32_t keys[RS_TILE];
  uint2 vals[RS_TILE];
  int32_t warp_cnt[RS_WARPS][256];  // the warps' digit counts, then offsets
  int32_t tile_start[256];          // digit segment starts within the tile
  int64_t digit_base[256];          // the segments' global starts
  int64_t wide[RS_WARPS];
  int32_t narrow[RS_WARPS];
  int64_t tile;
};

// Exclusive prefix over the block's 256 threads.
template <typename T>
__device__ __forceinline__ T block_exclusive(T x, T* warp_tot) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  T incl = x;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const T y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  if (lane == 31) warp_tot[warp] = incl;
  __syncthreads();
  T before = 0;
  for (int w = 0; w < warp; ++w) before += warp_tot[w];
  __syncthreads();
  return before + incl - x;
}

// One pass. state[0]: the tile counter; state[1 + t * 256 + d]: tile t's word of
// digit d (all zero at launch); hist: the pass's digit totals.
__global__ void __launch_bounds__(RS_THREADS, 3) k_radix_pass(
    const uint32_t* __restrict__ keys_in, const uint2* __restrict__ vals_in, int64_t n, int shift,
    const unsigned long long* __restrict__ hist, unsigned long long* __restrict__ state,
    uint32_t* __restrict__ keys_out, uint2* __restrict__ vals_out) {
  extern __shared__ __align__(16) unsigned char rs_raw[];
  RadixSmem& sm = *reinterpret_cast<RadixSmem*>(rs_raw);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, dd = threadIdx.x;
  if (threadIdx.x == 0) sm.tile = (int64_t)atomicAdd(state, 1ull);
  for (int w = 0; w < RS_WARPS; ++w) sm.warp_cnt[w][dd] = 0;
  __syncthreads();
  const int64_t tile = sm.tile, base = tile * RS_TILE;
  const int tile_n = (int)min((int64_t)RS_TILE, n - base);
  const int w0 = warp * 32 * RS_ITEMS;  // the warp's first element
  uint32_t key[RS_ITEMS];
  uint16_t rank[RS_ITEMS];
#pragma unroll
  for (int r = 0; r < RS_ITEMS; ++r) {
    const int e = w0 + r * 32 + lane;
    key[r] = e < tile_n ? keys_in[base + e] : 0u;
  }
  radix_rank(key, shift, tile_n - w0, lane, sm.warp_cnt[warp], rank);
  __syncthreads();
  int32_t c = 0;  // digit dd: offsets of the warps, then the tile's count
#pragma unroll
  for (int w = 0; w < RS_WARPS; ++w) {
    const int32_t x = sm.warp_cnt[w][dd];
    sm.warp_cnt[w][dd] = c;
    c += x;
  }
  unsigned long long* word = state + 1 + dd;
  lb_store(word + tile * 256, (tile == 0 ? LB_PREFIX : LB_SUM) | (unsigned long long)c);
  sm.tile_start[dd] = block_exclusive(c, sm.narrow);
  const int64_t first = block_exclusive((int64_t)hist[dd], sm.wide);
  int64_t before = 0;
  for (int64_t t = tile - 1; t >= 0; --t) {
    unsigned long long v = lb_wait(word + t * 256);
    if (v == 0ull) {  // not published in time: count the digit here
      int32_t x = 0;
      for (int64_t g = t * RS_TILE; g < (t + 1) * RS_TILE; ++g)
        x += ((keys_in[g] >> shift) & 255u) == (uint32_t)dd;
      v = LB_SUM | (unsigned long long)x;
    }
    before += (int64_t)(v & LB_VALUE);
    if ((v & ~LB_VALUE) == LB_PREFIX) break;
  }
  if (tile > 0) lb_store(word + tile * 256, LB_PREFIX | (unsigned long long)(before + c));
  sm.digit_base[dd] = first + before;
  __syncthreads();
#pragma unroll
  for (int r = 0; r < RS_ITEMS; ++r) {
    const int e = w0 + r * 32 + lane;
    if (e < tile_n) {
      const uint32_t d = (key[r] >> shift) & 255u;
      const int pos = sm.tile_start[d] + sm.warp_cnt[warp][d] + rank[r];
      sm.keys[pos] = key[r];
      sm.vals[pos] = vals_in[base + e];
    }
  }
  __syncthreads();
#pragma unroll 4
  for (int e = threadIdx.x; e < tile_n; e += RS_THREADS) {
    const uint32_t k = sm.keys[e];
    const uint32_t d = (k >> shift) & 255u;
    const int64_t pos = sm.digit_base[d] + (e - sm.tile_start[d]);
    keys_out[pos] = k;
    vals_out[pos] = sm.vals[e];
  }
}

// At most RS_TILE elements: every pass in one block, in place. The passes move
// (key, index) in shared memory; the values follow once at the end.
__global__ void __launch_bounds__(RS_THREADS) k_radix_one(uint32_t* __restrict__ keys,
                                                          uint2* __restrict__ vals, int n,
                                                          int passes) {
  __shared__ uint32_t sk[RS_TILE];
  __shared__ uint16_t si[RS_TILE];
  __shared__ int32_t cnt[RS_WARPS][256];
  __shared__ int32_t start[256];
  __shared__ int32_t narrow[RS_WARPS];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, dd = threadIdx.x;
  const int w0 = warp * 32 * RS_ITEMS;
  for (int e = threadIdx.x; e < n; e += RS_THREADS) {
    sk[e] = keys[e];
    si[e] = (uint16_t)e;
  }
  for (int p = 0; p < passes; ++p) {
    for (int w = 0; w < RS_WARPS; ++w) cnt[w][dd] = 0;
    __syncthreads();
    uint32_t key[RS_ITEMS];
    uint16_t idx[RS_ITEMS], rank[RS_ITEMS];
#pragma unroll
    for (int r = 0; r < RS_ITEMS; ++r) {
      const int e = w0 + r * 32 + lane;
      key[r] = e < n ? sk[e] : 0u;
      idx[r] = e < n ? si[e] : (uint16_t)0;
    }
    radix_rank(key, 8 * p, n - w0, lane, cnt[warp], rank);
    __syncthreads();
    int32_t c = 0;
#pragma unroll
    for (int w = 0; w < RS_WARPS; ++w) {
      const int32_t x = cnt[w][dd];
      cnt[w][dd] = c;
      c += x;
    }
    start[dd] = block_exclusive(c, narrow);
    __syncthreads();
#pragma unroll
    for (int r = 0; r < RS_ITEMS; ++r) {
      if (w0 + r * 32 + lane < n) {
        const uint32_t d = (key[r] >> (8 * p)) & 255u;
        const int pos = start[d] + cnt[warp][d] + rank[r];
        sk[pos] = key[r];
        si[pos] = idx[r];
      }
    }
    __syncthreads();
  }
  uint2 v[RS_ITEMS];
#pragma unroll
  for (int r = 0; r < RS_ITEMS; ++r) {
    const int e = r * RS_THREADS + threadIdx.x;
    if (e < n) v[r] = vals[si[e]];
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < RS_ITEMS; ++r) {
    const int e = r * RS_THREADS + threadIdx.x;
    if (e < n) {
      keys[e] = sk[e];
      vals[e] = v[r];
    }
  }
}

}  // namespace

void exclusive_scan_i32_to_i64(evoc_ctx* ctx, const int32_t* in, int64_t* out, int64_t n) {
  scan_impl<int32_t>(ctx, in, out, n);
}

void exclusive_scan_i64(evoc_ctx* ctx, const int64_t* in, int64_t* out, int64_t n) {
  scan_impl<int64_t>(ctx, in, out, n);
}

void radix_sort_pairs(evoc_ctx* ctx, DevBuf<uint32_t>& keys, DevBuf<uint2>& vals, int64_t n,
                      int key_bits) {
  if (n <= 1 || key_bits <= 0) return;
  cudaStream_t s = ctx->stream;
  const int passes = (key_bits + 7) / 8;
  if (n <= RS_TILE) {
    k_radix_one<<<1, RS_THREADS, 0, s>>>(keys.get(), vals.get(), (int)n, passes);
    EVOC_CHECK_LAUNCH();
    return;
  }
  EVOC_CUDA(cudaFuncSetAttribute((const void*)k_radix_pass,  // the staged tile > 48 KB
                                 cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)sizeof(RadixSmem)));
  const int64_t tiles = (n + RS_TILE - 1) / RS_TILE;
  const int64_t per_pass = 1 + 256 * tiles;  // the counter and the tiles' words
  DevBuf<uint32_t> k2(keys.count, s);
  DevBuf<uint2> v2(vals.count, s);
  DevBuf<unsigned long long> work(passes * (256 + per_pass), s);
  EVOC_CUDA(cudaMemsetAsync(work.get(), 0, work.bytes(), s));
  unsigned long long* state = work.get() + passes * 256;
  const int64_t hgrid = std::min<int64_t>(tiles, 8 * (int64_t)ctx->num_sms);
  k_radix_hist<<<(unsigned)hgrid, RS_THREADS, 0, s>>>(keys.get(), n, passes, work.get());
  EVOC_CHECK_LAUNCH();
  for (int p = 0; p < passes; ++p) {
    k_radix_pass<<<(unsigned)tiles, RS_THREADS, sizeof(RadixSmem), s>>>(
        keys.get(), vals.get(), n, 8 * p, work.get() + p * 256, state + p * per_pass, k2.get(),
        v2.get());
    EVOC_CHECK_LAUNCH();
    std::swap(keys, k2);
    std::swap(vals, v2);
  }
}

}  // namespace evoc
