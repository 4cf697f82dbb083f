// row_groups.cuh — a CSR row's entries grouped by a label of their column, each
// group summed serially in row order (f32, one rounding per addition): the step
// that the label-propagation votes, the coarse graph and the expansion share.
//
// A warp takes a row of at most RG_MID entries: (label, position) keys are
// sorted in registers (bitonic, 1 to 32 keys per lane), runs of equal labels are
// found by ballot and a lane sums each run in position order from shared
// memory. Nothing leaves the SM, where a global stable radix sort of all
// entries moves 24 bytes per entry and digit. Rows above RG_CAP entries go
// through a list to a second launch with more shared memory per warp, so that
// the many short rows keep their occupancy. Rows above RG_MID take a block each:
// 1024 entries at a time are sorted the same way in shared memory, and each
// run's sum is continued in a dense table of one float per label, so a row may
// have any length and the additions keep its order.
#pragma once

#include "evoc_device.cuh"

namespace evoc {

constexpr int RG_CAP = 128;        // entries of a short row
constexpr int RG_MID = 1024;       // entries of a row that one warp still sorts
constexpr int RG_POS_BITS = 10;    // a key is label << RG_POS_BITS | position
constexpr uint32_t RG_POS = (1u << RG_POS_BITS) - 1u;
constexpr int RG_LABELS = 16384;   // labels are below this (the long rows' dense table)
constexpr int RG_WARPS = 8;        // warps per block of the short-row kernels
constexpr int RG_BLOCKS = 6;       // and their blocks per SM (the rows' load chains need warps)
constexpr int RG_NODE_WARPS = 12;  // warps per SM below which a warp takes fewer rows
constexpr int RG_MID_WARPS = 4;    // and of the middle-row kernels

template <int CAP>
struct RgWarp {
  uint32_t key[CAP];
  float val[CAP];   // by position
  float sum[CAP];   // by run
  uint16_t start[CAP];
};

// The rows left to a later launch: counts and row lists (n rows each).
struct RgLists {
  uint32_t* mid;
  uint32_t* longs;
  int32_t* count;  // [0] mid, [1] longs, [2] next of mid (zeroed)
};

// Files row i of len entries; false when it is short.
__device__ __forceinline__ bool rg_defer(const RgLists& l, int64_t i, int64_t len, int lane) {
  if (len <= RG_CAP) return false;
  if (lane == 0) {
    if (len <= RG_MID)
      l.mid[atomicAdd(l.count, 1)] = (uint32_t)i;
    else
      l.longs[atomicAdd(l.count + 1, 1)] = (uint32_t)i;
  }
  return true;
}

// The next row of the mid list for this warp, or -1.
__device__ __forceinline__ int64_t rg_next_mid(const RgLists& l, int lane) {
  int32_t at = 0;
  if (lane == 0) at = atomicAdd(l.count + 2, 1);
  at = __shfl_sync(0xffffffffu, at, 0);
  return at < l.count[0] ? (int64_t)l.mid[at] : -1;
}

// Ascending bitonic sort of 32 R keys, element lane * R + r in k[r].
template <int R>
__device__ __forceinline__ void rg_sort(uint32_t (&k)[R], int lane) {
#pragma unroll
  for (int size = 2; size <= 32 * R; size <<= 1) {
#pragma unroll
    for (int stride = size >> 1; stride >= 1; stride >>= 1) {
      if (stride >= R) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const uint32_t o = __shfl_xor_sync(0xffffffffu, k[r], stride / R);
          const int e = lane * R + r;
          const bool low = ((e & size) == 0) == ((e & stride) == 0);
          k[r] = low ? min(k[r], o) : max(k[r], o);
        }
      } else {
#pragma unroll
        for (int r = 0; r < R; ++r) {
          if ((r & stride) == 0) {
            const bool up = ((lane * R + r) & size) == 0;
            const uint32_t a = k[r], b = k[r | stride];
            k[r] = up ? min(a, b) : max(a, b);
            k[r | stride] = up ? max(a, b) : min(a, b);
          }
        }
      }
    }
  }
}

template <int R, int CAP>
__device__ __forceinline__ void rg_sort_smem(RgWarp<CAP>& sm, int m, int lane) {
  uint32_t k[R];
#pragma unroll
  for (int r = 0; r < R; ++r) k[r] = lane * R + r < m ? sm.key[lane * R + r] : 0xffffffffu;
  rg_sort<R>(k, lane);
  __syncwarp();
#pragma unroll
  for (int r = 0; r < R; ++r) sm.key[lane * R + r] = k[r];
}

// Groups the m <= CAP entries staged in sm.key (label << RG_POS_BITS | position)
// and sm.val (by position). Returns the run count; run r has label
// sm.key[sm.start[r]] >> RG_POS_BITS and sum sm.sum[r], labels ascending.
template <int CAP>
__device__ __forceinline__ int rg_group(RgWarp<CAP>& sm, int m, int lane) {
  const unsigned FULL = 0xffffffffu;
  __syncwarp();
  if constexpr (CAP <= RG_CAP) {
    if (m <= 32)
      rg_sort_smem<1>(sm, m, lane);
    else if (m <= 64)
      rg_sort_smem<2>(sm, m, lane);
    else
      rg_sort_smem<4>(sm, m, lane);
  } else {
    if (m <= 256)
      rg_sort_smem<8>(sm, m, lane);
    else if (m <= 512)
      rg_sort_smem<16>(sm, m, lane);
    else
      rg_sort_smem<32>(sm, m, lane);
  }
  __syncwarp();
  int runs = 0;
  for (int b = 0; b < m; b += 32) {
    const int e = b + lane;
    const bool head = e < m && (e == 0 || (sm.key[e] >> RG_POS_BITS) != (sm.key[e - 1] >> RG_POS_BITS));
    const uint32_t hb = __ballot_sync(FULL, head);
    if (head) sm.start[runs + __popc(hb & ((1u << lane) - 1u))] = (uint16_t)e;
    runs += __popc(hb);
  }
  __syncwarp();
  for (int r = lane; r < runs; r += 32) {
    const int a = sm.start[r], b = r + 1 < runs ? sm.start[r + 1] : m;
    float s = sm.val[sm.key[a] & RG_POS];
    for (int e = a + 1; e < b; ++e) s = fadd(s, sm.val[sm.key[e] & RG_POS]);
    sm.sum[r] = s;
  }
  __syncwarp();
  return runs;
}

// Long rows, one block of RG_LONG_THREADS per row.
constexpr int RG_LONG_ROW = 2048;  // a warp reads no row longer than this, however few entries count
constexpr int RG_LONG_THREADS = 256;
constexpr int RG_CHUNK = 1024;

struct RgLong {
  float acc[RG_LABELS];          // sums of the labels whose bit is set
  uint16_t list[RG_LABELS];      // present labels, ascending (rg_long_list)
  uint32_t bits[RG_LABELS / 32];
  uint32_t key[RG_CHUNK];
  float val[RG_CHUNK];
  int32_t warp_tot[RG_LONG_THREADS / 32];
};
// The votes also need the row position of each label's first entry.
struct RgLongVotes : RgLong {
  uint32_t first[RG_LABELS];
};

__device__ __forceinline__ void rg_long_clear(RgLong& sm) {
  __syncthreads();
  for (int q = threadIdx.x; q < RG_LABELS / 32; q += RG_LONG_THREADS) sm.bits[q] = 0u;
  __syncthreads();
}

// Adds the chunk staged in sm.key (label << 10 | position in the chunk, or all
// ones for none) and sm.val to the table. With `first`, the labels' first row
// positions are kept (pos0: the chunk's).
__device__ __forceinline__ void rg_long_chunk(RgLong& sm, uint32_t* first, uint32_t pos0) {
  for (int size = 2; size <= RG_CHUNK; size <<= 1)
    for (int stride = size >> 1; stride >= 1; stride >>= 1) {
      __syncthreads();
      for (int q = threadIdx.x; q < RG_CHUNK / 2; q += RG_LONG_THREADS) {
        const int i = 2 * q - (q & (stride - 1)), j = i + stride;
        const uint32_t a = sm.key[i], b = sm.key[j];
        if ((a > b) == ((i & size) == 0)) {
          sm.key[i] = b;
          sm.key[j] = a;
        }
      }
    }
  __syncthreads();
  for (int e = threadIdx.x; e < RG_CHUNK; e += RG_LONG_THREADS) {
    const uint32_t k = sm.key[e];
    if (k == 0xffffffffu) continue;
    const uint32_t l = k >> 10;
    if (e > 0 && (sm.key[e - 1] >> 10) == l) continue;
    const bool seen = (sm.bits[l >> 5] >> (l & 31u)) & 1u;
    float s = sm.val[k & (RG_CHUNK - 1)];
    if (seen)
      s = fadd(sm.acc[l], s);
    else if (first)
      first[l] = pos0 + (k & (RG_CHUNK - 1));
    for (int f = e + 1; f < RG_CHUNK && (sm.key[f] >> 10) == l; ++f)
      s = fadd(s, sm.val[sm.key[f] & (RG_CHUNK - 1)]);
    sm.acc[l] = s;
  }
  __syncthreads();
  for (int e = threadIdx.x; e < RG_CHUNK; e += RG_LONG_THREADS) {
    const uint32_t k = sm.key[e];
    if (k != 0xffffffffu) atomicOr(&sm.bits[k >> 15], 1u << ((k >> 10) & 31u));
  }
  __syncthreads();
}

// The present labels in ascending order into sm.list; returns their count.
__device__ __forceinline__ int rg_long_list(RgLong& sm) {
  const unsigned FULL = 0xffffffffu;
  constexpr int PER = RG_LABELS / 32 / RG_LONG_THREADS;  // bitmap words per thread
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  int c = 0;
#pragma unroll
  for (int q = 0; q < PER; ++q) c += __popc(sm.bits[threadIdx.x * PER + q]);
  int incl = c;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(FULL, incl, o);
    if (lane >= o) incl += y;
  }
  if (lane == 31) sm.warp_tot[wid] = incl;
  __syncthreads();
  int before = 0, total = 0;
  for (int w = 0; w < RG_LONG_THREADS / 32; ++w) {
    if (w < wid) before += sm.warp_tot[w];
    total += sm.warp_tot[w];
  }
  int at = before + incl - c;
#pragma unroll
  for (int q = 0; q < PER; ++q) {
    const int word = threadIdx.x * PER + q;
    for (uint32_t b = sm.bits[word]; b; b &= b - 1) sm.list[at++] = (uint16_t)(32 * word + __ffs(b) - 1);
  }
  __syncthreads();
  return total;
}

}  // namespace evoc
