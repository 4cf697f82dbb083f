// label_prop.cu — the partition step of the label-propagation initialisation
// (evoc-rs 0.2.7, src/graph/label_prop.rs:45-230) on the GPU.
//
//   seed      approx_n_parts random nodes get labels 0.. (a later draw of the
//             same node overwrites: label_prop.rs:216-219);
//   iterate   n_iter conservative rounds (label_prop.rs:45-92): an unlabelled
//             node sums its neighbours' weights per label in row order, and
//             adopts the label with the largest total if that total is at
//             least 1.0 (ties: the label that first appears last);
//   mop up    unlabelled nodes walk a LIFO stack of at most 64 pops for a
//             labelled node, else take a random existing label
//             (label_prop.rs:105-142); the reference's sequential order is
//             kept by resolving walks that meet earlier outliers afterwards;
//   remap     labels to 0..n_parts in sorted order, any -1 to new ids in
//             node order (label_prop.rs:155-180).
//
// The vote sums are the same f32 additions in the same order as the
// reference's loop, so labels match the CPU restatement exactly. Random draws
// come from Philox4x32-10 (counters below) instead of rand::SmallRng. With
// labels below RG_LABELS (every call of the initialisation) a row's votes are
// grouped on the SM (k_lp_iter_rows). With more labels each node keeps its vote
// table in its own CSR row range of a scratch array (a row has at most as many
// distinct labels as entries), so no node can overflow it; rows longer than 64
// also get a hash index (at most half full) in four entries per row of two more
// scratch arrays (k_lp_iter).
#include "evoc_internal.h"
#include "evoc_device.cuh"
#include "row_groups.cuh"

#include <algorithm>

namespace evoc {
namespace {

__device__ __forceinline__ uint32_t lp_seed_draw(uint64_t seed, uint32_t i, uint32_t n) {
  const uint4 o = philox4x32_10(make_uint4(i, 0u, 0x4C50u, 0x53454544u),
                                make_uint2((uint32_t)seed, (uint32_t)(seed >> 32)));
  return __umulhi(o.x, n);
}
__device__ __forceinline__ uint32_t lp_outlier_draw(uint64_t seed, uint64_t i, uint32_t range) {
  const uint4 o = philox4x32_10(make_uint4((uint32_t)i, (uint32_t)(i >> 32), 0x4C50u, 0x4F555431u),
                                make_uint2((uint32_t)seed, (uint32_t)(seed >> 32)));
  return __umulhi(o.x, range);
}

// Unlabelled nodes, and the length of the longest row (starts below 0).
__global__ void __launch_bounds__(256) k_lp_fill(int32_t* __restrict__ labels,
                                                 const int64_t* __restrict__ indptr, int64_t n,
                                                 int32_t* __restrict__ longest) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  int32_t len = 0;
  if (i < n) {
    labels[i] = -1;
    len = (int32_t)min(indptr[i + 1] - indptr[i], (int64_t)0x7fffffff);
  }
  len = __reduce_max_sync(0xffffffffu, len);
  if ((threadIdx.x & 31) == 0 && len > *(volatile int32_t*)longest) atomicMax(longest, len);
}

// Draw i labels node lp_seed_draw(i); the largest i drawn for a node is the
// last write of the reference's sequential loop.
__global__ void k_lp_seed(int32_t* __restrict__ labels, int64_t n, int64_t parts, uint64_t seed) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < parts) atomicMax(&labels[lp_seed_draw(seed, (uint32_t)i, (uint32_t)n)], (int32_t)i);
}

// One conservative iteration, thread per node.
// Rows up to this degree search their vote table linearly; longer rows (hubs)
// index it through a hash table, so a vote costs O(1) instead of O(distinct).
constexpr int64_t LP_LINEAR_DEG = 64;

__global__ void k_lp_iter(const int64_t* __restrict__ indptr, const uint32_t* __restrict__ indices,
                          const float* __restrict__ w, int64_t n, const int32_t* __restrict__ in,
                          int32_t* __restrict__ out, int32_t* __restrict__ vlab,
                          float* __restrict__ vsum, const int64_t* __restrict__ hoff,
                          int32_t* __restrict__ hkey, int32_t* __restrict__ hpos,
                          int32_t* __restrict__ changed) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int32_t cur = in[i];
  if (cur >= 0) {
    out[i] = cur;
    return;
  }
  const int64_t b = indptr[i], e = indptr[i + 1], deg = e - b;
  int64_t cnt = 0;  // distinct labelled labels, in first-appearance order
  if (deg <= LP_LINEAR_DEG) {
    for (int64_t q = b; q < e; ++q) {
      const int32_t l = in[indices[q]];
      if (l < 0) continue;  // unlabelled votes never win
      int64_t k = 0;
      while (k < cnt && vlab[b + k] != l) ++k;
      if (k < cnt) {
        vsum[b + k] = __fadd_rn(vsum[b + k], w[q]);
      } else {
        vlab[b + cnt] = l;
        vsum[b + cnt] = w[q];
        ++cnt;
      }
    }
  } else {
    // long row: an open-addressing table (label -> position in vlab/vsum) in
    // the row's own range [hoff[i], hoff[i + 1]) of hkey/hpos, at most half full
    const int64_t cap = hoff[i + 1] - hoff[i];
    int32_t* key = hkey + hoff[i];
    int32_t* hp = hpos + hoff[i];
    for (int64_t h = 0; h < cap; ++h) key[h] = -1;
    const int64_t mask = cap - 1;
    for (int64_t q = b; q < e; ++q) {
      const int32_t l = in[indices[q]];
      if (l < 0) continue;
      int64_t h = (int64_t)(((uint32_t)l * 2654435761u) & (uint32_t)mask);
      while (key[h] != -1 && key[h] != l) h = (h + 1) & mask;
      if (key[h] == l) {
        const int64_t k = hp[h];
        vsum[b + k] = __fadd_rn(vsum[b + k], w[q]);
      } else {
        key[h] = l;
        hp[h] = (int32_t)cnt;
        vlab[b + cnt] = l;
        vsum[b + cnt] = w[q];
        ++cnt;
      }
    }
  }
  int32_t best = -1;
  float max_vote = 1.0f;  // threshold
  for (int64_t k = 0; k < cnt; ++k) {
    const float v = vsum[b + k];
    if (v > max_vote) {
      max_vote = v;
      best = vlab[b + k];
    } else if (v == max_vote) {
      best = vlab[b + k];  // last encountered wins
    }
  }
  out[i] = best;
  if (best >= 0) *changed = 1;
}

// Hash-table slots of each row: the power of two >= 2 deg for rows longer
// than LP_LINEAR_DEG, none for the others (they search their votes linearly).
__global__ void k_lp_hcap(const int64_t* __restrict__ indptr, int64_t n,
                          int64_t* __restrict__ cap_out) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int64_t deg = indptr[i + 1] - indptr[i];
  int64_t cap = 0;
  if (deg > LP_LINEAR_DEG) {
    cap = 1;
    while (cap < 2 * deg) cap <<= 1;
  }
  cap_out[i] = cap;
}

// Marks the neighbours of newly labelled nodes for the round that comes next.
__device__ __forceinline__ void lp_mark_row(const uint32_t* __restrict__ indices, int64_t b,
                                            int64_t e, int first, int stride, uint8_t tag,
                                            uint8_t* __restrict__ mark) {
  for (int64_t q = b + first; q < e; q += stride) mark[indices[q]] = tag;
}

__global__ void k_lp_mark_seeds(const int64_t* __restrict__ indptr,
                                const uint32_t* __restrict__ indices, int64_t n, int64_t parts,
                                uint64_t seed, uint8_t* __restrict__ mark) {
  const int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (i >= parts) return;
  const uint32_t v = lp_seed_draw(seed, (uint32_t)i, (uint32_t)n);
  lp_mark_row(indices, indptr[v], indptr[v + 1], threadIdx.x & 31, 32, 0, mark);
}

// What the round before wrote. In an overlapped launch that one may still run when this
// one comes onto the SMs: then it is not read-only while this grid lives.
template <bool OVERLAP, typename T>
__device__ __forceinline__ T lp_read(const T* p) {
  if constexpr (OVERLAP)
    return load_l2(p);
  else
    return __ldg(p);
}

// One conservative iteration for labels below RG_LABELS, a warp per npw nodes:
// labelled nodes pass their label on, and each unlabelled node's row is read by
// the whole warp (coalesced, 32 label gathers in flight), its labelled entries
// are compacted and grouped on the SM (row_groups.cuh). The winner is the
// largest sum of at least 1.0, among equal sums the label whose first entry
// comes last, as in k_lp_iter. Rows with more than RG_CAP labelled or RG_LONG_ROW
// entries go to `longs`. A round after one that labelled nobody returns at once:
// both label arrays are equal then, so no round needs the host.
// With `mark` (symmetric graphs) only nodes with a neighbour labelled in the
// round before are looked at: the others' votes, and so their outcome, are the
// ones they had. A winner marks its neighbours with the next round's number in
// the other of two arrays, so no mark that this round still reads is overwritten.
// With OVERLAP the launch comes onto the SMs before the round before has ended, so
// everything that a round writes (labels, marks, flags, the list) is read by lp_read;
// the graph is constant.
template <bool OVERLAP>
__global__ void __launch_bounds__(32 * RG_WARPS, RG_BLOCKS) k_lp_iter_rows(
    const int64_t* __restrict__ indptr, const uint32_t* __restrict__ indices,
    const float* __restrict__ w, int64_t n, const int32_t* in, int32_t* __restrict__ out,
    const int32_t* prev_changed, int32_t* __restrict__ changed, uint32_t* __restrict__ longs,
    int32_t* __restrict__ n_long, int32_t round, const uint8_t* mark,
    uint8_t* __restrict__ next_mark, int npw) {
  __shared__ RgWarp<RG_CAP> sm_all[RG_WARPS];
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  // OVERLAP: launched while the round before ends (see the launch); the next may come likewise
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (prev_changed && lp_read<OVERLAP>(prev_changed) == 0) return;
  const int64_t v0 = ((int64_t)blockIdx.x * RG_WARPS + wid) * npw;
  if (v0 >= n) return;
  RgWarp<RG_CAP>& sm = sm_all[wid];
  const int64_t v = v0 + lane;
  const bool node = lane < npw && v < n;
  int32_t mine = node ? lp_read<OVERLAP>(in + v) : 0;
  const bool look = mine < 0 && (!mark || lp_read<OVERLAP>(mark + v) == (uint8_t)round);
  const int64_t pb = look ? indptr[v] : 0, pe = look ? indptr[v + 1] : 0;
  const uint32_t lt = (1u << lane) - 1u;
  bool won = false;
  for (uint32_t todo = __ballot_sync(FULL, look); todo; todo &= todo - 1) {
    const int src = __ffs(todo) - 1;
    const int64_t b = __shfl_sync(FULL, pb, src), e = __shfl_sync(FULL, pe, src);
    int m = 0;
    float votes = 0.0f;  // the lane's share of the row's votes
    bool fits = e - b <= RG_LONG_ROW;
    __syncwarp();  // the previous node's readers are done
    for (int64_t q0 = b; q0 < e && fits; q0 += 32) {
      const int64_t q = q0 + lane;
      const int32_t l = q < e ? lp_read<OVERLAP>(in + indices[q]) : -1;
      const uint32_t has = __ballot_sync(FULL, l >= 0);
      const int at = m + __popc(has & lt);
      m += __popc(has);
      fits = m <= RG_CAP;
      if (fits && l >= 0) {
        const float wq = w[q];
        sm.key[at] = ((uint32_t)l << RG_POS_BITS) | (uint32_t)at;
        sm.val[at] = wq;
        votes += fabsf(wq);
      }
    }
    if (!fits) {
      if (lane == 0) longs[atomicAdd(n_long, 1)] = (uint32_t)(v0 + src);
      continue;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) votes += __shfl_xor_sync(FULL, votes, o);
    // no label reaches 1.0 if all votes together, rounding included, do not
    if (votes < 0.999f) continue;
    const int runs = rg_group(sm, m, lane);
    float best = 1.0f;  // threshold
    int first = -1;     // position of the best label's first entry
    uint32_t lab = 0;
    for (int r = lane; r < runs; r += 32) {
      const uint32_t k = sm.key[sm.start[r]];
      const float s = sm.sum[r];
      const int pos = (int)(k & RG_POS);
      if (s > best || (s == best && pos > first)) {
        best = s;
        first = pos;
        lab = k >> RG_POS_BITS;
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float s = __shfl_xor_sync(FULL, best, o);
      const int p = __shfl_xor_sync(FULL, first, o);
      const uint32_t l = __shfl_xor_sync(FULL, lab, o);
      if (s > best || (s == best && p > first)) {
        best = s;
        first = p;
        lab = l;
      }
    }
    if (first >= 0) {
      if (lane == src) {
        mine = (int32_t)lab;
        won = true;
      }
      if (mark) lp_mark_row(indices, b, e, lane, 32, (uint8_t)(round + 1), next_mark);
    }
  }
  if (node) out[v] = mine;
  if (won) *changed = 1;
}

// The rows of `longs`, a block per row.
template <bool OVERLAP>
__global__ void __launch_bounds__(RG_LONG_THREADS) k_lp_iter_long(
    const int64_t* __restrict__ indptr, const uint32_t* __restrict__ indices,
    const float* __restrict__ w, const int32_t* in, int32_t* __restrict__ out,
    int32_t* __restrict__ changed, const uint32_t* longs, const int32_t* n_long, int32_t round,
    uint8_t* __restrict__ next_mark) {
  extern __shared__ __align__(16) unsigned char rg_raw[];
  RgLongVotes& sm = *reinterpret_cast<RgLongVotes*>(rg_raw);
  __shared__ int any;
  __shared__ float wb[RG_LONG_THREADS / 32];
  __shared__ uint32_t wf[RG_LONG_THREADS / 32], wl[RG_LONG_THREADS / 32];
  const unsigned FULL = 0xffffffffu;
  // OVERLAP: launched while the short rows' kernel ends, and the next round while this one does
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int nl = lp_read<OVERLAP>(n_long);
  for (int item = blockIdx.x; item < nl; item += gridDim.x) {
    const uint32_t i = lp_read<OVERLAP>(longs + item);
    const int64_t b = indptr[i], e = indptr[i + 1];
    rg_long_clear(sm);
    for (int64_t c = b; c < e; c += RG_CHUNK) {
      constexpr int PER = RG_CHUNK / RG_LONG_THREADS;
      int32_t l[PER];  // all on their way before the first is stored
#pragma unroll
      for (int k = 0; k < PER; ++k) {
        const int64_t q = c + k * RG_LONG_THREADS + threadIdx.x;
        l[k] = q < e ? lp_read<OVERLAP>(in + indices[q]) : -1;
      }
#pragma unroll
      for (int k = 0; k < PER; ++k) {
        const int q = k * RG_LONG_THREADS + threadIdx.x;
        sm.key[q] = l[k] >= 0 ? ((uint32_t)l[k] << 10) | (uint32_t)q : 0xffffffffu;
        sm.val[q] = l[k] >= 0 ? w[c + q] : 0.0f;
      }
      rg_long_chunk(sm, sm.first, (uint32_t)(c - b));
    }
    float best = 1.0f;  // threshold; first + 1 of the best label, 0 for none
    uint32_t first = 0, lab = 0;
    for (int l = threadIdx.x; l < RG_LABELS; l += RG_LONG_THREADS) {
      if (!((sm.bits[l >> 5] >> (l & 31)) & 1u)) continue;
      const float s = sm.acc[l];
      const uint32_t p = sm.first[l] + 1u;
      if (s > best || (s == best && p > first)) {
        best = s;
        first = p;
        lab = (uint32_t)l;
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float s = __shfl_xor_sync(FULL, best, o);
      const uint32_t p = __shfl_xor_sync(FULL, first, o), l = __shfl_xor_sync(FULL, lab, o);
      if (s > best || (s == best && p > first)) {
        best = s;
        first = p;
        lab = l;
      }
    }
    if ((threadIdx.x & 31) == 0) {
      wb[threadIdx.x >> 5] = best;
      wf[threadIdx.x >> 5] = first;
      wl[threadIdx.x >> 5] = lab;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      for (int q = 1; q < RG_LONG_THREADS / 32; ++q)
        if (wb[q] > best || (wb[q] == best && wf[q] > first)) {
          best = wb[q];
          first = wf[q];
          lab = wl[q];
        }
      any = first > 0;
      if (first > 0) {
        out[i] = (int32_t)lab;
        *changed = 1;
      }
    }
    __syncthreads();
    if (next_mark && any)
      lp_mark_row(indices, b, e, threadIdx.x, RG_LONG_THREADS, (uint8_t)(round + 1), next_mark);
  }
}

__global__ void k_lp_max(const int32_t* __restrict__ labels, int64_t n, int32_t* __restrict__ mx,
                         int32_t* __restrict__ unl) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int32_t l = labels[i];
  unl[i] = l < 0 ? 1 : 0;
  if (l >= 0) atomicMax(mx, l);
}

__global__ void k_lp_list(const int32_t* __restrict__ unl, const int64_t* __restrict__ pos,
                          int64_t n, uint32_t* __restrict__ list) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n && unl[i]) list[pos[i]] = (uint32_t)i;
}

// The mop-up (label_prop.rs:105-142) in parallel. In the reference's
// sequential order, outlier i's walk stops at the first node that is labelled
// by then: a node labelled before the mop-up, or an earlier outlier j < i
// (every processed outlier has a label). So each walk runs against the
// labels before the mop-up and yields a label, a pointer to an earlier
// outlier (-2 - its list index), or the fallback draw; k_lp_jump then
// resolves the pointers. A walk pops at most 64 nodes, so only the top 64
// stack entries can ever be popped: the stack is a 64-entry ring that drops
// its bottom entry when full.
// A warp per walk: it reads a popped node's row 32 entries at a time (one node's
// row can hold thousands), stops at the first entry that ends the walk, and
// pushes the others in row order.
constexpr int LP_WALK_WARPS = 8;
__global__ void __launch_bounds__(32 * LP_WALK_WARPS) k_lp_walk(
    const int64_t* __restrict__ indptr, const uint32_t* __restrict__ indices,
    const int32_t* __restrict__ labels, const int64_t* __restrict__ pos,
    const uint32_t* __restrict__ list, int64_t count, int32_t max_label, uint64_t seed,
    int32_t* __restrict__ res) {
  __shared__ uint32_t ring_all[LP_WALK_WARPS][64];
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int64_t u = (int64_t)blockIdx.x * LP_WALK_WARPS + wid;
  if (u >= count) return;
  uint32_t* ring = ring_all[wid];
  const uint32_t i = list[u];
  int64_t top = 1, bottom = 0;  // entries [bottom, top), slot = index % 64
  if (lane == 0) ring[0] = i;
  __syncwarp();
  for (int step = 0; step < 64 && top > bottom; ++step) {
    --top;
    const uint32_t node = ring[top & 63];
    __syncwarp();  // read before the slot is pushed over
    const int64_t b = indptr[node], e = indptr[node + 1];
    for (int64_t q0 = b; q0 < e; q0 += 32) {
      const int64_t q = q0 + lane;
      uint32_t j = 0;
      int32_t l = -1;
      if (q < e) {
        j = indices[q];
        l = labels[j];
      }
      // labelled, or an earlier outlier (unlabelled here): labelled by then
      const uint32_t hit = __ballot_sync(FULL, q < e && (l >= 0 || j < i));
      const int cnt = hit ? __ffs(hit) - 1 : (int)min((int64_t)32, e - q0);
      if (hit) {
        if (lane == cnt) res[u] = l >= 0 ? l : (int32_t)(-2 - pos[j]);
        return;
      }
      __syncwarp();  // a long row's earlier pushes to these slots come first
      if (lane < cnt) ring[(top + lane) & 63] = j;
      top += cnt;
      if (top - bottom > 64) bottom = top - 64;
    }
    __syncwarp();
  }
  if (lane == 0) res[u] = (int32_t)lp_outlier_draw(seed, i, (uint32_t)max_label + 1u);
}

// Pointer jumping over the walk results, up to LP_HOPS pointers a pass; pointers
// only go to earlier outliers, so the chains end. *changed: one is left.
constexpr int LP_HOPS = 64;
__global__ void k_lp_jump(int32_t* res, int64_t count, int32_t* __restrict__ changed) {
  const int64_t u = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (u >= count) return;
  int32_t r = res[u];
  if (r >= 0) return;
  // others' results are read as they are written: each is on the chain's way on
  for (int h = 0; h < LP_HOPS && r < 0; ++h)
    r = *(volatile const int32_t*)(res + (-2 - (int64_t)r));
  *(volatile int32_t*)(res + u) = r;
  if (r < 0) *changed = 1;
}

__global__ void k_lp_assign(const uint32_t* __restrict__ list, const int32_t* __restrict__ res,
                            int64_t count, int32_t* __restrict__ labels) {
  const int64_t u = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (u < count) labels[list[u]] = res[u];
}

__global__ void k_lp_present(const int32_t* __restrict__ labels, int64_t n,
                             int32_t* __restrict__ present, int32_t* __restrict__ neg) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int32_t l = labels[i];
  neg[i] = l < 0 ? 1 : 0;
  if (l >= 0) present[l] = 1;
}

__global__ void k_lp_remap(const int32_t* __restrict__ labels, int64_t n,
                           const int64_t* __restrict__ newid, int64_t n_unique,
                           const int64_t* __restrict__ negrank, uint32_t* __restrict__ part) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int32_t l = labels[i];
  part[i] = (uint32_t)(l >= 0 ? newid[l] : n_unique + negrank[i]);
}

inline unsigned grid_for(int64_t n, int t = 256) { return (unsigned)((n + t - 1) / t); }

// The rounds for labels of any size (k_lp_iter): thread per node, vote tables in
// global memory; one look at the host per round.
void lp_rounds_any_label(evoc_ctx* ctx, const evoc_graph* g, int32_t n_iter, DevBuf<int32_t>& la,
                         DevBuf<int32_t>& lb, int32_t* flag) {
  cudaStream_t s = ctx->stream;
  const int64_t n = g->n, nnz = g->nnz;
  DevBuf<int32_t> vlab(std::max<int64_t>(nnz, 1), s);
  DevBuf<float> vsum(std::max<int64_t>(nnz, 1), s);
  // hash tables only for the long rows, packed by a prefix sum of their sizes
  DevBuf<int64_t> hcap(n, s), hoff(n + 1, s);
  k_lp_hcap<<<grid_for(n), 256, 0, s>>>(g->indptr.get(), n, hcap.get());
  EVOC_CHECK_LAUNCH();
  exclusive_scan_i64(ctx, hcap.get(), hoff.get(), n);
  int64_t htot = 0;
  EVOC_CUDA(cudaMemcpyAsync(&htot, hoff.get() + n, sizeof(int64_t), cudaMemcpyDeviceToHost, s));
  EVOC_CUDA(cudaStreamSynchronize(s));
  hcap.release();
  DevBuf<int32_t> hkey(std::max<int64_t>(htot, 1), s), hpos(std::max<int64_t>(htot, 1), s);
  // a round that labels no node is a fixed point: the rest would leave the
  // labels unchanged and are skipped
  for (int32_t it = 0; it < n_iter; ++it) {
    EVOC_CUDA(cudaMemsetAsync(flag, 0, sizeof(int32_t), s));
    k_lp_iter<<<grid_for(n, 128), 128, 0, s>>>(g->indptr.get(), g->indices.get(),
                                               g->weights.get(), n, la.get(), lb.get(),
                                               vlab.get(), vsum.get(), hoff.get(), hkey.get(),
                                               hpos.get(), flag);
    EVOC_CHECK_LAUNCH();
    std::swap(la, lb);
    int32_t h = 0;
    EVOC_CUDA(cudaMemcpyAsync(&h, flag, sizeof(int32_t), cudaMemcpyDeviceToHost, s));
    EVOC_CUDA(cudaStreamSynchronize(s));
    if (!h) break;
  }
}

}  // namespace

int64_t label_prop_partition(evoc_ctx* ctx, const evoc_graph* g, int64_t approx_n_parts,
                             int32_t n_iter, uint64_t seed, uint32_t* d_partition) {
  cudaStream_t s = ctx->stream;
  const int64_t n = g->n, nnz = g->nnz;
  if (n == 0) return 0;
  if (approx_n_parts < 0 || approx_n_parts >= (1LL << 31))
    throw Error(EVOC_ERR_INVALID_ARGUMENT, "approx_n_parts outside [0, 2^31)");
  if (n_iter < 0) throw Error(EVOC_ERR_INVALID_ARGUMENT, "n_iter < 0");
  DevBuf<int32_t> la(n, s), lb(n, s), flag(std::max(n_iter, 1), s);
  DevBuf<int32_t> mx(2, s);  // largest label, longest row
  EVOC_CUDA(cudaMemsetAsync(mx.get(), 0xff, mx.bytes(), s));  // -1
  k_lp_fill<<<grid_for(n), 256, 0, s>>>(la.get(), g->indptr.get(), n, mx.get() + 1);
  if (approx_n_parts > 0)
    k_lp_seed<<<grid_for(approx_n_parts), 256, 0, s>>>(la.get(), n, approx_n_parts, seed);
  EVOC_CHECK_LAUNCH();
  if (approx_n_parts <= RG_LABELS) {
    int32_t longest = 0;  // read while the seeds' kernels run
    EVOC_CUDA(cudaMemcpyAsync(&longest, mx.get() + 1, sizeof(int32_t), cudaMemcpyDeviceToHost, s));
    // n_iter rounds without the host: a round sees from the one before whether
    // anything is left to do
    DevBuf<uint32_t> longs(n, s);
    DevBuf<int32_t> n_long(std::max(n_iter, 1), s);
    EVOC_CUDA(cudaMemsetAsync(flag.get(), 0, flag.bytes(), s));
    EVOC_CUDA(cudaMemsetAsync(n_long.get(), 0, n_long.bytes(), s));
    // rows of a symmetric graph list the nodes that see a new label; a round's
    // number has to fit a mark
    DevBuf<uint8_t> marks;
    const bool use_marks = g->canonical && n_iter < 255;
    if (use_marks) {
      marks.alloc(2 * n, s);
      EVOC_CUDA(cudaMemsetAsync(marks.get(), 0xff, marks.bytes(), s));
      if (approx_n_parts > 0) {
        k_lp_mark_seeds<<<grid_for(approx_n_parts * 32), 256, 0, s>>>(
            g->indptr.get(), g->indices.get(), n, approx_n_parts, seed, marks.get());
        EVOC_CHECK_LAUNCH();
      }
    }
    // A warp takes its nodes' rows one after the other, 1 us and more each: as many
    // as leave RG_NODE_WARPS warps per SM, down to one.
    int npw = 32;
    while (npw > 1 && n < (int64_t)npw * ctx->num_sms * RG_NODE_WARPS) npw /= 2;
    const unsigned grid = (unsigned)((n + npw * RG_WARPS - 1) / (npw * RG_WARPS));
    const unsigned lgrid = (unsigned)std::max<int64_t>(1, std::min<int64_t>(ctx->num_sms, nnz / RG_CAP));
    // Rounds overlap while one fits on the chip in one wave: their gaps are then a part of
    // them (20 rounds, k 15: 1,500 nodes 0.36 -> 0.25 ms, 57k 0.58 -> 0.49, 230k 0.88 -> 0.80).
    // With more waves the loads that an overlapped launch needs cost more than the gaps
    // (260k 1.00 -> 1.24, 500k 1.57 -> 2.37; 2M, k 30: 6.4 -> 9.1 ms).
    const bool overlap = grid <= (unsigned)(RG_BLOCKS * ctx->num_sms);
    auto* rows = overlap ? k_lp_iter_rows<true> : k_lp_iter_rows<false>;
    auto* hubs = overlap ? k_lp_iter_long<true> : k_lp_iter_long<false>;
    EVOC_CUDA(cudaFuncSetAttribute((const void*)hubs, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)sizeof(RgLongVotes)));
    EVOC_CUDA(cudaStreamSynchronize(s));
    for (int32_t it = 0; it < n_iter; ++it) {
      uint8_t* mark = use_marks ? marks.get() + (it & 1) * n : nullptr;
      uint8_t* next = use_marks ? marks.get() + (1 - (it & 1)) * n : nullptr;
      // An overlapped round is brought onto the SMs while the one before still runs and
      // waits there for its end (and for all that came before: the first has no such leave).
      cudaLaunchAttribute attr;
      attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
      attr.val.programmaticStreamSerializationAllowed = 1;
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(grid);
      cfg.blockDim = dim3(32 * RG_WARPS);
      cfg.stream = s;
      cfg.attrs = &attr;
      cfg.numAttrs = overlap && it > 0 ? 1 : 0;
      EVOC_CUDA(cudaLaunchKernelEx(
          &cfg, rows, (const int64_t*)g->indptr.get(),
          (const uint32_t*)g->indices.get(), (const float*)g->weights.get(), n,
          (const int32_t*)la.get(), lb.get(),
          (const int32_t*)(it > 0 ? flag.get() + it - 1 : nullptr), flag.get() + it, longs.get(),
          n_long.get() + it, it, (const uint8_t*)mark, next, npw));
      if (longest > RG_CAP) {  // else no row can be left over
        cfg.gridDim = dim3(lgrid);
        cfg.blockDim = dim3(RG_LONG_THREADS);
        cfg.dynamicSmemBytes = sizeof(RgLongVotes);
        cfg.numAttrs = overlap ? 1 : 0;
        EVOC_CUDA(cudaLaunchKernelEx(
            &cfg, hubs, (const int64_t*)g->indptr.get(),
            (const uint32_t*)g->indices.get(), (const float*)g->weights.get(),
            (const int32_t*)la.get(), lb.get(), flag.get() + it, (const uint32_t*)longs.get(),
            (const int32_t*)(n_long.get() + it), it, next));
      }
      std::swap(la, lb);
    }
  } else {
    lp_rounds_any_label(ctx, g, n_iter, la, lb, flag.get());
  }
  // mop-up of the nodes still unlabelled, in node order
  DevBuf<int32_t> unl(n, s);
  DevBuf<int64_t> pos(n + 1, s);
  k_lp_max<<<grid_for(n), 256, 0, s>>>(la.get(), n, mx.get(), unl.get());
  EVOC_CHECK_LAUNCH();
  exclusive_scan_i32_to_i64(ctx, unl.get(), pos.get(), n);
  int64_t count = 0;
  EVOC_CUDA(cudaMemcpyAsync(&count, pos.get() + n, sizeof(int64_t), cudaMemcpyDeviceToHost, s));
  int32_t max_label = -1;
  EVOC_CUDA(cudaMemcpyAsync(&max_label, mx.get(), sizeof(int32_t), cudaMemcpyDeviceToHost, s));
  EVOC_CUDA(cudaStreamSynchronize(s));
  if (count > 0 && max_label >= 0) {
    DevBuf<uint32_t> list(count, s);
    DevBuf<int32_t> res(count, s);
    k_lp_list<<<grid_for(n), 256, 0, s>>>(unl.get(), pos.get(), n, list.get());
    k_lp_walk<<<grid_for(count, LP_WALK_WARPS), 32 * LP_WALK_WARPS, 0, s>>>(
        g->indptr.get(), g->indices.get(), la.get(), pos.get(), list.get(), count, max_label,
        seed + 2000, res.get());
    EVOC_CHECK_LAUNCH();
    for (int pass = 0; pass < 64; ++pass) {  // chains shrink at least by half per pass
      EVOC_CUDA(cudaMemsetAsync(flag.get(), 0, sizeof(int32_t), s));
      k_lp_jump<<<grid_for(count), 256, 0, s>>>(res.get(), count, flag.get());
      EVOC_CHECK_LAUNCH();
      int32_t h = 0;
      EVOC_CUDA(cudaMemcpyAsync(&h, flag.get(), sizeof(int32_t), cudaMemcpyDeviceToHost, s));
      EVOC_CUDA(cudaStreamSynchronize(s));
      if (!h) break;
    }
    k_lp_assign<<<grid_for(count), 256, 0, s>>>(list.get(), res.get(), count, la.get());
    EVOC_CHECK_LAUNCH();
  }
  // remap: labels are below approx_n_parts, or -1 if nothing was labelled
  const int64_t np = std::max<int64_t>(approx_n_parts, 1);
  DevBuf<int32_t> present(np, s), neg(n, s);
  DevBuf<int64_t> newid(np + 1, s), negrank(n + 1, s);
  EVOC_CUDA(cudaMemsetAsync(present.get(), 0, np * sizeof(int32_t), s));
  k_lp_present<<<grid_for(n), 256, 0, s>>>(la.get(), n, present.get(), neg.get());
  EVOC_CHECK_LAUNCH();
  exclusive_scan_i32_to_i64(ctx, present.get(), newid.get(), np);
  exclusive_scan_i32_to_i64(ctx, neg.get(), negrank.get(), n);
  int64_t n_unique = 0, n_neg = 0;
  EVOC_CUDA(cudaMemcpyAsync(&n_unique, newid.get() + np, sizeof(int64_t), cudaMemcpyDeviceToHost, s));
  EVOC_CUDA(cudaMemcpyAsync(&n_neg, negrank.get() + n, sizeof(int64_t), cudaMemcpyDeviceToHost, s));
  EVOC_CUDA(cudaStreamSynchronize(s));
  k_lp_remap<<<grid_for(n), 256, 0, s>>>(la.get(), n, newid.get(), n_unique, negrank.get(),
                                         d_partition);
  EVOC_CHECK_LAUNCH();
  return n_unique + n_neg;
}

}  // namespace evoc
