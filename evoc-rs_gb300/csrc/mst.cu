// mst.cu — build_mst (src/clustering/mst.rs:82-166, evoc-rs 0.2.7) on the
// GPU: Boruvka's minimum spanning tree over mutual reachability distance, the
// first step of the clustering stage that turns the embedding into labels.
//
// Spatial index. An implicit complete binary tree over leaves of 32 points
// (heap order: node v has children 2v and 2v + 1, leaves are P..2P-1), each node's
// points split along the widest side of their bounding box: the points of every
// node are ordered by that coordinate and the first half of the node's leaves
// takes the first ones. Nodes above KD_BLOCK points are ordered by one radix sort
// per level over (node, coordinate), the levels below by a block per node in
// shared memory. Against Morton order (whose 8 bits per dimension cut clusters at
// fixed planes) the boxes are tighter and a search meets far fewer of them.
// It plays the part of the reference's KD-tree (kd_tree.rs:93-236): only
// pruning bounds come from it, never a result.
//
// Core distances (mst.rs:101-113): per point, the k-th smallest squared
// distance to another point, k = min(min_samples, n - 1); a warp walks the
// tree for 32 consecutive points at once (see the traversal kernels), nearer
// child first, and skips a node whose box lower bound exceeds every lane's
// current k-th distance (knn_recurse, kd_tree.rs:489-535).
//
// Boruvka rounds (mst.rs:115-160):
//   1. what each node holds of the components, bottom-up (k_mst_leaf_parts; the
//      reference's update_node_components, kd_tree.rs:387-419, marks pure nodes);
//   2. per point, the nearest point of another component under squared mutual
//      reachability max(d^2, core_i, core_j) (nearest_other_component,
//      kd_tree.rs:275-378), with the same three pruning rules; among equal
//      values the smallest point index. A point whose nearest foreign point is
//      known from an earlier round or from the kNN lists is not searched for
//      again (k_mst_near_init); late rounds search for the points of a leaf together
//      (k_mst_noc_group). A per-component bound starts each other
//      query just above it and is lowered while the round runs: first the
//      smallest known value leaving the component (k_mst_bound), then the best
//      value found so far by its points.
//      Each is the value of a real edge leaving the component, so no
//      component's pick changes;
//   3. per component (its id is its smallest point index), the pick with the
//      smallest value, then the smallest point index: one 64-bit atomicMin of
//      (value bits, point index);
//   4. merge. The reference adds the picks one at a time through a disjoint
//      set and skips those that would close a cycle. Taken in ascending
//      component id, the skipped picks are exactly, on each cycle of the pick
//      graph (component -> component of its pick's other end), the pick of the
//      largest component id: the rest of a functional graph's weak component
//      hangs off its cycle in trees. Pointer doubling (2^K >= m steps) lands
//      every component on its cycle and gathers the cycle's maximum; pointer
//      jumping to the skipped component gives the merged components; kept
//      edges are appended in ascending component id.
// Squared distances are serial left folds over the dimensions with IEEE
// round-to-nearest operations and weights are square roots of them, so the
// edge list equals the oracle's edge for edge, weights bit for bit.
#include "evoc_device.cuh"
#include "evoc_internal.h"

#include <cfloat>
#include <cstring>

namespace evoc {
namespace {

constexpr int MST_LEAF = 32;     // points per leaf
constexpr uint32_t NO_POINT = 0xffffffffu;
constexpr uint32_t FMAX_BITS = 0x7f7fffffu;  // FLT_MAX

inline unsigned grid_of(int64_t n, int t = 256) { return (unsigned)((n + t - 1) / t); }

// Order-preserving integer image of a float (for min / max atomics).
__device__ __forceinline__ uint32_t ord_of(float f) {
  const uint32_t u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float of_ord(uint32_t u) {
  return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u);
}

// Every coordinate must be finite.
__global__ void k_mst_finite(const float* __restrict__ x, int64_t count,
                             int32_t* __restrict__ status) {
  bool bad = false;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < count;
       i += (int64_t)gridDim.x * blockDim.x)
    bad |= !isfinite(x[i]);
  if (bad) set_status(status, ST_BAD_VALUE);
}

__global__ void k_mst_iota_pairs(uint2* __restrict__ val, int64_t n) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) val[i] = make_uint2((uint32_t)i, 0u);
}

// Bounding boxes of the nodes of `size` consecutive points (size a multiple of
// 32 KD_RUN): a warp reduces KD_RUN runs of 32 points, then one atomic per side.
constexpr int KD_RUN = 32;
__global__ void k_kd_box(const float* __restrict__ x, int64_t n, int dim, int64_t size,
                         const uint2* __restrict__ val, uint32_t* __restrict__ bmin,
                         uint32_t* __restrict__ bmax) {
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int64_t p0 = (((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * (32 * KD_RUN);
  if (p0 >= n) return;
  const int64_t node = p0 / size;
  for (int d = 0; d < dim; ++d) {
    uint32_t lo = 0xffffffffu, hi = 0u;
#pragma unroll 8
    for (int r = 0; r < KD_RUN; ++r) {
      const int64_t pos = p0 + 32 * r + lane;
      if (pos < n) {
        const uint32_t o = ord_of(x[(int64_t)val[pos].x * dim + d]);
        lo = min(lo, o);
        hi = max(hi, o);
      }
    }
    lo = __reduce_min_sync(FULL, lo);
    hi = __reduce_max_sync(FULL, hi);
    if (lane == 0) {
      atomicMin(&bmin[node * dim + d], lo);
      atomicMax(&bmax[node * dim + d], hi);
    }
  }
}

// Widest side of a box.
__device__ __forceinline__ int kd_side(const uint32_t* bmin, const uint32_t* bmax, int dim) {
  int side = 0;
  float wide = -1.0f;
  for (int d = 0; d < dim; ++d) {
    const float w = of_ord(bmax[d]) - of_ord(bmin[d]);
    if (w > wide) {
      wide = w;
      side = d;
    }
  }
  return side;
}

// Sort key of a level: node, then the coordinate along the node's widest side
// on `bits` bits of its extent.
__global__ void k_kd_key(const float* __restrict__ x, int64_t n, int dim, int64_t size, int bits,
                         const uint2* __restrict__ val, const uint32_t* __restrict__ bmin,
                         const uint32_t* __restrict__ bmax, uint32_t* __restrict__ key) {
  const int64_t pos = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (pos >= n) return;
  const int64_t node = pos / size;
  const int side = kd_side(bmin + node * dim, bmax + node * dim, dim);
  const float lo = of_ord(bmin[node * dim + side]), hi = of_ord(bmax[node * dim + side]);
  const float maxq = (float)((1u << bits) - 1u), span = hi - lo;
  const float t = span > 0.0f ? (x[(int64_t)val[pos].x * dim + side] - lo) / span * maxq : 0.0f;
  key[pos] = ((uint32_t)node << bits) | (uint32_t)fminf(fmaxf(t, 0.0f), maxq);
}

// All levels of the nodes of at most KD_BLOCK points, a block per such node: per
// level the boxes of the nodes inside, then a bitonic sort of (coordinate, slot)
// within each of them. Bound by shared memory; the coordinates come from L2.
constexpr int KD_BLOCK = 4096;
constexpr int KD_THREADS = 512;
struct KdSmem {
  unsigned long long key[KD_BLOCK];  // coordinate image << 32 | slot
  uint32_t id[KD_BLOCK];             // point of each slot
  uint32_t bmin[KD_BLOCK / 64][16], bmax[KD_BLOCK / 64][16];
  uint8_t side[KD_BLOCK / 64];
};
__global__ void __launch_bounds__(KD_THREADS) k_kd_block(const float* __restrict__ x, int64_t n,
                                                         int dim, int top,
                                                         uint2* __restrict__ val) {
  extern __shared__ __align__(16) unsigned char kd_raw[];
  KdSmem& sm = *reinterpret_cast<KdSmem*>(kd_raw);
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t base = (int64_t)blockIdx.x * top;
  const int cnt = (int)min((int64_t)top, n - base);
  for (int e = threadIdx.x; e < top; e += KD_THREADS) {
    sm.id[e] = e < cnt ? val[base + e].x : 0u;
    sm.key[e] = (unsigned long long)e;  // slots past the end stay behind (all-ones coordinate)
  }
  for (int size = top; size >= 2 * MST_LEAF; size >>= 1) {
    const int nodes = top / size;
    for (int q = threadIdx.x; q < nodes * dim; q += KD_THREADS) {
      sm.bmin[q / dim][q % dim] = 0xffffffffu;
      sm.bmax[q / dim][q % dim] = 0u;
    }
    __syncthreads();
    for (int c = warp; c < top / 32; c += KD_THREADS / 32) {
      const int slot = (int)(uint32_t)sm.key[32 * c + lane];
      const bool on = slot < cnt;
      const float* p = x + (int64_t)sm.id[slot] * dim;
      for (int d = 0; d < dim; ++d) {
        const uint32_t o = on ? ord_of(p[d]) : 0u;
        const uint32_t lo = __reduce_min_sync(FULL, on ? o : 0xffffffffu);
        const uint32_t hi = __reduce_max_sync(FULL, o);
        if (lane == 0) {
          atomicMin(&sm.bmin[32 * c / size][d], lo);
          atomicMax(&sm.bmax[32 * c / size][d], hi);
        }
      }
    }
    __syncthreads();
    if (threadIdx.x < nodes)
      sm.side[threadIdx.x] = (uint8_t)kd_side(sm.bmin[threadIdx.x], sm.bmax[threadIdx.x], dim);
    __syncthreads();
    for (int e = threadIdx.x; e < top; e += KD_THREADS) {
      const uint32_t slot = (uint32_t)sm.key[e];
      const uint32_t o = (int)slot < cnt
                             ? ord_of(x[(int64_t)sm.id[slot] * dim + sm.side[e / size]])
                             : 0xffffffffu;
      sm.key[e] = ((unsigned long long)o << 32) | slot;
    }
    for (int run = 2; run <= size; run <<= 1)
      for (int stride = run >> 1; stride >= 1; stride >>= 1) {
        __syncthreads();
        for (int q = threadIdx.x; q < top / 2; q += KD_THREADS) {
          const int i = 2 * q - (q & (stride - 1)), j = i + stride;
          const unsigned long long a = sm.key[i], b = sm.key[j];
          const bool up = run == size || (i & run) == 0;  // every node ascends
          if ((a > b) == up) {
            sm.key[i] = b;
            sm.key[j] = a;
          }
        }
      }
    __syncthreads();
  }
  __syncthreads();
  for (int e = threadIdx.x; e < cnt; e += KD_THREADS)
    val[base + e].x = sm.id[(uint32_t)sm.key[e]];
}

// Sorted copy of the points, padded with zeros to DIMP (a zero pad adds +0 to
// a squared distance, which leaves it unchanged).
template <int DIMP>
__global__ void k_mst_gather(const float* __restrict__ x, int64_t n, int dim,
                             const uint2* __restrict__ val, float* __restrict__ xs,
                             uint32_t* __restrict__ orig, uint32_t* __restrict__ pos_of) {
  const int64_t pos = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (pos >= n) return;
  const uint32_t p = val[pos].x;
  orig[pos] = p;
  pos_of[p] = (uint32_t)pos;
#pragma unroll
  for (int d = 0; d < DIMP; ++d) xs[pos * DIMP + d] = d < dim ? x[(int64_t)p * dim + d] : 0.0f;
}

template <int DIMP>
__device__ __forceinline__ void mst_load(const float* __restrict__ xs, int64_t pos,
                                         float (&p)[DIMP]) {
  const float4* s = reinterpret_cast<const float4*>(xs + pos * DIMP);
#pragma unroll
  for (int q = 0; q < DIMP / 4; ++q) {
    const float4 v = __ldg(s + q);
    p[4 * q] = v.x;
    p[4 * q + 1] = v.y;
    p[4 * q + 2] = v.z;
    p[4 * q + 3] = v.w;
  }
}

// sum_d (a_d - b_d)^2, serial over the dimensions (mst.rs's squared metric); the
// differences and squares are packed pairs (the same roundings).
template <int DIMP>
__device__ __forceinline__ float mst_sqd(const float (&a)[DIMP], const float (&b)[DIMP]) {
  float s = 0.0f;
#pragma unroll
  for (int d = 0; d < DIMP; d += 2) {
    const float2 t = fsub2(make_float2(a[d], a[d + 1]), make_float2(b[d], b[d + 1]));
    const float2 t2 = fmul2(t, t);
    s = fadd(fadd(s, t2.x), t2.y);
  }
  return s;
}

// Squared distance from p to node v's box (aabb_sq, kd_tree.rs:247-265). It
// never exceeds the squared distance to a point inside the box: every step is
// a monotone rounded operation on a smaller operand.
template <int DIMP>
__device__ __forceinline__ float mst_box_lb(const float* __restrict__ lo,
                                            const float* __restrict__ hi, int64_t v,
                                            const float (&p)[DIMP]) {
  const float4* l4 = reinterpret_cast<const float4*>(lo + v * DIMP);
  const float4* h4 = reinterpret_cast<const float4*>(hi + v * DIMP);
  float r = 0.0f;
#pragma unroll
  for (int q = 0; q < DIMP / 4; ++q) {
    const float4 a = __ldg(l4 + q), b = __ldg(h4 + q);
    const float2 p0 = make_float2(p[4 * q], p[4 * q + 1]), p1 = make_float2(p[4 * q + 2], p[4 * q + 3]);
    const float2 l0 = fsub2(make_float2(a.x, a.y), p0), l1 = fsub2(make_float2(a.z, a.w), p1);
    const float2 h0 = fsub2(p0, make_float2(b.x, b.y)), h1 = fsub2(p1, make_float2(b.z, b.w));
    const float2 d0 = make_float2(fmaxf(fmaxf(l0.x, h0.x), 0.0f), fmaxf(fmaxf(l0.y, h0.y), 0.0f));
    const float2 d1 = make_float2(fmaxf(fmaxf(l1.x, h1.x), 0.0f), fmaxf(fmaxf(l1.y, h1.y), 0.0f));
    const float2 s0 = fmul2(d0, d0), s1 = fmul2(d1, d1);
    r = fadd(fadd(fadd(fadd(r, s0.x), s0.y), s1.x), s1.y);
  }
  return r;
}

// Leaf boxes (empty leaves: +inf / -inf, so every bound to them is +inf).
template <int DIMP>
__global__ void k_mst_leaf_boxes(const float* __restrict__ xs, int64_t n, int64_t P, int64_t L,
                                 float* __restrict__ lo, float* __restrict__ hi) {
  const int64_t l = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (l >= P) return;
  float a[DIMP], b[DIMP];
#pragma unroll
  for (int d = 0; d < DIMP; ++d) {
    a[d] = __int_as_float(0x7f800000);
    b[d] = -__int_as_float(0x7f800000);
  }
  if (l < L) {
    const int64_t e = min(n, (l + 1) * MST_LEAF);
    for (int64_t j = l * MST_LEAF; j < e; ++j) {
      float y[DIMP];
      mst_load<DIMP>(xs, j, y);
#pragma unroll
      for (int d = 0; d < DIMP; ++d) {
        a[d] = fminf(a[d], y[d]);
        b[d] = fmaxf(b[d], y[d]);
      }
    }
  }
  float4* lo4 = reinterpret_cast<float4*>(lo + (P + l) * DIMP);
  float4* hi4 = reinterpret_cast<float4*>(hi + (P + l) * DIMP);
#pragma unroll
  for (int q = 0; q < DIMP / 4; ++q) {
    lo4[q] = make_float4(a[4 * q], a[4 * q + 1], a[4 * q + 2], a[4 * q + 3]);
    hi4[q] = make_float4(b[4 * q], b[4 * q + 1], b[4 * q + 2], b[4 * q + 3]);
  }
}

// Internal boxes, up to eight levels per launch: a block takes 256 nodes of the
// level that starts at `first` (of count = first nodes) and goes up while it has
// two nodes left.
constexpr int UP_NODES = 256;
template <int DIMP>
__global__ void __launch_bounds__(UP_NODES / 2) k_mst_boxes_up(float* __restrict__ lo,
                                                             float* __restrict__ hi,
                                                             int64_t first) {
  constexpr int Q = DIMP / 4;
  float4* lo4 = reinterpret_cast<float4*>(lo);
  float4* hi4 = reinterpret_cast<float4*>(hi);
  const int64_t n0 = first + (int64_t)blockIdx.x * UP_NODES;
  int64_t base = n0 >> 1;
  for (int cnt = (int)min((int64_t)UP_NODES, first) >> 1; cnt >= 1; cnt >>= 1, base >>= 1) {
    if ((int)threadIdx.x < cnt) {
      const int64_t v = base + threadIdx.x;
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        const float4 a = lo4[2 * v * Q + q], b = lo4[(2 * v + 1) * Q + q];
        const float4 c = hi4[2 * v * Q + q], e = hi4[(2 * v + 1) * Q + q];
        lo4[v * Q + q] = make_float4(fminf(a.x, b.x), fminf(a.y, b.y), fminf(a.z, b.z), fminf(a.w, b.w));
        hi4[v * Q + q] = make_float4(fmaxf(c.x, e.x), fmaxf(c.y, e.y), fmaxf(c.z, e.z), fmaxf(c.w, e.w));
      }
    }
    __syncthreads();  // the level is written (the block reads only its own nodes)
  }
}

// Searches. A warp serves one point and walks the tree 32 nodes at a time: the
// descendants five levels below a node are consecutive in heap order, so each
// lane tests one of them, the nearest that can still matter is entered first, and
// a leaf's 32 points are measured by one lane each. The earlier form, 32 points
// per warp walking the union of their searches in lockstep, kept 7 of 32 lanes
// busy in a leaf and left single warps with thousands of serial steps (1M points,
// 8-d blobs, the same tree: core distances 26.8 ms against 7.3 here, and 8 to 13 ms
// in each early round for one straggling warp against 0.8 to 1.1). The instruction
// count bounds it (0.88 issued a cycle and scheduler, 400k points): about 20 leaves
// and 10 groups per point, and 12 blocks per SM (40 registers) gain only a tenth over 8.
constexpr int MST_WARPS = 4;   // warps per block
template <int DIMP>
constexpr int mst_blocks() { return DIMP <= 8 ? 12 : 8; }  // blocks per SM (registers)
constexpr int MST_LEVELS = 6;  // of five binary levels: 2^28 leaves at most
constexpr uint32_t INF_BITS = 0x7f800000u;

template <int DIMP>
struct MstTree {
  const float* xs;
  const float* lo;
  const float* hi;
  int64_t n, P;
  int depth;  // binary levels: P = 2^depth leaves
};

// Position of a walk: the group of nodes in hand, each lane holding the bound of
// its node (INF: done, pruned or none). The groups above wait in shared memory.
struct MstWalk {
  int64_t base;  // first node of the group
  int level;     // depth of the group's nodes
  int up;        // groups waiting above
  float p;       // this lane's bound
};

__device__ __forceinline__ int mst_first_bits(int depth) {
  return depth == 0 ? 0 : (depth - 1) % 5 + 1;
}

// The next node whose bound does not exceed `limit`, nearest first, or -1 when
// the group is done.
__device__ __forceinline__ int64_t mst_next(MstWalk& w, float limit, int lane) {
  const unsigned FULL = 0xffffffffu;
  const uint32_t m = __reduce_min_sync(FULL, __float_as_uint(w.p));
  if (m == INF_BITS || __uint_as_float(m) > limit) return -1;
  const int sel = __ffs(__ballot_sync(FULL, __float_as_uint(w.p) == m)) - 1;
  if (lane == sel) w.p = __uint_as_float(INF_BITS);
  return w.base + sel;
}

// Back to the waiting group above; false at the top.
__device__ __forceinline__ bool mst_ascend(MstWalk& w, const float (*stack)[32], int first_bits,
                                           int lane) {
  if (w.up == 0) return false;
  --w.up;
  w.p = stack[w.up][lane];
  w.base = w.up == 0 ? (int64_t)1 << first_bits : (w.base >> 5) & ~(int64_t)31;
  w.level -= 5;
  return true;
}

__device__ __forceinline__ void mst_descend(MstWalk& w, float (*stack)[32], int64_t node, int lane) {
  stack[w.up][lane] = w.p;
  ++w.up;
  w.base = node << 5;
  w.level += 5;
}

// Ascending bitonic sort of (d, j) across the warp.
__device__ __forceinline__ void mst_sort32(float& d, uint32_t& j, int lane) {
#pragma unroll
  for (int size = 2; size <= 32; size <<= 1)
#pragma unroll
    for (int stride = size >> 1; stride >= 1; stride >>= 1) {
      const float od = __shfl_xor_sync(0xffffffffu, d, stride);
      const uint32_t oj = __shfl_xor_sync(0xffffffffu, j, stride);
      const bool low = ((lane & size) == 0) == ((lane & stride) == 0);
      const bool take = low ? (od < d || (od == d && oj < j)) : (od > d || (od == d && oj > j));
      if (take) {
        d = od;
        j = oj;
      }
    }
}

// Core distances: per sorted point, the k-th smallest squared distance to
// another point; a node is skipped when its box bound exceeds the current k-th
// distance (kd_tree.rs:499). The k smallest are kept sorted across the lanes
// (entry t in lane t, with WIDE entries 32.. in a second register), started
// from the point's own leaf.
template <int DIMP, bool WIDE>
__global__ void __launch_bounds__(32 * MST_WARPS, mst_blocks<DIMP>()) k_mst_core(
    MstTree<DIMP> tree, int k, unsigned long long* __restrict__ work, float* __restrict__ core,
    uint32_t* __restrict__ knn_j, float* __restrict__ knn_d, uint8_t* __restrict__ tie_out) {
  __shared__ float stack_s[MST_WARPS][MST_LEVELS][32];
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  float (*stack)[32] = stack_s[wid];
  const float INF = __uint_as_float(INF_BITS);
  const int g0 = mst_first_bits(tree.depth);
  for (;;) {
    int64_t pos = 0;
    if (lane == 0) pos = (int64_t)atomicAdd(work, 1ull);
    pos = __shfl_sync(FULL, pos, 0);
    if (pos >= tree.n) return;
    float q[DIMP];
    mst_load<DIMP>(tree.xs, pos, q);
    float kd0 = INF, kd1 = INF;
    uint32_t kj0 = NO_POINT, kj1 = NO_POINT;
    const int64_t own = pos / MST_LEAF;
    {
      const int64_t j = own * MST_LEAF + lane;
      if (j < tree.n && j != pos) {
        float y[DIMP];
        mst_load<DIMP>(tree.xs, j, y);
        kd0 = mst_sqd<DIMP>(q, y);
        if (kd0 < INF) kj0 = (uint32_t)j;
      }
      mst_sort32(kd0, kj0, lane);
    }
    const bool high = WIDE && k > 32;  // the k-th entry is in the second register
    float kth = __shfl_sync(FULL, high ? kd1 : kd0, (k - 1) & 31);
    // a point outside the first k is exactly kth away
    bool tie = !high && __any_sync(FULL, lane >= k && kd0 == kth);
    MstWalk w{(int64_t)1 << g0, g0, 0, INF};
    if (tree.depth > 0 && lane < (1 << g0)) w.p = mst_box_lb<DIMP>(tree.lo, tree.hi, w.base + lane, q);
    for (;;) {
      if (w.level == tree.depth && w.base + lane == tree.P + own) w.p = INF;  // its own leaf is in
      const int64_t node = mst_next(w, kth, lane);
      if (node < 0) {
        if (!mst_ascend(w, stack, g0, lane)) break;
        continue;
      }
      if (w.level < tree.depth) {
        mst_descend(w, stack, node, lane);
        w.p = mst_box_lb<DIMP>(tree.lo, tree.hi, w.base + lane, q);
        continue;
      }
      const int64_t j = (node - tree.P) * MST_LEAF + lane;
      float d = INF;
      if (j < tree.n) {
        float y[DIMP];
        mst_load<DIMP>(tree.xs, j, y);
        d = mst_sqd<DIMP>(q, y);
      }
      for (uint32_t in; (in = __ballot_sync(FULL, d < kth)) != 0u;) {
        const int src = __ffs(in) - 1;
        const float dv = __shfl_sync(FULL, d, src);
        const uint32_t jv = (uint32_t)(j - lane + src);
        if (lane == src) d = INF;
        const int at = __popc(__ballot_sync(FULL, kd0 <= dv));  // after equal entries
        const float ud = __shfl_up_sync(FULL, kd0, 1);
        const uint32_t uj = __shfl_up_sync(FULL, kj0, 1);
        if (WIDE) {
          const int at1 = 32 + __popc(__ballot_sync(FULL, kd1 <= dv)), slot = at < 32 ? at : at1;
          const float ld = __shfl_sync(FULL, kd0, 31);
          const uint32_t lj = __shfl_sync(FULL, kj0, 31);
          const float vd = __shfl_up_sync(FULL, kd1, 1);
          const uint32_t vj = __shfl_up_sync(FULL, kj1, 1);
          if (lane + 32 == slot) {
            kd1 = dv;
            kj1 = jv;
          } else if (lane + 32 > slot) {
            kd1 = lane == 0 ? ld : vd;
            kj1 = lane == 0 ? lj : vj;
          }
        }
        if (lane == at) {
          kd0 = dv;
          kj0 = jv;
        } else if (lane > at) {
          kd0 = ud;
          kj0 = uj;
        }
        const float was = kth;
        kth = __shfl_sync(FULL, high ? kd1 : kd0, (k - 1) & 31);
        tie = was == kth;  // the entry pushed out was at the distance that stays
      }
      tie = tie || __any_sync(FULL, d == kth && j < tree.n);
    }
    if (lane < k) {
      knn_j[pos * k + lane] = kj0;
      knn_d[pos * k + lane] = kd0;
    }
    if (WIDE && lane + 32 < k) {
      knn_j[pos * k + lane + 32] = kj1;
      knn_d[pos * k + lane + 32] = kd1;
    }
    if (lane == 0) {
      core[pos] = kth;
      tie_out[pos] = tie ? 1 : 0;
    }
  }
}

// What a point knows of its nearest point of another component carries over
// between rounds, because components only grow: near_j is that point (or
// NO_POINT) and near_v its value, or, without a point, a value below which there
// is none. A point whose near_j is still foreign needs no search, and neither
// does one whose near_v is not below its component's bound.
//
// First round, from the kNN lists: every value is at least the point's own core
// distance, and the points at exactly that value are those within it whose own
// core distance is no larger, that is entries of its list (unless a point outside
// the list ties with the last one). The smallest index among them is the answer.
__global__ void k_mst_near_init(int64_t n, int k, const uint32_t* __restrict__ knn_j,
                                const uint8_t* __restrict__ tie, const float* __restrict__ core,
                                const uint32_t* __restrict__ orig, uint32_t* __restrict__ near_j,
                                float* __restrict__ near_v) {
  const int64_t pos = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (pos >= n) return;
  const float cq = core[pos];
  uint32_t best = NO_POINT, bo = NO_POINT;
  if (k > 0 && cq < __uint_as_float(FMAX_BITS) && !tie[pos]) {
    for (int t = 0; t < k; ++t) {
      const uint32_t j = knn_j[pos * k + t];
      if (j >= n || core[j] > cq) continue;  // unfilled, or a larger value
      const uint32_t oj = orig[j];
      if (oj < bo) {
        bo = oj;
        best = j;
      }
    }
  }
  near_j[pos] = best;
  near_v[pos] = cq;
}

// Upper bounds before a round's queries: per component, the smallest value of its
// points' nearest foreign points where those are known, of the kNN edges
// (from the core-distance pass) that leave it, and of the neighbours in tree order
// that do (a component of a whole cluster often has no other). Each is the value of a real edge
// leaving the component, so it is never below the component's pick and starting
// the queries just above it changes no pick.
template <int DIMP>
__global__ void k_mst_bound(const float* __restrict__ xs, int64_t n, int k,
                            const uint32_t* __restrict__ knn_j,
                            const float* __restrict__ knn_d, const uint32_t* __restrict__ comp,
                            const float* __restrict__ core, uint32_t* __restrict__ near_j,
                            const float* __restrict__ near_v, uint32_t* __restrict__ cbest) {
  const int64_t pos = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (pos >= n) return;
  const uint32_t qc = comp[pos], nj = near_j[pos];
  if (pos + 1 < n && comp[pos + 1] != qc) {
    const uint32_t oc = comp[pos + 1];
    float a[DIMP], b[DIMP];
    mst_load<DIMP>(xs, pos, a);
    mst_load<DIMP>(xs, pos + 1, b);
    const float mr = fmaxf(fmaxf(mst_sqd<DIMP>(a, b), core[pos]), core[pos + 1]);
    const uint32_t v = __float_as_uint(mr);
    if (v < __ldcg(cbest + qc)) atomicMin(cbest + qc, v);
    if (v < __ldcg(cbest + oc)) atomicMin(cbest + oc, v);
  }
  if (nj != NO_POINT) {
    if (comp[nj] != qc) {
      const uint32_t v = __float_as_uint(near_v[pos]);
      if (v < __ldcg(cbest + qc)) atomicMin(cbest + qc, v);
      return;  // its nearest: no kNN edge of it leaves with less
    }
    near_j[pos] = NO_POINT;
  }
  const float cq = core[pos];
  float best = __uint_as_float(FMAX_BITS);
  for (int t = 0; t < k; ++t) {
    const uint32_t j = knn_j[pos * k + t];
    if (j >= n || comp[j] == qc) continue;  // an unfilled entry (no finite distance)
    best = fminf(best, fmaxf(fmaxf(knn_d[pos * k + t], cq), core[j]));
  }
  const uint32_t v = __float_as_uint(best);
  if (v < __ldcg(cbest + qc)) atomicMin(cbest + qc, v);
}

// Known nearest points enter their component's pick; need[pos] = 1 for the
// points that have to search. With `groups`, the searching points of one component
// in `width` consecutive places are put up for a common search
// (k_mst_noc_group) when they are at least half of them: (leaf, lanes) is appended.
__global__ void k_mst_select(int64_t n, const uint32_t* __restrict__ comp,
                             const float* __restrict__ core, const uint32_t* __restrict__ orig,
                             const uint32_t* __restrict__ near_j, const float* __restrict__ near_v,
                             const uint32_t* __restrict__ cbest,
                             unsigned long long* __restrict__ ckey, int32_t* __restrict__ need,
                             uint2* __restrict__ groups, unsigned long long* __restrict__ n_groups,
                             int width) {
  const unsigned FULL = 0xffffffffu;
  const int64_t pos = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const bool on = pos < n;
  uint32_t qc = NO_POINT;
  bool search = false;
  if (on) {
    qc = comp[pos];
    const uint32_t cb = cbest[qc];
    const float v = near_v[pos];
    if (near_j[pos] != NO_POINT) {
      const uint32_t vb = __float_as_uint(v);
      if (vb <= cb) atomicMin(ckey + qc, ((unsigned long long)vb << 32) | orig[pos]);
    } else {
      const float bd = __uint_as_float(cb < FMAX_BITS ? cb + 1u : FMAX_BITS);
      search = v < bd && !(core[pos] > bd);
    }
  }
  if (groups && __popc(__ballot_sync(FULL, search)) >= width / 2) {  // the same in the warp
    const uint32_t peers = __match_any_sync(FULL, search ? qc : NO_POINT);
    const int same = search ? __popc(peers) : 0;
    const int most = __reduce_max_sync(FULL, same);
    const uint32_t c = __reduce_min_sync(FULL, search && same == most ? qc : NO_POINT);
    if (most >= width / 2) {
      const uint32_t lanes = __ballot_sync(FULL, search && qc == c);
      const int lane = threadIdx.x & 31;
      for (int at = 0; at < 32; at += width) {
        const uint32_t some = lanes & (0xffffffffu >> (32 - width) << at);
        if (__popc(some) >= width / 2 && lane == 0)
          groups[atomicAdd(n_groups, 1ull)] = make_uint2((uint32_t)(pos / MST_LEAF), some);
      }
    }
  }
  if (on) need[pos] = search ? 1 : 0;
}

// Takes the groups' points off the others' list, unless there are fewer groups than
// warps to serve them: a group's search is the longer one, and then sets the
// round's time (1M points, the round of 1,465 components: 1.21 ms with, 0.79 without).
__global__ void k_mst_take_groups(const uint2* __restrict__ groups,
                                  const unsigned long long* __restrict__ n_groups,
                                  unsigned long long min_groups, int32_t* __restrict__ need) {
  const unsigned long long ng = *n_groups;
  const unsigned long long g = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (ng < min_groups || g >= ng) return;
  const uint2 group = groups[g];
  for (uint32_t m = group.y; m; m &= m - 1)
    need[(int64_t)group.x * MST_LEAF + __ffs(m) - 1] = 0;
}

__global__ void k_mst_search_list(int64_t n, const int32_t* __restrict__ need,
                                  const int64_t* __restrict__ off, uint32_t* __restrict__ list) {
  const int64_t pos = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (pos < n && need[pos]) list[off[pos]] = (uint32_t)pos;
}

// What a round's queries see of a node: a component `maj` that many of its points
// belong to, the box of its other points, and the smallest core distance of all
// (core_all) and of the other points (core_rest). A query of that component is
// bounded by the other points' box and core (infinite for a node wholly of one
// component), any other query by the full box and core_all. Otherwise a few stray
// points next to a cluster keep the cluster's own points in every leaf that holds
// one of them, although their large core distances rule them out (1M points: the
// last three rounds 51.7 ms with pure-node marks only, 29.7 with this, walked by points).
template <int DIMP>
struct MstParts {
  uint32_t* maj;
  int32_t* cnt;
  float* lo;
  float* hi;
  float* core_all;
  float* core_rest;
};

// Leaves: a warp per leaf; the most frequent component (the smallest id among
// equals). No point belongs to NO_POINT, the majority of an empty leaf.
template <int DIMP>
__global__ void k_mst_leaf_parts(MstTree<DIMP> tree, const uint32_t* __restrict__ comp,
                                 const float* __restrict__ core, MstParts<DIMP> parts) {
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int64_t l = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (l >= tree.P) return;
  const int64_t j = l * MST_LEAF + lane;
  const bool on = j < tree.n;
  const uint32_t c = on ? comp[j] : NO_POINT;
  const uint32_t peers = __match_any_sync(FULL, c);  // every lane takes part
  const int same = on ? __popc(peers) : 0;
  const int most = __reduce_max_sync(FULL, same);
  const uint32_t m = __reduce_min_sync(FULL, on && same == most ? c : NO_POINT);
  const bool other = on && c != m;
  float y[DIMP];
  if (other) mst_load<DIMP>(tree.xs, j, y);
  const bool any = __any_sync(FULL, other);
  float* vl = parts.lo + (tree.P + l) * DIMP;
  float* vh = parts.hi + (tree.P + l) * DIMP;
  const uint32_t cb = on ? __float_as_uint(core[j]) : INF_BITS;  // not negative: bits order them
  const uint32_t c_all = __reduce_min_sync(FULL, cb);
  const uint32_t c_rest = __reduce_min_sync(FULL, other ? cb : INF_BITS);
#pragma unroll
  for (int d = 0; d < DIMP; ++d) {
    float a = __uint_as_float(INF_BITS), b = -a;
    if (any) {
      const uint32_t o = other ? ord_of(y[d]) : 0u;
      const uint32_t mn = __reduce_min_sync(FULL, other ? o : 0xffffffffu);
      const uint32_t mx = __reduce_max_sync(FULL, o);
      a = of_ord(mn);
      b = of_ord(mx);
    }
    if (lane == 0) {
      vl[d] = a;
      vh[d] = b;
    }
  }
  if (lane == 0) {
    parts.maj[tree.P + l] = m;
    parts.cnt[tree.P + l] = most;
    parts.core_all[tree.P + l] = __uint_as_float(c_all);
    parts.core_rest[tree.P + l] = __uint_as_float(c_rest);
  }
}

// Inner nodes, up to eight levels per launch (as k_mst_boxes_up): the majority
// of the child whose majority is larger, and the union of what the children hold
// besides it.
template <int DIMP>
__global__ void __launch_bounds__(UP_NODES / 2) k_mst_parts_up(MstTree<DIMP> tree,
                                                             MstParts<DIMP> parts, int64_t first) {
  constexpr int Q = DIMP / 4;
  float4* lo4 = reinterpret_cast<float4*>(parts.lo);
  float4* hi4 = reinterpret_cast<float4*>(parts.hi);
  const float4* fl4 = reinterpret_cast<const float4*>(tree.lo);
  const float4* fh4 = reinterpret_cast<const float4*>(tree.hi);
  int64_t base = (first + (int64_t)blockIdx.x * UP_NODES) >> 1;
  for (int c = (int)min((int64_t)UP_NODES, first) >> 1; c >= 1; c >>= 1, base >>= 1) {
    if ((int)threadIdx.x < c) {
      const int64_t v = base + threadIdx.x, l = 2 * v, r = 2 * v + 1;
      const uint32_t ml = parts.maj[l], mr = parts.maj[r];
      const int32_t cl = parts.cnt[l], cr = parts.cnt[r];
      const uint32_t m = cl >= cr ? ml : mr;
      parts.maj[v] = m;
      parts.cnt[v] = ml == mr ? cl + cr : max(cl, cr);
      parts.core_all[v] = fminf(parts.core_all[l], parts.core_all[r]);
      parts.core_rest[v] = fminf(ml == m ? parts.core_rest[l] : parts.core_all[l],
                                 mr == m ? parts.core_rest[r] : parts.core_all[r]);
      const float4* la = (ml == m ? lo4 : fl4) + l * Q;
      const float4* ha = (ml == m ? hi4 : fh4) + l * Q;
      const float4* lb = (mr == m ? lo4 : fl4) + r * Q;
      const float4* hb = (mr == m ? hi4 : fh4) + r * Q;
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        const float4 a = la[q], b = lb[q], e = ha[q], f = hb[q];
        lo4[v * Q + q] = make_float4(fminf(a.x, b.x), fminf(a.y, b.y), fminf(a.z, b.z), fminf(a.w, b.w));
        hi4[v * Q + q] = make_float4(fmaxf(e.x, f.x), fmaxf(e.y, f.y), fmaxf(e.z, f.z), fmaxf(e.w, f.w));
      }
    }
    __syncthreads();
  }
}

__global__ void k_mst_round_reset(const uint32_t* __restrict__ A, int64_t m,
                                  uint32_t* __restrict__ cbest,
                                  unsigned long long* __restrict__ ckey) {
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= m) return;
  const uint32_t c = A[k];
  cbest[c] = FMAX_BITS;
  ckey[c] = ~0ull;
}

// Nearest point of another component under squared mutual reachability
// (kd_tree.rs:318-378), for the listed points: a node is kept when the bound of
// its foreign points and the point's own core distance do not exceed the best
// value so far. After each leaf the bound is
// lowered to just above the component's best value so far this round; a pick
// above that bound is dropped (it cannot be the component's pick).
template <int DIMP>
__global__ void __launch_bounds__(32 * MST_WARPS, mst_blocks<DIMP>()) k_mst_noc(
    MstTree<DIMP> tree, MstParts<DIMP> parts, const uint32_t* __restrict__ comp,
    const float* __restrict__ core, const uint32_t* __restrict__ orig,
    const uint32_t* __restrict__ list, const int64_t* __restrict__ n_list,
    unsigned long long* __restrict__ work, uint32_t* __restrict__ cbest,
    unsigned long long* __restrict__ ckey, uint32_t* __restrict__ near_j,
    float* __restrict__ near_v) {
  __shared__ float stack_s[MST_WARPS][MST_LEVELS][32];
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  float (*stack)[32] = stack_s[wid];
  const float INF = __uint_as_float(INF_BITS);
  const int g0 = mst_first_bits(tree.depth);
  const int64_t items = *n_list;
  for (;;) {
    int64_t item = 0;
    if (lane == 0) item = (int64_t)atomicAdd(work, 1ull);
    item = __shfl_sync(FULL, item, 0);
    if (item >= items) return;
    const int64_t pos = list[item];
    const uint32_t qc = comp[pos];
    const float cq = core[pos];
    float q[DIMP];
    mst_load<DIMP>(tree.xs, pos, q);
    float bd = __uint_as_float(FMAX_BITS);
    uint32_t bj = NO_POINT, bo = 0;
    auto refresh = [&]() {  // the component's best so far, found by other warps
      // one lane reads it (it changes meanwhile) and tells the others: the warp's
      // path through the tree has to be one
      const uint32_t cb = __shfl_sync(FULL, lane == 0 ? __ldcg(cbest + qc) : 0u, 0);
      const float nb = __uint_as_float(cb < FMAX_BITS ? cb + 1u : FMAX_BITS);
      if (nb < bd) {
        bd = nb;
        bj = NO_POINT;
      }
    };
    refresh();
    auto bound = [&](int64_t v) {
      const bool own = parts.maj[v] == qc;
      const float c = own ? parts.core_rest[v] : parts.core_all[v];
      return fmaxf(mst_box_lb<DIMP>(own ? parts.lo : tree.lo, own ? parts.hi : tree.hi, v, q), c);
    };
    MstWalk w{(int64_t)1 << g0, g0, 0, INF};
    if (lane < (1 << g0)) w.p = bound(w.base + lane);
    while (!(cq > bd)) {
      const int64_t node = mst_next(w, bd, lane);
      if (node < 0) {
        if (!mst_ascend(w, stack, g0, lane)) break;
        continue;
      }
      if (w.level < tree.depth) {
        mst_descend(w, stack, node, lane);
        w.p = bound(w.base + lane);
        continue;
      }
      const int64_t j = (node - tree.P) * MST_LEAF + lane;
      float mr = INF;
      if (j < tree.n && comp[j] != qc) {
        const float cj = core[j];
        if (!(cj > bd)) {
          float y[DIMP];
          mst_load<DIMP>(tree.xs, j, y);
          mr = fmaxf(fmaxf(mst_sqd<DIMP>(q, y), cq), cj);
        }
      }
      const uint32_t mb = __float_as_uint(mr), best = __reduce_min_sync(FULL, mb);
      if (best < __float_as_uint(bd) || (best == __float_as_uint(bd) && bj != NO_POINT)) {
        const uint32_t oj = mb == best ? orig[j] : NO_POINT;
        const uint32_t o = __reduce_min_sync(FULL, oj);
        if (best < __float_as_uint(bd) || o < bo) {
          const int src = __ffs(__ballot_sync(FULL, mb == best && oj == o)) - 1;
          if (lane == 0 && best < __float_as_uint(bd)) atomicMin(cbest + qc, best);
          bd = __uint_as_float(best);
          bo = o;
          bj = (uint32_t)(j - lane + src);
        }
      }
      refresh();
    }
    if (lane == 0) {
      near_j[pos] = bj;
      near_v[pos] = fmaxf(near_v[pos], bd);  // the value found, or nothing below the last bound
      if (bj != NO_POINT) {
        const uint32_t db = __float_as_uint(bd);
        atomicMin(ckey + qc, ((unsigned long long)db << 32) | orig[pos]);
      }
    }
  }
}

// The same for the searching points of one component in one leaf, a warp per
// group: late rounds have most points search again up to their component's bound
// and find nothing (1M points: 60 node groups and 63 leaves per point in the round
// of 24 components, 34 of 727,000 points have a find), and neighbours walk the same
// nodes. The walk tests nodes against the box of the group's points, so a node is
// met once for all of them; at a leaf each lane tests its own point against the
// leaf's box, and the leaf's foreign points (one per lane) are measured against
// each point that it may still matter to. Bound by instructions (0.70 issued a cycle and
// scheduler with 27 warps an SM, 400k points), about 35 for a point and leaf and 100 for
// a node group, as the walk by points. The last four rounds 26.7 -> 9.5 ms (the test of the points before a group of nodes is entered: 24.6 ->
// 22.5 of the whole tree, in the middle rounds, whose groups' boxes are loose).
constexpr int MST_GROUP_BLOCKS = 8;  // per SM (registers)
template <int DIMP>
__global__ void __launch_bounds__(32 * MST_WARPS, MST_GROUP_BLOCKS) k_mst_noc_group(
    MstTree<DIMP> tree, MstParts<DIMP> parts, const uint32_t* __restrict__ comp,
    const float* __restrict__ core, const uint32_t* __restrict__ orig,
    const uint2* __restrict__ groups, const unsigned long long* __restrict__ n_groups,
    unsigned long long min_groups, unsigned long long* __restrict__ work,
    uint32_t* __restrict__ cbest,
    unsigned long long* __restrict__ ckey, uint32_t* __restrict__ near_j,
    float* __restrict__ near_v) {
  constexpr int Q = DIMP / 4;
  __shared__ float stack_s[MST_WARPS][MST_LEVELS][32];
  __shared__ float4 q_s[MST_WARPS][32][Q];
  __shared__ float4 box_s[MST_WARPS][2][Q];  // of the group's points
  __shared__ float cq_s[MST_WARPS][32];
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  float (*stack)[32] = stack_s[wid];
  const float INF = __uint_as_float(INF_BITS);
  const int g0 = mst_first_bits(tree.depth);
  const unsigned long long items = *n_groups;
  if (items < min_groups) return;  // their points are on the others' list
  for (;;) {
    unsigned long long item = 0;
    if (lane == 0) item = atomicAdd(work, 1ull);
    item = __shfl_sync(FULL, item, 0);
    if (item >= items) return;
    const uint2 group = groups[item];
    const int64_t pos = (int64_t)group.x * MST_LEAF + lane;
    const bool active = (group.y >> lane) & 1u;
    const uint32_t qc = comp[(int64_t)group.x * MST_LEAF + __ffs(group.y) - 1];
    float q[DIMP];
    float cq = INF;
#pragma unroll
    for (int d = 0; d < DIMP; ++d) q[d] = 0.0f;
    if (active) {
      mst_load<DIMP>(tree.xs, pos, q);
      cq = core[pos];
    }
    const float cmin = __uint_as_float(__reduce_min_sync(FULL, __float_as_uint(cq)));
    float blo[DIMP], bhi[DIMP];
#pragma unroll
    for (int d = 0; d < DIMP; ++d) {
      const uint32_t o = ord_of(q[d]);
      blo[d] = of_ord(__reduce_min_sync(FULL, active ? o : 0xffffffffu));
      bhi[d] = of_ord(__reduce_max_sync(FULL, active ? o : 0u));
    }
    __syncwarp();  // the group before is done with the shared copies
    cq_s[wid][lane] = cq;
#pragma unroll
    for (int t = 0; t < Q; ++t) {
      q_s[wid][lane][t] = make_float4(q[4 * t], q[4 * t + 1], q[4 * t + 2], q[4 * t + 3]);
      if (lane == 0) {
        box_s[wid][0][t] = make_float4(blo[4 * t], blo[4 * t + 1], blo[4 * t + 2], blo[4 * t + 3]);
        box_s[wid][1][t] = make_float4(bhi[4 * t], bhi[4 * t + 1], bhi[4 * t + 2], bhi[4 * t + 3]);
      }
    }
    __syncwarp();
    float bd = __uint_as_float(FMAX_BITS), limit = bd;  // limit: of the component, at least bd
    uint32_t bj = NO_POINT, bo = 0;
    auto refresh = [&]() {
      const uint32_t cb = __shfl_sync(FULL, lane == 0 ? __ldcg(cbest + qc) : 0u, 0);
      limit = __uint_as_float(cb < FMAX_BITS ? cb + 1u : FMAX_BITS);
      if (limit < bd) {
        bd = limit;
        bj = NO_POINT;
      }
    };
    refresh();
    auto bound = [&](int64_t v) {  // box to box, monotone as mst_box_lb
      const bool own = parts.maj[v] == qc;
      const float c = own ? parts.core_rest[v] : parts.core_all[v];
      const float4* l4 = reinterpret_cast<const float4*>(own ? parts.lo : tree.lo) + v * Q;
      const float4* h4 = reinterpret_cast<const float4*>(own ? parts.hi : tree.hi) + v * Q;
      float r = 0.0f;
#pragma unroll
      for (int t = 0; t < Q; ++t) {
        const float4 a = __ldg(l4 + t), b = __ldg(h4 + t);
        const float4 ql = box_s[wid][0][t], qh = box_s[wid][1][t];
        const float2 l0 = fsub2(make_float2(a.x, a.y), make_float2(qh.x, qh.y));
        const float2 l1 = fsub2(make_float2(a.z, a.w), make_float2(qh.z, qh.w));
        const float2 h0 = fsub2(make_float2(ql.x, ql.y), make_float2(b.x, b.y));
        const float2 h1 = fsub2(make_float2(ql.z, ql.w), make_float2(b.z, b.w));
        const float2 d0 = make_float2(fmaxf(fmaxf(l0.x, h0.x), 0.0f), fmaxf(fmaxf(l0.y, h0.y), 0.0f));
        const float2 d1 = make_float2(fmaxf(fmaxf(l1.x, h1.x), 0.0f), fmaxf(fmaxf(l1.y, h1.y), 0.0f));
        const float2 s0 = fmul2(d0, d0), s1 = fmul2(d1, d1);
        r = fadd(fadd(fadd(fadd(r, s0.x), s0.y), s1.x), s1.y);
      }
      return fmaxf(r, c);
    };
    MstWalk w{(int64_t)1 << g0, g0, 0, INF};
    if (lane < (1 << g0)) w.p = bound(w.base + lane);
    while (!(cmin > limit)) {
      const int64_t node = mst_next(w, limit, lane);
      if (node < 0) {
        if (!mst_ascend(w, stack, g0, lane)) break;
        continue;
      }
      // the points that the node may still matter to
      const bool own = parts.maj[node] == qc;
      const float lb = fmaxf(mst_box_lb<DIMP>(own ? parts.lo : tree.lo, own ? parts.hi : tree.hi,
                                              node, q),
                             own ? parts.core_rest[node] : parts.core_all[node]);
      uint32_t todo = __ballot_sync(FULL, active && !(cq > bd) && !(lb > bd));
      if (todo == 0u) continue;
      if (w.level < tree.depth) {
        mst_descend(w, stack, node, lane);
        w.p = bound(w.base + lane);
        continue;
      }
      const int64_t j = (node - tree.P) * MST_LEAF + lane;
      float cj = INF;
      bool foreign = false;
      if (j < tree.n && comp[j] != qc) {
        cj = core[j];
        foreign = !(cj > limit);
      }
      if (__ballot_sync(FULL, foreign) == 0u) continue;
      float y[DIMP];
#pragma unroll
      for (int d = 0; d < DIMP; ++d) y[d] = 0.0f;
      if (foreign) mst_load<DIMP>(tree.xs, j, y);
      for (; todo; todo &= todo - 1) {
        const int src = __ffs(todo) - 1;
        float p[DIMP];
#pragma unroll
        for (int t = 0; t < Q; ++t) {
          const float4 x = q_s[wid][src][t];
          p[4 * t] = x.x, p[4 * t + 1] = x.y, p[4 * t + 2] = x.z, p[4 * t + 3] = x.w;
        }
        const float mr = foreign ? fmaxf(fmaxf(mst_sqd<DIMP>(p, y), cq_s[wid][src]), cj) : INF;
        if (__ballot_sync(FULL, mr <= limit) == 0u) continue;
        const uint32_t mb = __float_as_uint(mr), best = __reduce_min_sync(FULL, mb);
        const uint32_t sb = __float_as_uint(__shfl_sync(FULL, bd, src));
        const uint32_t sj = __shfl_sync(FULL, bj, src);
        if (best < sb || (best == sb && sj != NO_POINT)) {  // as in k_mst_noc
          const uint32_t oj = mb == best ? orig[j] : NO_POINT;
          const uint32_t o = __reduce_min_sync(FULL, oj);
          const int at = __ffs(__ballot_sync(FULL, mb == best && oj == o)) - 1;
          if (lane == src && (best < sb || o < bo)) {
            if (best < sb) atomicMin(cbest + qc, best);
            bd = __uint_as_float(best);
            bo = o;
            bj = (uint32_t)(j - lane + at);
          }
        }
      }
      refresh();
    }
    if (active) {
      near_j[pos] = bj;
      near_v[pos] = fmaxf(near_v[pos], bd);
      if (bj != NO_POINT)
        atomicMin(ckey + qc, ((unsigned long long)__float_as_uint(bd) << 32) | orig[pos]);
    }
  }
}

// Per active component k (id A[k]): its pick (point, other point, value bits)
// and the component of the other end.
__global__ void k_mst_picks(const uint32_t* __restrict__ A, int64_t m,
                            const unsigned long long* __restrict__ ckey,
                            const uint32_t* __restrict__ pos_of, const uint32_t* __restrict__ bj,
                            const uint32_t* __restrict__ orig, const uint32_t* __restrict__ comp,
                            uint32_t* __restrict__ succ, uint32_t* __restrict__ eu,
                            uint32_t* __restrict__ ev, uint32_t* __restrict__ ew,
                            int32_t* __restrict__ has) {
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= m) return;
  const uint32_t c = A[k];
  const unsigned long long key = ckey[c];
  if (key == ~0ull) {
    succ[c] = c;
    has[k] = 0;
    return;
  }
  const uint32_t i = (uint32_t)key, pj = bj[pos_of[i]];
  succ[c] = comp[pj];
  eu[k] = i;
  ev[k] = orig[pj];
  ew[k] = (uint32_t)(key >> 32);
  has[k] = 1;
}

__global__ void k_mst_dbl_init(const uint32_t* __restrict__ A, int64_t m,
                               const uint32_t* __restrict__ succ, uint32_t* __restrict__ jmp,
                               uint32_t* __restrict__ mx, uint32_t* __restrict__ oncyc) {
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= m) return;
  const uint32_t c = A[k], s = succ[c];
  jmp[c] = s;
  mx[c] = max(c, s);
  oncyc[c] = 0u;
}

// One doubling step: jmp becomes succ applied twice as often, and mx the
// maximum over the path c .. jmp (both inclusive).
__global__ void k_mst_dbl_step(const uint32_t* __restrict__ A, int64_t m,
                               const uint32_t* __restrict__ jin, const uint32_t* __restrict__ min_,
                               uint32_t* __restrict__ jout, uint32_t* __restrict__ mout) {
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= m) return;
  const uint32_t c = A[k], j = jin[c];
  jout[c] = jin[j];
  mout[c] = max(min_[c], min_[j]);
}

__global__ void k_mst_mark(const uint32_t* __restrict__ A, int64_t m,
                           const uint32_t* __restrict__ jmp, uint32_t* __restrict__ oncyc) {
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= m) return;
  oncyc[jmp[A[k]]] = 1u;
}

// The skipped pick of each cycle: its largest component (also a component
// without a pick). par: the skipped component itself, else the pick's target.
__global__ void k_mst_skip(const uint32_t* __restrict__ A, int64_t m,
                           const uint32_t* __restrict__ succ, const uint32_t* __restrict__ mx,
                           const uint32_t* __restrict__ oncyc, const int32_t* __restrict__ has,
                           uint32_t* __restrict__ par, uint32_t* __restrict__ nid,
                           int32_t* __restrict__ keep) {
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= m) return;
  const uint32_t c = A[k];
  const bool root = oncyc[c] != 0u && mx[c] == c;
  par[c] = root ? c : succ[c];
  nid[c] = 0xffffffffu;
  keep[k] = (has[k] && !root) ? 1 : 0;
}

__global__ void k_mst_jump(const uint32_t* __restrict__ A, int64_t m,
                           const uint32_t* __restrict__ pin, uint32_t* __restrict__ pout) {
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= m) return;
  const uint32_t c = A[k];
  pout[c] = pin[pin[c]];
}

__global__ void k_mst_newid(const uint32_t* __restrict__ A, int64_t m,
                            const uint32_t* __restrict__ par, uint32_t* __restrict__ nid) {
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= m) return;
  const uint32_t c = A[k];
  atomicMin(nid + par[c], c);
}

__global__ void k_mst_label(const uint32_t* __restrict__ A, int64_t m,
                            const uint32_t* __restrict__ par, const uint32_t* __restrict__ nid,
                            uint32_t* __restrict__ lab, int32_t* __restrict__ alive) {
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= m) return;
  const uint32_t c = A[k], l = nid[par[c]];
  lab[c] = l;
  alive[k] = l == c ? 1 : 0;
}

// Kept picks appended at base in ascending component id; weights square-rooted.
__global__ void k_mst_emit(int64_t m, const int32_t* __restrict__ keep,
                           const int64_t* __restrict__ off, const uint32_t* __restrict__ eu,
                           const uint32_t* __restrict__ ev, const uint32_t* __restrict__ ew,
                           int64_t base, int64_t* __restrict__ u, int64_t* __restrict__ v,
                           float* __restrict__ w) {
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= m || !keep[k]) return;
  const int64_t o = base + off[k];
  u[o] = eu[k];
  v[o] = ev[k];
  w[o] = fsqrt(__uint_as_float(ew[k]));
}

__global__ void k_mst_relabel(uint32_t* __restrict__ comp, int64_t n,
                              const uint32_t* __restrict__ lab) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) comp[i] = lab[comp[i]];
}

__global__ void k_mst_compact(const uint32_t* __restrict__ A, int64_t m,
                              const int32_t* __restrict__ alive, const int64_t* __restrict__ off,
                              uint32_t* __restrict__ A2) {
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k < m && alive[k]) A2[off[k]] = A[k];
}

// The whole merge (k_mst_picks to k_mst_compact but the relabelling) of at most
// MERGE_ONE components in one block: by itself each of the 2 K + 10 steps is a launch
// of 2 us for a microsecond's work. Components are held by their rank in A (ascending
// ids, so ranks order them the same), everything but the picks and the outputs in
// shared memory. tot: picks kept, components left. Rounds of 2,003, 63, 15 and 2
// components take 344 us in all, 690 in launches of their own.
constexpr int MERGE_ONE = 2048;
constexpr int MERGE_THREADS = MERGE_ONE / 2;  // ranks 2 t and 2 t + 1 each
struct MergeArgs {
  const uint32_t* A;
  const unsigned long long* ckey;
  const uint32_t* pos_of;
  const uint32_t* bj;
  const uint32_t* orig;
  const uint32_t* comp;
  uint32_t* rank;  // scratch by component id
  uint32_t* lab;   // out, by component id
  uint32_t* A2;    // out: components left
  int64_t* u;      // out: edges from base on
  int64_t* v;
  float* w;
  int64_t base;
  int64_t* tot;
  int m, K;
};
__global__ void __launch_bounds__(MERGE_THREADS) k_mst_merge_one(MergeArgs a) {
  __shared__ uint16_t succ[MERGE_ONE], ja[MERGE_ONE], jb[MERGE_ONE], ma[MERGE_ONE], mb[MERGE_ONE];
  __shared__ uint8_t oncyc[MERGE_ONE];
  __shared__ uint32_t nid[MERGE_ONE];
  __shared__ int2 sums[32];
  const unsigned FULL = 0xffffffffu;
  const int t = threadIdx.x, lane = t & 31, k0 = 2 * t;
  uint32_t id[2], eu[2], ev[2], ew[2];
  bool has[2];
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    id[q] = 0;
    if (k0 + q < a.m) {
      id[q] = a.A[k0 + q];
      a.rank[id[q]] = (uint32_t)(k0 + q);
    }
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const int k = k0 + q;
    has[q] = false;
    if (k >= a.m) continue;
    const unsigned long long key = a.ckey[id[q]];
    uint32_t s = (uint32_t)k;
    if (key != ~0ull) {
      eu[q] = (uint32_t)key;
      const uint32_t pj = a.bj[a.pos_of[eu[q]]];
      s = *(volatile const uint32_t*)(a.rank + a.comp[pj]);
      ev[q] = a.orig[pj];
      ew[q] = (uint32_t)(key >> 32);
      has[q] = true;
    }
    succ[k] = ja[k] = (uint16_t)s;
    ma[k] = (uint16_t)max((uint32_t)k, s);
    oncyc[k] = 0;
    nid[k] = 0xffffffffu;
  }
  __syncthreads();
  uint16_t *jin = ja, *jout = jb, *min_ = ma, *mout = mb;
  for (int step = 0; step < a.K; ++step) {  // as k_mst_dbl_step
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      const int k = k0 + q;
      if (k >= a.m) continue;
      const uint16_t j = jin[k];
      jout[k] = jin[j];
      mout[k] = max(min_[k], min_[j]);
    }
    __syncthreads();
    uint16_t* x = jin;
    jin = jout;
    jout = x;
    x = min_;
    min_ = mout;
    mout = x;
  }
#pragma unroll
  for (int q = 0; q < 2; ++q)
    if (k0 + q < a.m) oncyc[jin[k0 + q]] = 1;
  __syncthreads();
  bool keep[2], alive[2];
  uint16_t *pin = jout, *pout = mout;
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const int k = k0 + q;
    keep[q] = alive[q] = false;
    if (k >= a.m) continue;
    const bool root = oncyc[k] != 0 && min_[k] == k;
    pin[k] = root ? (uint16_t)k : succ[k];
    keep[q] = has[q] && !root;
  }
  __syncthreads();
  for (int step = 0; step <= a.K; ++step) {
#pragma unroll
    for (int q = 0; q < 2; ++q)
      if (k0 + q < a.m) pout[k0 + q] = pin[pin[k0 + q]];
    __syncthreads();
    uint16_t* x = pin;
    pin = pout;
    pout = x;
  }
#pragma unroll
  for (int q = 0; q < 2; ++q)
    if (k0 + q < a.m) atomicMin(nid + pin[k0 + q], (uint32_t)(k0 + q));
  __syncthreads();
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const int k = k0 + q;
    if (k >= a.m) continue;
    const uint32_t l = nid[pin[k]];
    a.lab[id[q]] = a.A[l];
    alive[q] = l == (uint32_t)k;
  }
  // ranks among the kept and the living before this thread's
  int2 c = make_int2((int)keep[0] + (int)keep[1], (int)alive[0] + (int)alive[1]), inc = c;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int x = __shfl_up_sync(FULL, inc.x, o), y = __shfl_up_sync(FULL, inc.y, o);
    if (lane >= o) {
      inc.x += x;
      inc.y += y;
    }
  }
  if (lane == 31) sums[t >> 5] = inc;
  __syncthreads();
  int2 all = sums[lane];
  const int2 own = all;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int x = __shfl_up_sync(FULL, all.x, o), y = __shfl_up_sync(FULL, all.y, o);
    if (lane >= o) {
      all.x += x;
      all.y += y;
    }
  }
  const int before = t >> 5;
  const int bx = __shfl_sync(FULL, all.x - own.x, before), by = __shfl_sync(FULL, all.y - own.y, before);
  if (t == MERGE_THREADS - 1) {
    a.tot[0] = bx + inc.x;
    a.tot[1] = by + inc.y;
  }
  int64_t e = a.base + bx + inc.x - c.x;
  int l = by + inc.y - c.y;
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    if (keep[q]) {
      a.u[e] = eu[q];
      a.v[e] = ev[q];
      a.w[e] = fsqrt(__uint_as_float(ew[q]));
      ++e;
    }
    if (alive[q]) a.A2[l++] = id[q];
  }
}

__global__ void k_mst_iota(uint32_t* __restrict__ a, int64_t n) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) a[i] = (uint32_t)i;
}

int log2_ceil(int64_t m) {
  int k = 0;
  while (((int64_t)1 << k) < m) ++k;
  return k;
}

template <int DIMP>
int64_t mst_run(evoc_ctx* ctx, const float* d_data, int64_t n, int dim, int k, int64_t* d_u,
                int64_t* d_v, float* d_w) {
  cudaStream_t s = ctx->stream;
  int32_t* st = ctx->status.get();
  StageTrace tr(s);
  {
    const unsigned g = (unsigned)std::min<int64_t>(grid_of(n * dim), 4 * ctx->num_sms);
    k_mst_finite<<<g, 256, 0, s>>>(d_data, n * dim, st);
    EVOC_CHECK_LAUNCH();
  }
  check_status(ctx, "build_mst");  // non-finite coordinates are rejected before any search
  // tree order of the points
  const int64_t L = (n + MST_LEAF - 1) / MST_LEAF;
  int64_t P = 1;
  while (P < L) P <<= 1;
  DevBuf<uint32_t> key(n, s);
  DevBuf<uint2> val(n, s);
  k_mst_iota_pairs<<<grid_of(n), 256, 0, s>>>(val.get(), n);
  EVOC_CHECK_LAUNCH();
  {
    int64_t size = P * MST_LEAF;
    const int64_t max_nodes = (n + 2 * KD_BLOCK - 1) / (2 * KD_BLOCK);
    DevBuf<uint32_t> box(2 * max_nodes * dim, s);
    for (; size > KD_BLOCK; size >>= 1) {
      const int64_t nodes = (n + size - 1) / size;
      uint32_t *bmin = box.get(), *bmax = box.get() + nodes * dim;
      EVOC_CUDA(cudaMemsetAsync(bmin, 0xff, nodes * dim * sizeof(uint32_t), s));
      EVOC_CUDA(cudaMemsetAsync(bmax, 0, nodes * dim * sizeof(uint32_t), s));
      k_kd_box<<<grid_of((n + KD_RUN - 1) / KD_RUN, 128), 128, 0, s>>>(d_data, n, dim, size,
                                                                     val.get(), bmin, bmax);
      EVOC_CHECK_LAUNCH();
      const int nb = bits_for((uint64_t)(nodes - 1)), bits = std::min(24, 32 - nb);
      k_kd_key<<<grid_of(n), 256, 0, s>>>(d_data, n, dim, size, bits, val.get(), bmin, bmax,
                                          key.get());
      EVOC_CHECK_LAUNCH();
      radix_sort_pairs(ctx, key, val, n, nb + bits);
    }
    if (size >= 2 * MST_LEAF) {
      EVOC_CUDA(cudaFuncSetAttribute((const void*)k_kd_block,
                                     cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)sizeof(KdSmem)));
      k_kd_block<<<(unsigned)((n + size - 1) / size), KD_THREADS, sizeof(KdSmem), s>>>(
          d_data, n, dim, (int)size, val.get());
      EVOC_CHECK_LAUNCH();
    }
  }
  DevBuf<float> xs(n * DIMP, s);
  DevBuf<uint32_t> orig(n, s), pos_of(n, s);
  k_mst_gather<DIMP><<<grid_of(n), 256, 0, s>>>(d_data, n, dim, val.get(), xs.get(), orig.get(),
                                                pos_of.get());
  EVOC_CHECK_LAUNCH();
  key.release();
  val.release();
  tr.mark("tree order");
  DevBuf<float> lo(2 * P * DIMP, s), hi(2 * P * DIMP, s);
  k_mst_leaf_boxes<DIMP><<<grid_of(P), 256, 0, s>>>(xs.get(), n, P, L, lo.get(), hi.get());
  EVOC_CHECK_LAUNCH();
  for (int64_t first = P; first > 1; first = std::max<int64_t>(first / UP_NODES, 1)) {
    k_mst_boxes_up<DIMP><<<grid_of(first, UP_NODES), UP_NODES / 2, 0, s>>>(lo.get(), hi.get(),
                                                                         first);
    EVOC_CHECK_LAUNCH();
  }
  tr.mark("tree boxes");
  // core distances
  const MstTree<DIMP> tree{xs.get(), lo.get(), hi.get(), n, P, log2_ceil(P)};
  auto search_grid = [&](int64_t items) {
    return (unsigned)std::max<int64_t>(1, std::min<int64_t>((int64_t)mst_blocks<DIMP>() * ctx->num_sms,
                                                           (items + MST_WARPS - 1) / MST_WARPS));
  };
  DevBuf<unsigned long long> work(3, s);  // the searches' next point, groups and their next
  EVOC_CUDA(cudaMemsetAsync(work.get(), 0, work.bytes(), s));
  DevBuf<float> core(n, s), knn_d(n * (int64_t)k, s);
  DevBuf<uint32_t> knn_j(n * (int64_t)k, s);
  DevBuf<uint8_t> tie(n, s);
  if (k == 0) {
    EVOC_CUDA(cudaMemsetAsync(core.get(), 0, core.bytes(), s));
  } else {
    auto* kern = k <= 32 ? k_mst_core<DIMP, false> : k_mst_core<DIMP, true>;
    kern<<<search_grid(n), 32 * MST_WARPS, 0, s>>>(tree, k, work.get(), core.get(), knn_j.get(),
                                                   knn_d.get(), tie.get());
    EVOC_CHECK_LAUNCH();
  }
  tr.mark("core distances");
  // Boruvka rounds
  DevBuf<uint32_t> comp(n, s), maj(2 * P, s), cbest(n, s), near_j(n, s), list(n, s), succ(n, s);
  DevBuf<float> near_v(n, s), plo(2 * P * DIMP, s), phi(2 * P * DIMP, s), pcore(4 * P, s);
  DevBuf<int32_t> mcnt(2 * P, s);
  const MstParts<DIMP> parts{maj.get(), mcnt.get(),  plo.get(),
                             phi.get(), pcore.get(), pcore.get() + 2 * P};
  DevBuf<unsigned long long> ckey(n, s);
  // Groups pay where their searches fill the chip: none below one leaf per resident
  // warp of that kernel (100 k points: 4.7 ms without, 5.0 to 5.5 with), half leaves up
  // to four (200 k: 9.2 ms without, 7.9 by 16, 8.3 by 32 points; 16 dimensions,
  // 300 k: 88, 49 and 55 ms), whole leaves above (1 M: 38.8, 23.3 and 22.5 ms).
  const int64_t resident = (int64_t)MST_GROUP_BLOCKS * MST_WARPS * ctx->num_sms;
  const bool by_group = L >= resident;
  const int width = L >= 4 * resident ? 32 : 16;
  const int64_t max_groups = by_group ? L * (MST_LEAF / width) : 0;
  // 16 dimensions: searches are so long that few groups still beat them (48.7 and 58.0 ms)
  const unsigned long long min_groups = DIMP > 8 ? 1 : (unsigned long long)resident;
  DevBuf<uint2> groups(max_groups, s);
  const unsigned group_grid = (unsigned)(MST_GROUP_BLOCKS * ctx->num_sms);
  DevBuf<uint32_t> jA(n, s), jB(n, s), mA(n, s), mB(n, s), oncyc(n, s), nid(n, s), lab(n, s);
  DevBuf<uint32_t> A(n, s), A2(n, s), eu(n, s), ev(n, s), ew(n, s);
  DevBuf<int32_t> has(n, s), keep(n, s), alive(n, s);
  DevBuf<int64_t> off(n + 1, s), off2(n + 1, s), tot(2, s);
  EVOC_CUDA(cudaMemcpyAsync(comp.get(), orig.get(), comp.bytes(), cudaMemcpyDeviceToDevice, s));
  k_mst_iota<<<grid_of(n), 256, 0, s>>>(A.get(), n);
  EVOC_CHECK_LAUNCH();
  k_mst_near_init<<<grid_of(n), 256, 0, s>>>(n, k, knn_j.get(), tie.get(), core.get(), orig.get(),
                                             near_j.get(), near_v.get());
  EVOC_CHECK_LAUNCH();
  int64_t m = n, len = 0;
  int64_t h_tot[2];
  while (m > 1 && len < n - 1) {
    const unsigned gm = grid_of(m), gn = grid_of(n);
    k_mst_leaf_parts<DIMP><<<grid_of(P * 32), 256, 0, s>>>(tree, comp.get(), core.get(), parts);
    EVOC_CHECK_LAUNCH();
    for (int64_t first = P; first > 1; first = std::max<int64_t>(first / UP_NODES, 1)) {
      k_mst_parts_up<DIMP><<<grid_of(first, UP_NODES), UP_NODES / 2, 0, s>>>(tree, parts, first);
      EVOC_CHECK_LAUNCH();
    }
    k_mst_round_reset<<<gm, 256, 0, s>>>(A.get(), m, cbest.get(), ckey.get());
    EVOC_CHECK_LAUNCH();
    k_mst_bound<DIMP><<<gn, 256, 0, s>>>(xs.get(), n, k, knn_j.get(), knn_d.get(), comp.get(), core.get(),
                                   near_j.get(), near_v.get(), cbest.get());
    EVOC_CHECK_LAUNCH();
    EVOC_CUDA(cudaMemsetAsync(work.get(), 0, work.bytes(), s));
    k_mst_select<<<gn, 256, 0, s>>>(n, comp.get(), core.get(), orig.get(), near_j.get(),
                                    near_v.get(), cbest.get(), ckey.get(), has.get(),
                                    by_group ? groups.get() : nullptr, work.get() + 1, width);
    EVOC_CHECK_LAUNCH();
    if (by_group) {
      k_mst_take_groups<<<grid_of(max_groups), 256, 0, s>>>(groups.get(), work.get() + 1,
                                                            min_groups, has.get());
      EVOC_CHECK_LAUNCH();
    }
    exclusive_scan_i32_to_i64(ctx, has.get(), off.get(), n);
    k_mst_search_list<<<gn, 256, 0, s>>>(n, has.get(), off.get(), list.get());
    EVOC_CHECK_LAUNCH();
    if (by_group) {
      k_mst_noc_group<DIMP><<<group_grid, 32 * MST_WARPS, 0, s>>>(
          tree, parts, comp.get(), core.get(), orig.get(), groups.get(), work.get() + 1,
          min_groups, work.get() + 2, cbest.get(), ckey.get(), near_j.get(), near_v.get());
      EVOC_CHECK_LAUNCH();
    }
    k_mst_noc<DIMP><<<search_grid(n), 32 * MST_WARPS, 0, s>>>(
        tree, parts, comp.get(), core.get(), orig.get(), list.get(), off.get() + n, work.get(),
        cbest.get(), ckey.get(), near_j.get(), near_v.get());
    EVOC_CHECK_LAUNCH();
    if (m <= MERGE_ONE) {
      const MergeArgs ma{A.get(),    ckey.get(), pos_of.get(), near_j.get(), orig.get(),
                         comp.get(), nid.get(),  lab.get(),    A2.get(),     d_u,
                         d_v,        d_w,        len,          tot.get(),    (int)m,
                         std::max(1, log2_ceil(m))};
      k_mst_merge_one<<<1, MERGE_THREADS, 0, s>>>(ma);
      EVOC_CHECK_LAUNCH();
      EVOC_CUDA(cudaMemcpyAsync(h_tot, tot.get(), sizeof(h_tot), cudaMemcpyDeviceToHost, s));
    } else {
      k_mst_picks<<<gm, 256, 0, s>>>(A.get(), m, ckey.get(), pos_of.get(), near_j.get(), orig.get(),
                                     comp.get(), succ.get(), eu.get(), ev.get(), ew.get(), has.get());
      EVOC_CHECK_LAUNCH();
      // cycles of the pick graph: 2^K >= m doubling steps
      const int K = std::max(1, log2_ceil(m));
      k_mst_dbl_init<<<gm, 256, 0, s>>>(A.get(), m, succ.get(), jA.get(), mA.get(), oncyc.get());
      EVOC_CHECK_LAUNCH();
      uint32_t *jin = jA.get(), *jout = jB.get(), *min_ = mA.get(), *mout = mB.get();
      for (int t = 0; t < K; ++t) {  // after t steps: jmp = succ^(2^(t+1)), mx over that path
        k_mst_dbl_step<<<gm, 256, 0, s>>>(A.get(), m, jin, min_, jout, mout);
        EVOC_CHECK_LAUNCH();
        std::swap(jin, jout);
        std::swap(min_, mout);
      }
      k_mst_mark<<<gm, 256, 0, s>>>(A.get(), m, jin, oncyc.get());
      EVOC_CHECK_LAUNCH();
      // the skipped picks, then the merged components by pointer jumping
      uint32_t *pin = jout, *pout = mout;  // free ping-pong buffers
      k_mst_skip<<<gm, 256, 0, s>>>(A.get(), m, succ.get(), min_, oncyc.get(), has.get(), pin,
                                    nid.get(), keep.get());
      EVOC_CHECK_LAUNCH();
      for (int t = 0; t <= K; ++t) {
        k_mst_jump<<<gm, 256, 0, s>>>(A.get(), m, pin, pout);
        EVOC_CHECK_LAUNCH();
        std::swap(pin, pout);
      }
      k_mst_newid<<<gm, 256, 0, s>>>(A.get(), m, pin, nid.get());
      EVOC_CHECK_LAUNCH();
      k_mst_label<<<gm, 256, 0, s>>>(A.get(), m, pin, nid.get(), lab.get(), alive.get());
      EVOC_CHECK_LAUNCH();
      exclusive_scan_i32_to_i64(ctx, keep.get(), off.get(), m);
      exclusive_scan_i32_to_i64(ctx, alive.get(), off2.get(), m);
      k_mst_emit<<<gm, 256, 0, s>>>(m, keep.get(), off.get(), eu.get(), ev.get(), ew.get(), len,
                                    d_u, d_v, d_w);
      EVOC_CHECK_LAUNCH();
      k_mst_compact<<<gm, 256, 0, s>>>(A.get(), m, alive.get(), off2.get(), A2.get());
      EVOC_CHECK_LAUNCH();
      EVOC_CUDA(cudaMemcpyAsync(&h_tot[0], off.get() + m, sizeof(int64_t), cudaMemcpyDeviceToHost, s));
      EVOC_CUDA(cudaMemcpyAsync(&h_tot[1], off2.get() + m, sizeof(int64_t), cudaMemcpyDeviceToHost, s));
    }
    k_mst_relabel<<<gn, 256, 0, s>>>(comp.get(), n, lab.get());
    EVOC_CHECK_LAUNCH();
    EVOC_CUDA(cudaStreamSynchronize(s));
    std::swap(A, A2);
    const int64_t kept = h_tot[0];
    len += kept;
    if (tr.on) {
      const std::string name = "round, " + std::to_string(m) + " components";
      tr.mark(name.c_str());
    }
    m = h_tot[1];
    if (kept == 0) break;  // no pick merged anything (mst.rs:143-160)
  }
  return len;
}

}  // namespace

int64_t build_mst_device(evoc_ctx* ctx, const float* d_data, int64_t n, int32_t dim,
                         int32_t min_samples, int64_t* d_u, int64_t* d_v, float* d_w) {
  if (n < 0) throw Error(EVOC_ERR_INVALID_ARGUMENT, "n must be >= 0");
  if (n > 0xfffffff0LL) throw Error(EVOC_ERR_UNSUPPORTED, "n must be below 2^32 - 16");
  if (dim < 1 || dim > 16) throw Error(EVOC_ERR_UNSUPPORTED, "dim must be in 1..16");
  if (min_samples < 0) throw Error(EVOC_ERR_INVALID_ARGUMENT, "min_samples must be >= 0");
  if (n <= 1) return 0;
  if (!d_data || !d_u || !d_v || !d_w)
    throw Error(EVOC_ERR_INVALID_ARGUMENT, "NULL argument");
  const int k = (int)std::min<int64_t>(min_samples, n - 1);
  if (k > 64) throw Error(EVOC_ERR_UNSUPPORTED, "min_samples above 64 is not supported");
  if (dim <= 4) return mst_run<4>(ctx, d_data, n, dim, k, d_u, d_v, d_w);
  if (dim <= 8) return mst_run<8>(ctx, d_data, n, dim, k, d_u, d_v, d_w);
  return mst_run<16>(ctx, d_data, n, dim, k, d_u, d_v, d_w);
}

}  // namespace evoc
