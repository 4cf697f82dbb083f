// fuzzy_set.cu — fuzzy simplicial set on the GPU.
//
// Replaces, in evoc-rs 0.2.7:
//   smooth_knn_dist            src/graph/fuzzy_graph.rs:33-98
//   knn_to_coo                 src/graph/fuzzy_graph.rs:114-159
//   symmetrise_graph           src/graph/fuzzy_graph.rs:174-228
//   coo_to_adjacency_list      src/graph/fuzzy_graph.rs:242-256
//   build_fuzzy_simplicial_set src/graph/fuzzy_graph.rs:275-295
//
// Pipeline (all on the context stream):
//   k_knn_rowlen     warp per row: row length (first EVOC_KNN_PAD) and index
//                    validation.
//   k_smooth_knn     lane per row: rho, the sigma bisection (steps whose outcome
//                    is certain are not evaluated) and the membership weights
//                    (fuzzy_graph.rs:138-145). An evaluated sum is serial in
//                    row order, as in the reference (fuzzy_graph.rs:72-76), so
//                    sigma is bit-identical to a serial CPU evaluation.
//   k_forward_*      drop self loops, sort by column keeping
//                    the last of equal columns (HashMap::insert overwrites,
//                    fuzzy_graph.rs:189), count in-degrees.
//   radix sort       stable sort of the forward entries by column: each
//                    column bucket lists its source rows in ascending order,
//                    which is the backward map of fuzzy_graph.rs:190.
//   k_union          warp per row: merge the sorted forward and backward
//                    lists, w = w_ij + w_ji - w_ij * w_ji, keep w > 0
//                    (fuzzy_graph.rs:196-204), into per-row scratch;
//                    k_union_compact copies the kept pairs into the CSR.
#include "evoc_device.cuh"
#include "evoc_internal.h"

#include <algorithm>
#include <cmath>

namespace evoc {
namespace {

constexpr uint32_t PAD = EVOC_KNN_PAD;

// ---------------------------------------------------------------------------
// Row lengths and index validation (warp per row, coalesced).
// ---------------------------------------------------------------------------
__global__ void k_knn_rowlen(const uint32_t* __restrict__ idx, int64_t n,
                             int32_t k, int32_t* __restrict__ row_len,
                             int32_t* __restrict__ status) {
  const int64_t row = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (row >= n) return;
  const uint32_t* r = idx + row * (int64_t)k;
  int32_t len = k;
  for (int32_t base = 0; base < k; base += 32) {
    const int32_t j = base + lane;
    const uint32_t c = (j < k) ? r[j] : PAD;
    const uint32_t pads = __ballot_sync(0xffffffffu, j < k && c == PAD);
    if (pads) {
      const int32_t first = base + __ffs(pads) - 1;
      if (j < first && (int64_t)c >= n) set_status(status, ST_BAD_INDEX);
      len = first;
      break;
    }
    if (j < k && (int64_t)c >= n) set_status(status, ST_BAD_INDEX);
  }
  if (lane == 0) row_len[row] = len;
}

// ---------------------------------------------------------------------------
// smooth_knn_dist (fuzzy_graph.rs:33-98): rho, the sigma bisection and the
// membership weights, one row per lane, a warp's rows staged in shared memory (odd
// row stride: lanes on different rows hit different banks).
//
// The bisection's outcome is defined by the f32 sum val(mid) of the row's
// exponentials, added serially in row order, and by the side of the target it
// falls on. Most of its steps (27 on average) lie so far from the target that the
// side is certain, so their sums are never formed. In real arithmetic S(x) = sum
// exp(-a_j x), x = 1 / mid, is decreasing and convex: Newton's iteration from
// x = 0 approaches the solution from below, with hardware ex2 (4 instructions per
// term, against about 45 of an exactly rounded term). Two points on either side of
// it are then certified: where the approximate sum is further than W from the
// target, with W = 1e-5 (the bisection's own tolerance) + a bound M on all
// rounding, val is on that side and not converged, and by monotony so it is for
// every mid beyond that point. Steps between the two points (about three) are
// evaluated exactly as written in the reference, so sigma and the step count are
// bit-identical to a serial evaluation of every step. Rows for which nothing can
// be certified (no solution, extreme distances) evaluate every step.
//
// M, for len terms of at most 1 each: the exact terms are off by at most 1.5e-7
// (quotient, own exp at 1.2 ulp), the approximate ones by 2.4e-7 (ex2.approx
// 2^-22.5, argument 3 roundings), either sum by len * sum * 2^-24, the target's
// rounding by 5e-7. 2M rows of 30: 3.3 ms when every step was evaluated, 0.90 now;
// bound by instruction issue (0.87 a cycle and scheduler at 500k rows). Rows that cannot
// be certified cost the Newton steps on top and hold their warp: 1M rows of 16, every
// step evaluated in pools of rows / now: exactly 4 zeros in each row 0.43 / 0.43 ms, in
// one of 32 0.79 / 0.43, an infinity in one of 32 0.79 / 0.70, distances of 3e38 in
// each row 1.14 / 0.97, in one of 32 1.17 / 1.09.
// ---------------------------------------------------------------------------
struct RowState {
  int32_t len;
  int32_t it;
  float rho, lo, hi, mid;
};

// Checks a row, takes its rho and replaces its distances by max(0, d - rho).
__device__ __forceinline__ bool sk_start_row(RowState& st, float* __restrict__ d, int32_t len,
                                             float lc, int32_t* __restrict__ status) {
  st.len = len;
  st.it = 0;
  st.lo = 0.0f;
  st.hi = 3.40282347e+38f;
  st.mid = 1.0f;
  st.rho = 0.0f;
  bool ok = true;
  for (int32_t j = 0; j < len; ++j)
    if (d[j] != d[j]) ok = false;
  if (!ok) set_status(status, ST_BAD_VALUE);
  if (lc > 0.0f) {  // fuzzy_graph.rs:49-62
    if (len <= 0) {
      set_status(status, ST_EMPTY_ROW);
      ok = false;
    } else {
      const float lm1 = max0(fsub(lc, 1.0f));
      const float fl = floorf(lm1);
      int64_t id = (int64_t)fl;
      if (id > len - 1) id = len - 1;
      const float frac = fsub(lm1, fl);
      if (frac > 0.0f && id + 1 < len)
        st.rho = fadd(fmul(d[id], fsub(1.0f, frac)), fmul(d[id + 1], frac));
      else
        st.rho = d[id];
    }
  }
  for (int32_t j = 0; j < len; ++j) d[j] = max0(fsub(d[j], st.rho));
  return ok;
}

__device__ __forceinline__ float sk_ex2(float x) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// Certified sides of the target: above for mid >= *up, below for mid <= *down
// (infinity and 0 where nothing is certified).
__device__ __forceinline__ void sk_certify(const float* __restrict__ a, int32_t len, double target,
                                           bool on, float* up, float* down) {
  const float INF = __int_as_float(0x7f800000);
  constexpr float LOG2E = 1.44269504f;
  const float t = (float)target, flen = (float)len;
  const float w = 1.05e-5f + 5e-7f + flen * (4e-7f + 1.2e-7f * (fabsf(t) + 1.0f));
  float sum = 0.0f;
  int32_t zeros = 0;
  for (int32_t j = 0; j < len; ++j) {
    sum += a[j];
    zeros += a[j] == 0.0f;
  }
  *up = INF;
  *down = 0.0f;
  if (on && (float)zeros - t > w) {  // the zeros alone exceed the target at every mid
    *up = 0.0f;
    on = false;
  }
  if (on && t - flen > w) {  // every term at 1 does not reach it
    *down = INF;
    on = false;
  }
  float x = (flen - t) / sum, g = 0.0f;
  on = on && x > 1e-30f && x < 1e30f;
  bool solved = false;
  for (int it = 0; it < 16; ++it) {
    if (!__any_sync(0xffffffffu, on && !solved)) break;
    if (on && !solved) {
      const float c = -x * LOG2E;
      float s = 0.0f, d = 0.0f;
#pragma unroll 4
      for (int32_t j = 0; j < len; ++j) {
        const float e = sk_ex2(a[j] * c);
        s += e;
        d = fmaf(a[j], e, d);
      }
      g = x * d;
      const float r = s - t;
      if (fabsf(r) <= 0.25f * w)
        solved = true;
      else
        x += r / d;
      on = x > 1e-30f && x < 1e30f;  // also not NaN
    }
  }
  const float del = 1.5f * w / g;
  if (on && solved && del < 0.3f) {
    const float xl = x * (1.0f - del), xh = x * (1.0f + del);
    const float cl = -xl * LOG2E, ch = -xh * LOG2E;
    float sl = 0.0f, sh = 0.0f;
#pragma unroll 4
    for (int32_t j = 0; j < len; ++j) {
      sl += sk_ex2(a[j] * cl);
      sh += sk_ex2(a[j] * ch);
    }
    if (sl - t > w) *up = 1.000001f / xl;
    if (t - sh > w) *down = 0.999999f / xh;
  }
}

__global__ void k_smooth_knn(const float* __restrict__ dist, const int32_t* __restrict__ row_len,
                             int64_t n, int32_t k, int32_t kp, double target, float lc,
                             int32_t n_iter, float* __restrict__ sigma_out,
                             float* __restrict__ rho_out, float* __restrict__ w_out,
                             int32_t* __restrict__ status, unsigned long long* __restrict__ steps) {
  extern __shared__ float sm[];
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  float* sd = sm + (size_t)wid * 32 * kp;
  const int64_t row0 = ((int64_t)blockIdx.x * (blockDim.x >> 5) + wid) * 32;
  if (row0 >= n) return;  // whole warp
  const int rows = (int)min((int64_t)32, n - row0);
  const uint32_t elems = (uint32_t)rows * (uint32_t)k;
  {
    const float* src = dist + row0 * (int64_t)k;
    for (uint32_t e = lane; e < elems; e += 32) {
      const uint32_t r = e / (uint32_t)k;
      sd[r * kp + (e - r * k)] = src[e];
    }
  }
  __syncwarp();
  float* a = sd + lane * kp;
  const int64_t row = row0 + lane;
  RowState st{};
  bool live = lane < rows, ok = false;
  if (live) ok = sk_start_row(st, a, row_len ? row_len[row] : k, lc, status);
  if (live && !ok) {
    st.mid = 0.0f;
    st.rho = 0.0f;
    live = false;
  }
  float up, down;
  sk_certify(a, live ? st.len : 0, target, live, &up, &down);
  uint32_t nsteps = 0;  // bisection steps of this lane's row
  while (__any_sync(FULL, live)) {
    // steps whose side is certain, then one exact evaluation (fuzzy_graph.rs:71-93)
    bool above = false;
    while (live) {
      if (st.it >= n_iter) {
        live = false;
        break;
      }
      const bool in_range = st.mid > 1e-30f && st.mid < 1e30f;
      above = in_range && st.mid >= up;
      if (!above && !(in_range && st.mid <= down)) break;
      ++nsteps;
      if (above) {
        st.hi = st.mid;
        st.mid = fdiv(fadd(st.lo, st.hi), 2.0f);
      } else {
        st.lo = st.mid;
        st.mid = st.hi == 3.40282347e+38f ? fmul(st.mid, 2.0f) : fdiv(fadd(st.lo, st.hi), 2.0f);
      }
      ++st.it;
    }
    __syncwarp();
    if (live) {
      ++nsteps;
      float val = 0.0f;
#pragma unroll 2
      for (int32_t j = 0; j < st.len; ++j) val = fadd(val, evoc_expf(-fdiv(a[j], st.mid)));
      const double vd = (double)val;
      if (fabs(vd - target) < 1e-5) {
        live = false;
      } else {
        if (vd > target) {
          st.hi = st.mid;
          st.mid = fdiv(fadd(st.lo, st.hi), 2.0f);
        } else {
          st.lo = st.mid;
          st.mid = st.hi == 3.40282347e+38f ? fmul(st.mid, 2.0f) : fdiv(fadd(st.lo, st.hi), 2.0f);
        }
        ++st.it;
      }
    }
  }
  if (lane < rows) {
    sigma_out[row] = st.mid;
    rho_out[row] = st.rho;
  }
  const unsigned tot = __reduce_add_sync(FULL, nsteps);
  if (lane == 0 && tot) atomicAdd(steps, (unsigned long long)tot);
  if (!w_out) return;
  // knn_to_coo's membership weights (fuzzy_graph.rs:138-145): w = exp(-max(0, d -
  // rho) / sigma), or 0 / 1 when sigma <= 0 (and 0 past the row's end; a rejected
  // row's are never read)
  __syncwarp();
  for (uint32_t e0 = 0; e0 < elems; e0 += 32) {
    const uint32_t e = e0 + lane;
    const int r = (int)min(e / (uint32_t)k, 31u);
    const int32_t j = (int32_t)(e - (uint32_t)r * k);
    const float mid = __shfl_sync(FULL, st.mid, r);
    const int32_t len = __shfl_sync(FULL, st.len, r);
    if (e < elems) {
      float out = 0.0f;
      if (j < len) {
        const float adjusted = sd[r * kp + j];
        out = mid > 0.0f ? evoc_expf(-fdiv(adjusted, mid)) : (adjusted > 0.0f ? 0.0f : 1.0f);
      }
      w_out[row0 * (int64_t)k + e] = out;
    }
  }
}

// ---------------------------------------------------------------------------
// Forward lists: drop self loops, sort by column (stable), keep the last entry
// of each column, count in-degrees. Rows stay padded to k. The lists leave twice:
// as (fcol, fw) for the union, and as (column, (row, weight)) pairs, PAD past a
// row's end, which the stable sort by column turns into the backward lists.
// Rows of up to 32: G lanes per row sort (column, position) in registers, 2M rows
// of 30 in 0.63 ms (the insertion sort 0.98, and 0.4 for the pairs). Longer rows: a
// thread per row, insertion sort in shared memory.
// ---------------------------------------------------------------------------
template <int G>
__global__ void __launch_bounds__(256) k_forward_short(
    const uint32_t* __restrict__ idx, const float* __restrict__ w,
    const int32_t* __restrict__ row_len, int64_t n, int32_t k, uint32_t* __restrict__ fcol,
    float* __restrict__ fw, uint32_t* __restrict__ keys, uint2* __restrict__ vals,
    int32_t* __restrict__ fcnt, int32_t* __restrict__ indeg) {
  const unsigned FULL = 0xffffffffu;
  const int64_t row = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / G;
  const int lane = threadIdx.x & 31, sub = threadIdx.x & (G - 1);
  const bool valid = row < n;
  const int32_t len = valid ? row_len[row] : 0;
  const int64_t at = row * (int64_t)k + sub;
  uint32_t c = PAD, pos = sub;
  float wv = 0.0f;
  if (sub < len) {
    c = idx[at];
    wv = w[at];
    if ((int64_t)c == row) c = PAD;  // self loop (fuzzy_graph.rs:135)
  }
#pragma unroll
  for (int size = 2; size <= G; size <<= 1)
#pragma unroll
    for (int stride = size >> 1; stride >= 1; stride >>= 1) {
      const uint32_t oc = __shfl_xor_sync(FULL, c, stride), op = __shfl_xor_sync(FULL, pos, stride);
      const bool low = ((sub & size) == 0) == ((sub & stride) == 0);
      const bool less = oc < c || (oc == c && op < pos);
      if (low == less) {
        c = oc;
        pos = op;
      }
    }
  wv = __shfl_sync(FULL, wv, (int)pos, G);
  const uint32_t next = __shfl_down_sync(FULL, c, 1, G);
  const bool keep = c != PAD && (sub == G - 1 || next != c);  // the last of equal columns
  uint32_t kept = __ballot_sync(FULL, keep);
  if (G < 32) kept = (kept >> (lane & ~(G - 1))) & ((1u << (G & 31)) - 1u);
  const int cnt = __popc(kept);
  if (!valid) return;
  if (keep) {
    const int64_t o = row * (int64_t)k + __popc(kept & ((1u << sub) - 1u));
    fcol[o] = c;
    fw[o] = wv;
    keys[o] = c;
    vals[o] = make_uint2((uint32_t)row, __float_as_uint(wv));
    atomicAdd(&indeg[c], 1);
  }
  if (sub >= cnt && sub < k) {
    keys[at] = PAD;
    vals[at] = make_uint2(0u, 0u);
  }
  if (sub == 0) fcnt[row] = cnt;
}

__global__ void k_forward_rows(const uint32_t* __restrict__ idx,
                               const float* __restrict__ w,
                               const int32_t* __restrict__ row_len, int64_t n,
                               int32_t k, int32_t kp,
                               uint32_t* __restrict__ fcol,
                               float* __restrict__ fw,
                               uint32_t* __restrict__ keys,
                               uint2* __restrict__ vals,
                               int32_t* __restrict__ fcnt,
                               int32_t* __restrict__ indeg) {
  extern __shared__ uint32_t smu[];
  const int R = blockDim.x;
  uint32_t* sc = smu;
  float* sw = reinterpret_cast<float*>(smu + (size_t)R * kp);
  const int64_t row0 = (int64_t)blockIdx.x * R;
  const int64_t rows_here = min((int64_t)R, n - row0);
  const int64_t elems = rows_here * k;
  for (int64_t e = threadIdx.x; e < elems; e += R) {
    const int64_t r = e / k, j = e - r * k;
    sc[r * kp + j] = idx[row0 * (int64_t)k + e];
    sw[r * kp + j] = w[row0 * (int64_t)k + e];
  }
  __syncthreads();
  if (threadIdx.x < rows_here) {
    const int64_t i = row0 + threadIdx.x;
    uint32_t* c = sc + threadIdx.x * kp;
    float* ww = sw + threadIdx.x * kp;
    const int32_t len = row_len[i];
    int32_t m = 0;  // compact: drop self loops (fuzzy_graph.rs:135)
    for (int32_t j = 0; j < len; ++j)
      if ((int64_t)c[j] != i) {
        c[m] = c[j];
        ww[m] = ww[j];
        ++m;
      }
    for (int32_t j = 1; j < m; ++j) {  // stable insertion sort by column
      const uint32_t cj = c[j];
      const float wj = ww[j];
      int32_t q = j - 1;
      while (q >= 0 && c[q] > cj) {
        c[q + 1] = c[q];
        ww[q + 1] = ww[q];
        --q;
      }
      c[q + 1] = cj;
      ww[q + 1] = wj;
    }
    int32_t cnt = 0;  // keep the last of each run of equal columns
    for (int32_t j = 0; j < m; ++j)
      if (j + 1 == m || c[j + 1] != c[j]) {
        c[cnt] = c[j];
        ww[cnt] = ww[j];
        ++cnt;
      }
    fcnt[i] = cnt;
    for (int32_t j = 0; j < cnt; ++j) atomicAdd(&indeg[c[j]], 1);
    for (int32_t j = cnt; j < k; ++j) c[j] = PAD;
  }
  __syncthreads();
  for (int64_t e = threadIdx.x; e < elems; e += R) {
    const int64_t r = e / k, j = e - r * k;
    const int64_t o = row0 * (int64_t)k + e;
    fcol[o] = sc[r * kp + j];
    fw[o] = sw[r * kp + j];
    keys[o] = sc[r * kp + j];
    vals[o] = make_uint2((uint32_t)(row0 + r), __float_as_uint(sw[r * kp + j]));
  }
}

// Fuzzy union of row i (fuzzy_graph.rs:193-205), warp per row: the forward
// list (sorted by column, at most k entries) merged with the backward list
// (sorted by source row). Each step loads the next 32 entries of both lists
// (coalesced); every entry finds its rank in the other chunk by a shuffle
// search, a column present in both is emitted once with both weights, and
// only columns up to the smaller of the two chunks' last entries are final.
// Emitted entries are placed by merged rank in shared memory, then the kept
// ones (w_sym > 0) are written in order. Output goes to the row's scratch
// region at i * k + bptr[i]; out_cnt[i] gets the kept count.
__global__ void __launch_bounds__(256) k_union(const uint32_t* __restrict__ fcol,
                                               const float* __restrict__ fw,
                                               const int32_t* __restrict__ fcnt,
                                               const int64_t* __restrict__ bptr,
                                               const uint2* __restrict__ bvals, int64_t n,
                                               int32_t k, int32_t* __restrict__ out_cnt,
                                               uint2* __restrict__ tmp) {
  __shared__ uint2 stage_all[8][64];
  uint2* stage = stage_all[threadIdx.x >> 5];
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const uint32_t lt = (1u << lane) - 1u;
  const int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (i >= n) return;
  const uint32_t* fa = fcol + i * (int64_t)k;
  const float* fwa = fw + i * (int64_t)k;
  const int32_t na = fcnt[i];
  const int64_t b0 = bptr[i], nb = bptr[i + 1] - b0;
  const uint2* bv = bvals + b0;
  uint2* out = tmp + i * (int64_t)k + b0;
  int32_t ia = 0;
  int64_t ib = 0;
  int32_t cnt = 0;
  while (ia < na || ib < nb) {
    const bool has_a = ia + lane < na, has_b = ib + lane < nb;
    const uint32_t a = has_a ? fa[ia + lane] : PAD;
    const float wa = has_a ? fwa[ia + lane] : 0.0f;
    const uint2 bb = has_b ? bv[ib + lane] : make_uint2(PAD, 0u);
    const uint32_t b = bb.x;
    const int ca = (int)min((int64_t)32, (int64_t)(na - ia));
    const int cb = (int)min((int64_t)32, nb - ib);
    // columns up to `bound` are final: every unread entry is larger
    uint32_t bound = 0xffffffffu;
    if (ia + 32 < na) bound = min(bound, __shfl_sync(FULL, a, 31));
    if (ib + 32 < nb) bound = min(bound, __shfl_sync(FULL, b, 31));
    // rank of a in the b chunk (# b < a) and of b in the a chunk (# a < b)
    int ra = 0, rb = 0;
#pragma unroll
    for (int step = 16; step >= 1; step >>= 1) {
      if (__shfl_sync(FULL, b, ra + step - 1) < a) ra += step;
      if (__shfl_sync(FULL, a, rb + step - 1) < b) rb += step;
    }
    if (ra < 32 && __shfl_sync(FULL, b, ra) < a) ++ra;  // lanes past the chunk hold PAD
    if (rb < 32 && __shfl_sync(FULL, a, rb) < b) ++rb;
    const uint32_t b_at = __shfl_sync(FULL, b, ra & 31);
    const uint32_t b_w = __shfl_sync(FULL, bb.y, ra & 31);
    const uint32_t a_at = __shfl_sync(FULL, a, rb & 31);
    const bool a_take = has_a && a <= bound;
    const bool a_match = a_take && ra < cb && b_at == a;
    const bool b_take = has_b && b <= bound;
    const bool b_match = b_take && rb < ca && a_at == b;
    const uint32_t ma = __ballot_sync(FULL, a_match), mb = __ballot_sync(FULL, b_match);
    // merged rank = # distinct columns before this one among the taken entries
    if (a_take) {
      const float w_ji = a_match ? __uint_as_float(b_w) : 0.0f;
      const float w_sym = fsub(fadd(wa, w_ji), fmul(wa, w_ji));
      stage[lane + ra - __popc(ma & lt)] = make_uint2(a, __float_as_uint(w_sym));
    }
    if (b_take && !b_match) {
      const float w_ji = __uint_as_float(bb.y);
      const float w_sym = fsub(fadd(0.0f, w_ji), fmul(0.0f, w_ji));
      stage[lane + rb - __popc(mb & lt)] = make_uint2(b, __float_as_uint(w_sym));
    }
    const int na_t = __popc(__ballot_sync(FULL, a_take));
    const int nb_t = __popc(__ballot_sync(FULL, b_take));
    const int m = na_t + nb_t - __popc(ma);  // distinct columns emitted
    __syncwarp();
    // kept entries (w_sym > 0) in merged order
    for (int base = 0; base < m; base += 32) {
      const int e = base + lane;
      const uint2 v = e < m ? stage[e] : make_uint2(0u, 0u);
      const bool keep = e < m && __uint_as_float(v.y) > 0.0f;
      const uint32_t kb = __ballot_sync(FULL, keep);
      if (keep) out[cnt + __popc(kb & lt)] = v;
      cnt += __popc(kb);
    }
    __syncwarp();
    ia += na_t;
    ib += nb_t;
  }
  if (lane == 0) out_cnt[i] = cnt;
}

// Warp per row: the row's kept pairs from its scratch region into the CSR.
__global__ void k_union_compact(const uint2* __restrict__ tmp,
                                const int64_t* __restrict__ bptr, int64_t n, int32_t k,
                                const int64_t* __restrict__ out_ptr,
                                uint32_t* __restrict__ out_idx, float* __restrict__ out_w) {
  const int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (i >= n) return;
  const uint2* src = tmp + i * (int64_t)k + bptr[i];
  const int64_t dst = out_ptr[i], len = out_ptr[i + 1] - dst;
  for (int64_t j = lane; j < len; j += 32) {
    const uint2 v = src[j];
    out_idx[dst + j] = v.x;
    out_w[dst + j] = __uint_as_float(v.y);
  }
}

// symmetrise == false: the directed COO of knn_to_coo in kNN order.
template <bool WRITE>
__global__ void k_directed(const uint32_t* __restrict__ idx,
                           const float* __restrict__ w,
                           const int32_t* __restrict__ row_len, int64_t n,
                           int32_t k, int32_t* __restrict__ out_cnt,
                           const int64_t* __restrict__ out_ptr,
                           uint32_t* __restrict__ out_idx,
                           float* __restrict__ out_w) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int32_t len = row_len[i];
  int64_t o = WRITE ? out_ptr[i] : 0;
  int32_t cnt = 0;
  for (int32_t j = 0; j < len; ++j) {
    const uint32_t c = idx[i * (int64_t)k + j];
    if ((int64_t)c == i) continue;
    if (WRITE) {
      out_idx[o] = c;
      out_w[o] = w[i * (int64_t)k + j];
      ++o;
    }
    ++cnt;
  }
  if (!WRITE) out_cnt[i] = cnt;
}

int rows_per_block(int32_t kp) {
  if ((size_t)128 * kp * 8 <= 48 * 1024) return 128;
  if ((size_t)64 * kp * 8 <= 96 * 1024) return 64;
  return 32;
}

void set_smem_limit(const void* fn, size_t bytes) {
  if (bytes > 48 * 1024)
    EVOC_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   (int)bytes));
}

}  // namespace

void smooth_knn_device(evoc_ctx* ctx, const float* d_dist,
                       const int32_t* d_row_len, int64_t n, int32_t k,
                       uint64_t k_target, float local_connectivity,
                       int32_t n_iter, float* d_sigma, float* d_rho,
                       float* d_weights_out) {
  if (n == 0) return;
  const int32_t kp = k | 1;
  // four warps per block, one where that leaves SMs idle or the rows are long
  int warps = 4;
  while (warps > 1 && (n < (int64_t)64 * warps * ctx->num_sms ||
                       (size_t)warps * 32 * kp * sizeof(float) > 200 * 1024))
    warps /= 2;
  const size_t smem = (size_t)warps * 32 * kp * sizeof(float);
  if ((size_t)4 * 32 * kp * sizeof(float) > 200 * 1024)
    throw Error(EVOC_ERR_UNSUPPORTED, "k too large (k <= 399 supported)");
  set_smem_limit((const void*)k_smooth_knn, smem);
  const double target = std::log2((double)k_target);
  const int64_t per_block = (int64_t)warps * 32;
  const int64_t blocks = (n + per_block - 1) / per_block;
  EVOC_CUDA(cudaMemsetAsync(ctx->sk_steps.get(), 0, sizeof(unsigned long long), ctx->stream));
  k_smooth_knn<<<(unsigned)blocks, 32 * warps, smem, ctx->stream>>>(
      d_dist, d_row_len, n, k, kp, target, local_connectivity, n_iter, d_sigma, d_rho,
      d_weights_out, ctx->status.get(), ctx->sk_steps.get());
  EVOC_CHECK_LAUNCH();
}

void fuzzy_set_device(evoc_ctx* ctx, const uint32_t* d_idx,
                      const float* d_dist, int64_t n, int32_t k,
                      float effective_n_neighbours, bool symmetrise,
                      float* d_sigmas_out, float* d_rhos_out, evoc_graph* out) {
  cudaStream_t s = ctx->stream;
  if (n <= 0)
    throw Error(EVOC_ERR_INVALID_ARGUMENT,
                "empty kNN graph (build_fuzzy_simplicial_set reads row 0)");
  if (k <= 0) throw Error(EVOC_ERR_INVALID_ARGUMENT, "k must be positive");
  if (n >= (int64_t)PAD) throw Error(EVOC_ERR_UNSUPPORTED, "n must be < 2^32-1");

  StageTrace trace(s);
  DevBuf<int32_t> row_len(n, s);
  {
    const int64_t threads = n * 32;
    k_knn_rowlen<<<(unsigned)((threads + 255) / 256), 256, 0, s>>>(
        d_idx, n, k, row_len.get(), ctx->status.get());
    EVOC_CHECK_LAUNCH();
  }
  trace.mark("row lengths");

  // k = effective_n_neighbors.to_usize().unwrap_or(knn_dists[0].len())
  // (fuzzy_graph.rs:284-286)
  uint64_t kk;
  const float e = effective_n_neighbours;
  if (e > -1.0f && e < 18446744073709551616.0f) {
    kk = (uint64_t)e;
  } else {
    int32_t len0 = 0;
    EVOC_CUDA(cudaMemcpyAsync(&len0, row_len.get(), sizeof(int32_t),
                              cudaMemcpyDeviceToHost, s));
    EVOC_CUDA(cudaStreamSynchronize(s));
    kk = (uint64_t)len0;
  }

  DevBuf<float> sig_local, rho_local;
  float* d_sig = d_sigmas_out;
  float* d_rho = d_rhos_out;
  if (!d_sig) { sig_local.alloc(n, s); d_sig = sig_local.get(); }
  if (!d_rho) { rho_local.alloc(n, s); d_rho = rho_local.get(); }
  DevBuf<float> wts(n * (int64_t)k, s);
  smooth_knn_device(ctx, d_dist, row_len.get(), n, k, kk, 1.0f, 64, d_sig,
                    d_rho, wts.get());
  check_status(ctx, "fuzzy set");
  trace.mark("smooth knn + weights");

  out->ctx = ctx;
  out->n = n;
  out->indptr.alloc(n + 1, s);
  const unsigned row_blocks = (unsigned)((n + 255) / 256);

  if (!symmetrise) {
    DevBuf<int32_t> cnt(n, s);
    k_directed<false><<<row_blocks, 256, 0, s>>>(d_idx, wts.get(), row_len.get(),
                                                  n, k, cnt.get(), nullptr,
                                                  nullptr, nullptr);
    EVOC_CHECK_LAUNCH();
    exclusive_scan_i32_to_i64(ctx, cnt.get(), out->indptr.get(), n);
    int64_t nnz = 0;
    EVOC_CUDA(cudaMemcpyAsync(&nnz, out->indptr.get() + n, sizeof(int64_t),
                              cudaMemcpyDeviceToHost, s));
    EVOC_CUDA(cudaStreamSynchronize(s));
    out->nnz = nnz;
    out->indices.alloc(nnz, s);
    out->weights.alloc(nnz, s);
    k_directed<true><<<row_blocks, 256, 0, s>>>(
        d_idx, wts.get(), row_len.get(), n, k, nullptr, out->indptr.get(),
        out->indices.get(), out->weights.get());
    EVOC_CHECK_LAUNCH();
    out->canonical = false;
    EVOC_CUDA(cudaStreamSynchronize(s));
    return;
  }

  // forward lists, and their pairs for the transpose
  const int64_t nk = n * (int64_t)k;
  DevBuf<uint32_t> fcol(nk, s), keys(nk, s);
  DevBuf<float> fw(nk, s);
  DevBuf<uint2> vals(nk, s);
  DevBuf<int32_t> fcnt(n, s), indeg(n, s);
  EVOC_CUDA(cudaMemsetAsync(indeg.get(), 0, n * sizeof(int32_t), s));
  if (k <= 32) {
    auto* kern = k <= 16 ? k_forward_short<16> : k_forward_short<32>;
    const int64_t threads = n * (k <= 16 ? 16 : 32);
    kern<<<(unsigned)((threads + 255) / 256), 256, 0, s>>>(
        d_idx, wts.get(), row_len.get(), n, k, fcol.get(), fw.get(), keys.get(), vals.get(),
        fcnt.get(), indeg.get());
  } else {
    const int32_t kp = k | 1;
    int R = rows_per_block(kp);
    const size_t smem = (size_t)R * kp * 8;
    if (smem > 200 * 1024)
      throw Error(EVOC_ERR_UNSUPPORTED, "k too large (k <= 1599 supported)");
    set_smem_limit((const void*)k_forward_rows, smem);
    k_forward_rows<<<(unsigned)((n + R - 1) / R), R, smem, s>>>(
        d_idx, wts.get(), row_len.get(), n, k, kp, fcol.get(), fw.get(), keys.get(), vals.get(),
        fcnt.get(), indeg.get());
  }
  EVOC_CHECK_LAUNCH();
  wts.release();
  trace.mark("forward rows");

  // stable transpose: the pairs by column (PAD, above every column, last)
  DevBuf<int64_t> bptr(n + 1, s);
  exclusive_scan_i32_to_i64(ctx, indeg.get(), bptr.get(), n);
  radix_sort_pairs(ctx, keys, vals, nk, bits_for((uint64_t)n));
  keys.release();
  trace.mark("transpose");

  DevBuf<int32_t> ucnt(n, s);
  DevBuf<uint2> utmp(2 * nk, s);  // at most k entries each way per row
  k_union<<<(unsigned)((n * 32 + 255) / 256), 256, 0, s>>>(
      fcol.get(), fw.get(), fcnt.get(), bptr.get(), vals.get(), n, k, ucnt.get(), utmp.get());
  EVOC_CHECK_LAUNCH();
  exclusive_scan_i32_to_i64(ctx, ucnt.get(), out->indptr.get(), n);
  int64_t nnz = 0;
  EVOC_CUDA(cudaMemcpyAsync(&nnz, out->indptr.get() + n, sizeof(int64_t),
                            cudaMemcpyDeviceToHost, s));
  EVOC_CUDA(cudaStreamSynchronize(s));
  out->nnz = nnz;
  out->indices.alloc(nnz, s);
  out->weights.alloc(nnz, s);
  trace.mark("union merge");
  k_union_compact<<<(unsigned)((n * 32 + 255) / 256), 256, 0, s>>>(
      utmp.get(), bptr.get(), n, k, out->indptr.get(), out->indices.get(),
      out->weights.get());
  EVOC_CHECK_LAUNCH();
  out->canonical = true;
  trace.mark("union compact");
  EVOC_CUDA(cudaStreamSynchronize(s));
}

}  // namespace evoc
