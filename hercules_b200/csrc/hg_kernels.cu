// hg_kernels.cu -- sm_100a kernels of the Hercules exact k-NN path.
//
// Data layout in HBM: the leaf-ordered rows, row-major -- the image of
// leaves_raw.idx.  A row of L floats is L/8 chunks of 32 bytes; the distance
// kernel reads a row four chunks (one 128-byte line) at a time and stops at
// the line where the row abandons.  Distances follow the reference's
// summation order exactly (hg_arith.cuh).
#include <cuda_runtime.h>
#include <stdint.h>

#include "hg_arith.cuh"
#include "hg_gen.cuh"
#include "hg_device.cuh"
#include "hg_kernels.h"

namespace hg {

// Adds the lanes' chunk sums 0 .. lim - 1 in chunk order, eight a turn, so the
// shuffles run ahead of the two chains of adds; a chunk past the end adds 0,
// which leaves the sums unchanged.
__device__ __forceinline__ void warp_add_chunks(float cs, float cq, int lim, float& sum, float& sumsq) {
  for (int j = 0; j < lim; j += 8) {
    float s8[8], q8[8];
#pragma unroll
    for (int t = 0; t < 8; ++t) {
      s8[t] = __shfl_sync(HG_FULL, cs, j + t);
      q8[t] = __shfl_sync(HG_FULL, cq, j + t);
    }
#pragma unroll
    for (int t = 0; t < 8; ++t) {
      sum = __fadd_rn(sum, s8[t]);
      sumsq = __fadd_rn(sumsq, q8[t]);
    }
  }
}

__device__ __forceinline__ void segment_stats(float sum, float sumsq, int count, float* mean, float* stdev) {
  const float fc = (float)count;
  *mean = __fdiv_rn(sum, fc);
  sumsq = __fsub_rn(sumsq, __fdiv_rn(__fmul_rn(sum, sum), fc));
  *stdev = __fsqrt_rn(__fdiv_rn(sumsq, fc));
}

// Mean and stdev of v[from, to) in the order of calc_mean_stdev_SIMD: the
// lanes compute the 8-chunk sums in parallel, then every lane accumulates
// them in chunk order (identical warp-uniform result).
__device__ void warp_mean_stdev(const float* v, int from, int to, float* mean, float* stdev) {
  const int lane = threadIdx.x & 31;
  const int count = to - from;
  if (count <= 0) {
    *mean = 0.0f;
    *stdev = 0.0f;
    return;
  }
  const int nch = (count + 7) >> 3;
  float sum = 0.0f, sumsq = 0.0f;
  for (int base = 0; base < nch; base += 32) {
    const int c = base + lane;
    float cs = 0.0f, cq = 0.0f;
    if (c < nch) {
      float x[8], x2[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int i = c * 8 + j;
        x[j] = i < count ? v[from + i] : 0.0f;
        x2[j] = __fmul_rn(x[j], x[j]);
      }
      cs = hg_hsum8(x[0], x[1], x[2], x[3], x[4], x[5], x[6], x[7]);
      cq = hg_hsum8(x2[0], x2[1], x2[2], x2[3], x2[4], x2[5], x2[6], x2[7]);
    }
    warp_add_chunks(cs, cq, min(32, nch - base), sum, sumsq);
  }
  segment_stats(sum, sumsq, count, mean, stdev);
}

// Walks the tree from the root (node_split_policy_route_to_left,
// hercules_node_split.c:172-193).  Returns the leaf index.
__device__ int warp_route(const float* q, const Tree& t) {
  int node = t.root;
  while (node >= 0) {
    const DNode n = t.nodes[node];
    float m, s;
    warp_mean_stdev(q, n.from, n.to, &m, &s);
    const float v = n.idx ? s : m;
    node = (v < n.value) ? n.left : n.right;
  }
  return ~node;
}

__device__ __forceinline__ uint32_t tiles_of_leaf(uint64_t start, uint32_t size) {
  if (size == 0) return 0;
  return (uint32_t)(((start + size - 1) >> 5) - (start >> 5) + 1);
}

// ---------------------------------------------------------------------------
// block-wide helpers
// ---------------------------------------------------------------------------

template <int THREADS>
__device__ uint32_t block_exclusive_scan(uint32_t v, uint32_t* tmp /* THREADS/32 + 1 */, uint32_t* total) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  uint32_t x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    uint32_t y = __shfl_up_sync(HG_FULL, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) tmp[w] = x;
  __syncthreads();
  if (w == 0) {
    uint32_t s = lane < THREADS / 32 ? tmp[lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      uint32_t y = __shfl_up_sync(HG_FULL, s, o);
      if (lane >= o) s += y;
    }
    if (lane < THREADS / 32) tmp[lane] = s;
    if (lane == THREADS / 32 - 1) tmp[THREADS / 32] = s;
  }
  __syncthreads();
  const uint32_t excl = x - v + (w > 0 ? tmp[w - 1] : 0);
  if (total) *total = tmp[THREADS / 32];
  __syncthreads();
  return excl;
}

// ---------------------------------------------------------------------------
// build kernels
// ---------------------------------------------------------------------------

// Mean and stdev as warp_mean_stdev, of a row in global memory: a chunk's
// eight floats in two 16-byte loads where the segment starts on 16 bytes.
__device__ void warp_mean_stdev_row(const float* x, int from, int to, float* mean, float* stdev) {
  const int lane = threadIdx.x & 31;
  const int count = to - from;
  *mean = 0.0f;
  *stdev = 0.0f;
  if (count <= 0) return;
  const float* v = x + from;
  const bool wide = (reinterpret_cast<uintptr_t>(v) & 15) == 0;
  const int nch = (count + 7) >> 3;
  float sum = 0.0f, sumsq = 0.0f;
  for (int base = 0; base < nch; base += 32) {
    const int c = base + lane;
    float cs = 0.0f, cq = 0.0f;
    if (c < nch) {
      float e[8], e2[8];
      if (wide && c * 8 + 8 <= count) {
        const float4 a = reinterpret_cast<const float4*>(v)[2 * c], b = reinterpret_cast<const float4*>(v)[2 * c + 1];
        e[0] = a.x; e[1] = a.y; e[2] = a.z; e[3] = a.w;
        e[4] = b.x; e[5] = b.y; e[6] = b.z; e[7] = b.w;
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) e[j] = c * 8 + j < count ? v[c * 8 + j] : 0.0f;
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) e2[j] = __fmul_rn(e[j], e[j]);
      cs = hg_hsum8(e[0], e[1], e[2], e[3], e[4], e[5], e[6], e[7]);
      cq = hg_hsum8(e2[0], e2[1], e2[2], e2[3], e2[4], e2[5], e2[6], e2[7]);
    }
    warp_add_chunks(cs, cq, min(32, nch - base), sum, sumsq);
  }
  segment_stats(sum, sumsq, count, mean, stdev);
}

// Series up to this length are staged 32 at a time in shared memory (a pitch
// of L + 1 floats: a lane per row reads without bank conflicts), longer ones
// are read by a warp each.  Staged, a lane adds its own row's chunks and a
// segment of 32 rows costs the instructions of one; a thread per row reading
// global memory, as both cases did, touched 32 lines per load (122 us to route
// 65,536 rows of 256, 56 us for the envelopes of 10,000; staged 20 and 9 us).
constexpr int kStagedL = 512;
constexpr int kStagedRows = 32;
__host__ __device__ inline size_t staged_bytes(int L) { return sizeof(float) * kStagedRows * (size_t)(L + 1); }

// `threads` threads bring rows row(0) .. row(n - 1) of X into the tile.
template <class Row>
__device__ __forceinline__ void stage_rows(const float* __restrict__ X, int L, int n, float* tile, int threads, Row row) {
  const int v4 = L >> 2, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = threads >> 5;
  for (int c = lane; c < v4; c += 32)
    for (int r0 = warp; r0 < n; r0 += 4 * nw) {
      float4 v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (r0 + u * nw < n) v[u] = reinterpret_cast<const float4*>(X + row(r0 + u * nw) * (uint64_t)L)[c];
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (r0 + u * nw < n) {
          float* d = tile + (r0 + u * nw) * (L + 1) + 4 * c;
          d[0] = v[u].x;
          d[1] = v[u].y;
          d[2] = v[u].z;
          d[3] = v[u].w;
        }
    }
}

// Walks the current tree to a leaf, a lane per staged row.
__global__ void __launch_bounds__(32) k_route_staged(const float* __restrict__ X, int L, uint64_t first, uint32_t count,
                                                     Tree t, int* __restrict__ node_of) {
  extern __shared__ float tile[];
  const uint32_t r0 = blockIdx.x * kStagedRows;
  const int n = (int)min((uint32_t)kStagedRows, count - r0);
  stage_rows(X, L, n, tile, 32, [&](int r) { return first + r0 + r; });
  __syncwarp();
  if ((int)threadIdx.x >= n) return;
  const float* x = tile + threadIdx.x * (L + 1);
  int node = t.root;
  while (node >= 0) {
    const DNode nd = t.nodes[node];
    float m, s;
    hg_mean_stdev(x, nd.from, nd.to, &m, &s);
    const float v = nd.idx ? s : m;
    node = (v < nd.value) ? nd.left : nd.right;
  }
  node_of[r0 + threadIdx.x] = ~node;
}

// The same with a warp per row.
__global__ void k_route_long(const float* __restrict__ X, int L, uint64_t first, uint32_t count, Tree t,
                             int* __restrict__ node_of) {
  const uint32_t r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (r >= count) return;
  const float* x = X + (first + r) * (uint64_t)L;
  int node = t.root;
  while (node >= 0) {
    const DNode nd = t.nodes[node];
    float m, s;
    warp_mean_stdev_row(x, nd.from, nd.to, &m, &s);
    const float v = nd.idx ? s : m;
    node = (v < nd.value) ? nd.left : nd.right;
  }
  if ((threadIdx.x & 31) == 0) node_of[r] = ~node;
}

// Order-preserving int image of a float for atomicMax/atomicMin.
__device__ __forceinline__ int fkey(float f) {
  int b = __float_as_int(f);
  return b >= 0 ? b : b ^ 0x7fffffff;
}

__device__ __forceinline__ int empty_key(int i) { return (i & 1) ? INT_MAX : INT_MIN; }  // odd: minima

// The rows of the leaves about to split, among the rows routed so far.
__global__ void k_collect_members(const int* __restrict__ node_of, uint64_t end, const int* __restrict__ slot_of,
                                  const uint64_t* __restrict__ start, const uint32_t* __restrict__ last,
                                  uint64_t members, uint32_t* __restrict__ list, uint32_t* counts, uint32_t* later,
                                  int* keys, int nsegs) {
  const uint64_t t0 = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const uint64_t step = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i = t0; i < 4ull * nsegs; i += step) keys[i] = empty_key((int)(i & 1));
  const int lane = threadIdx.x & 31;
  const uint64_t whole = (end + 31) & ~31ull;  // whole warps to the end
  for (uint64_t r = t0; r < whole; r += step) {
    const int p = r < end ? slot_of[node_of[r]] : -1;
    // -1: no row of a splitting leaf; -2: a later row; else the leaf
    const int who = p < 0 ? -1 : (r <= last[p] ? p : -2);
    if (!__any_sync(HG_FULL, who != -1)) continue;
    const uint32_t same = __match_any_sync(HG_FULL, who);
    const int leader = __ffs(same) - 1;
    uint32_t pos = 0;
    if (who != -1 && lane == leader) pos = atomicAdd(who == -2 ? later : &counts[who], (uint32_t)__popc(same));
    pos = __shfl_sync(HG_FULL, pos, leader) + (uint32_t)__popc(same & ((1u << lane) - 1));
    if (who != -1) list[(who == -2 ? members : start[who]) + pos] = (uint32_t)r;
  }
}

// Segment sketches (min/max of per-series segment mean and stdev) over groups
// of rows: node_segment_sketch_update_sketch_parallel applied to every member
// (hercules_node_split.c:86-120).  Min/max are order independent and
// fmaxf/fminf ignore NaN, so skipping NaN gives the same envelope.
struct SketchGroup {
  uint64_t first;
  uint32_t size;
  int seg0, nsegs;
};
__device__ __forceinline__ SketchGroup sketch_group(const SketchArgs& a, int g) {
  return SketchGroup{a.start[g], a.size[g], a.seg_off[g], a.seg_off[g + 1] - a.seg_off[g]};
}
__device__ __forceinline__ uint64_t sketch_row(const SketchArgs& a, const SketchGroup& g, uint64_t i) {
  return a.members ? (uint64_t)a.members[g.first + i] : g.first + i;
}

constexpr int kSketchThreads = 256;
// L <= kStagedL: grid (groups, parts); a tile of 32 rows at a time, a lane per
// row, a warp per segment, whose extremes stay with that warp.
__global__ void __launch_bounds__(kSketchThreads) k_sketch_staged(SketchArgs a) {
  extern __shared__ float tile[];
  int* sk = reinterpret_cast<int*>(tile + kStagedRows * (a.L + 1));  // [segments][4]
  const SketchGroup g = sketch_group(a, blockIdx.x);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if ((uint64_t)blockIdx.y * kStagedRows >= g.size) return;
  for (int i = threadIdx.x; i < 4 * g.nsegs; i += kSketchThreads) sk[i] = empty_key(i);
  for (uint64_t t0 = (uint64_t)blockIdx.y * kStagedRows; t0 < g.size; t0 += (uint64_t)gridDim.y * kStagedRows) {
    const int n = (int)min((uint64_t)kStagedRows, g.size - t0);
    __syncthreads();
    stage_rows(a.X, a.L, n, tile, kSketchThreads, [&](int r) { return sketch_row(a, g, t0 + r); });
    __syncthreads();
    const float* x = tile + min(lane, n - 1) * (a.L + 1);  // lanes past the rows repeat the last
    for (int s = warp; s < g.nsegs; s += kSketchThreads / 32) {
      float m, sd;
      hg_mean_stdev(x, a.seg_from[g.seg0 + s], a.seg_to[g.seg0 + s], &m, &sd);
      const int km = fkey(m), ks = fkey(sd);
      const int k0 = __reduce_max_sync(HG_FULL, m == m ? km : INT_MIN);
      const int k1 = __reduce_min_sync(HG_FULL, m == m ? km : INT_MAX);
      const int k2 = __reduce_max_sync(HG_FULL, sd == sd ? ks : INT_MIN);
      const int k3 = __reduce_min_sync(HG_FULL, sd == sd ? ks : INT_MAX);
      if (lane == 0) {
        sk[4 * s + 0] = max(sk[4 * s + 0], k0);
        sk[4 * s + 1] = min(sk[4 * s + 1], k1);
        sk[4 * s + 2] = max(sk[4 * s + 2], k2);
        sk[4 * s + 3] = min(sk[4 * s + 3], k3);
      }
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < 4 * g.nsegs; i += kSketchThreads) {
    if (i & 1) atomicMin(&a.keys[4 * (size_t)g.seg0 + i], sk[i]);
    else atomicMax(&a.keys[4 * (size_t)g.seg0 + i], sk[i]);
  }
}

// Longer series: a warp per (row, segment).
__global__ void __launch_bounds__(kSketchThreads) k_sketch_long(SketchArgs a) {
  extern __shared__ int sk_long[];
  const SketchGroup g = sketch_group(a, blockIdx.x);
  const int lane = threadIdx.x & 31;
  constexpr int W = kSketchThreads / 32;
  const uint64_t items = (uint64_t)g.size * g.nsegs;
  if ((uint64_t)blockIdx.y * W >= items) return;
  for (int i = threadIdx.x; i < 4 * g.nsegs; i += kSketchThreads) sk_long[i] = empty_key(i);
  __syncthreads();
  for (uint64_t it = (uint64_t)blockIdx.y * W + (threadIdx.x >> 5); it < items; it += (uint64_t)gridDim.y * W) {
    const uint64_t i = it / g.nsegs;
    const int s = (int)(it - i * g.nsegs);
    float m, sd;
    warp_mean_stdev_row(a.X + sketch_row(a, g, i) * (uint64_t)a.L, a.seg_from[g.seg0 + s], a.seg_to[g.seg0 + s], &m, &sd);
    if (lane == 0) {
      if (m == m) {
        atomicMax(&sk_long[4 * s + 0], fkey(m));
        atomicMin(&sk_long[4 * s + 1], fkey(m));
      }
      if (sd == sd) {
        atomicMax(&sk_long[4 * s + 2], fkey(sd));
        atomicMin(&sk_long[4 * s + 3], fkey(sd));
      }
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < 4 * g.nsegs; i += kSketchThreads) {
    if (i & 1) atomicMin(&a.keys[4 * (size_t)g.seg0 + i], sk_long[i]);
    else atomicMax(&a.keys[4 * (size_t)g.seg0 + i], sk_long[i]);
  }
}

// The redistribution of splits (hercules_node_split.c:1294-1333), a warp per
// row; a warp's rows are consecutive in the list, so it counts the left ones
// of a leaf itself and adds them once.
__global__ void k_split_members(const float* __restrict__ X, int L, int* __restrict__ node_of,
                                const uint32_t* __restrict__ list, uint64_t members, const uint32_t* later,
                                const int* __restrict__ slot_of, const SplitPolicy* __restrict__ splits,
                                uint32_t* n_left) {
  const int lane = threadIdx.x & 31;
  const uint64_t nw = ((uint64_t)gridDim.x * blockDim.x) >> 5, w = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint64_t total = members + *later, per = (total + nw - 1) / nw;
  int cur = -1;
  uint32_t left = 0;
  for (uint64_t i = w * per; i < min(total, w * per + per); ++i) {
    const uint64_t r = list[i];
    const int p = slot_of[node_of[r]];
    const SplitPolicy sp = splits[p];
    float m, s;
    warp_mean_stdev_row(X + r * (uint64_t)L, sp.from, sp.to, &m, &s);
    const bool l = (sp.idx ? s : m) < sp.value;
    __syncwarp();  // every lane has read node_of[r]
    if (lane == 0) node_of[r] = l ? sp.left : sp.right;
    if (i < members) {
      if (p != cur) {
        if (lane == 0 && left) atomicAdd(&n_left[cur], left);
        cur = p;
        left = 0;
      }
      left += l ? 1u : 0u;
    }
  }
  if (lane == 0 && left) atomicAdd(&n_left[cur], left);
}

__global__ void k_widen_ids(const uint32_t* __restrict__ perm, uint64_t n, int64_t* __restrict__ ids) {
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) ids[i] = (int64_t)perm[i];
}

// rows[r] = X[perm[r]], one thread per 16 bytes (a row is L/4 of them).
__global__ void k_gather_rows(const float* __restrict__ X, int L, const uint32_t* __restrict__ perm, uint64_t n,
                              float* __restrict__ rows) {
  const int v4 = L >> 2;
  const uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const uint64_t r = t / v4;
  if (r >= n) return;
  const int j = (int)(t % v4);
  reinterpret_cast<float4*>(rows + r * L)[j] = reinterpret_cast<const float4*>(X + (uint64_t)perm[r] * L)[j];
}

// iSAX word of every leaf-ordered row (sax_from_ts, sax.c:86-135): two rows
// per warp, a lane per (row, segment), which adds its segment in order and
// looks its symbol up.  A thread per row took 0.96 ms for 1M x 256 (1.1 TB/s),
// its 32 rows' lines leaving L1 between two of its reads.
__global__ void k_sax_rows(const float* __restrict__ rows, int L, uint64_t n, const float* __restrict__ bp,
                           uint8_t* __restrict__ sax) {
  __shared__ float sbp[256];
  for (int i = threadIdx.x; i < 255; i += blockDim.x) sbp[i] = bp[i];
  __syncthreads();
  const uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const uint64_t row = t / HG_PAA_SEGMENTS;
  if (row >= n) return;
  const int per = L / HG_PAA_SEGMENTS;
  const float* x = rows + row * L + (t % HG_PAA_SEGMENTS) * per;
  float acc = 0.0f;
  if (per % 4 == 0) {
    for (int i = 0; i < per / 4; ++i) {
      const float4 v = reinterpret_cast<const float4*>(x)[i];
      acc = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(acc, v.x), v.y), v.z), v.w);
    }
  } else {
    for (int i = 0; i < per; ++i) acc = __fadd_rn(acc, x[i]);
  }
  sax[t] = (uint8_t)hg_sax_symbol(__fdiv_rn(acc, (float)per), sbp);
}

// ---------------------------------------------------------------------------
// query kernels
// ---------------------------------------------------------------------------

// The approximate leaf of every query, a warp each; the threads also zero the
// batch's counters zero_a and zero_b (the next kernels').
__global__ void k_route_queries(const float* __restrict__ Q, int nq, int L, Tree t, int* __restrict__ leaf_out,
                                uint32_t* zero_a, uint32_t na, uint32_t* zero_b, uint32_t nb,
                                unsigned long long* stamp) {
  stamp_start(stamp);
  const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x, threads = gridDim.x * blockDim.x;
  for (uint32_t i = tid; i < na; i += threads) zero_a[i] = 0;
  for (uint32_t i = tid; i < nb; i += threads) zero_b[i] = 0;
  const int w = (int)(tid >> 5);
  if (w >= nq) return;
  const int leaf = warp_route(Q + (uint64_t)w * L, t);
  if ((threadIdx.x & 31) == 0) leaf_out[w] = leaf;
}

// The start of a group of queries, grid (slots, blocks), one launch instead of
// three on the way to the first scan: blocks y < gridDim.y - 1 compute
// LB_EAPCA of the leaves (a warp per leaf) and, with sax_tab set, block y <
// 16 the LB_SAX terms of segment y (sax_tab[y * 256 + s] =
// hg_lb_sax_lane(paa[y], s), reference arithmetic, sax.c:310-479); the last
// block routes the query (approximate_knn_search's traversal) and resets its
// state for a scan with an unbounded k-th distance.  Bound by latency: the
// routing is a chain of node and segment reads, one per tree level.
constexpr int kPrepThreads = 256;
__global__ void __launch_bounds__(kPrepThreads) k_query_prep(PrepArgs a) {
  extern __shared__ float qs[];
  __shared__ float s_paa;
  const uint32_t slot = blockIdx.x;
  const float* q = a.q + (uint64_t)slot * a.L;
  for (int i = threadIdx.x; i < a.L; i += kPrepThreads) qs[i] = q[i];
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (blockIdx.y == gridDim.y - 1) {
    if (!a.approx_leaf || warp != 0) return;
    if (lane < 8) a.counters[8 * slot + lane] = 0;
    for (int i = lane; i < kMaxK; i += 32) a.kslots[slot * kMaxK + i] = 0x7f800000u;  // +inf
    const int leaf = warp_route(qs, a.tree);
    if (lane == 0) {
      a.approx_leaf[slot] = leaf;
      a.bound[slot] = 0x7f800000u;  // +inf
      a.topk_count[slot] = 0;
    }
    return;
  }
  if (a.sax_tab && blockIdx.y < HG_PAA_SEGMENTS) {
    // paa_from_ts (sax.c:46-56): a sequential sum, one division
    const int t = blockIdx.y, per = a.L / HG_PAA_SEGMENTS;
    if (threadIdx.x == 0) {
      float acc = 0.0f;
#pragma unroll 8
      for (int i = 0; i < per; ++i) acc = __fadd_rn(acc, qs[t * per + i]);
      s_paa = __fdiv_rn(acc, (float)per);
    }
    __syncthreads();
    static_assert(kPrepThreads == HG_SAX_CARD, "a thread per symbol");
    a.sax_tab[(uint64_t)slot * (HG_PAA_SEGMENTS * HG_SAX_CARD) + t * HG_SAX_CARD + threadIdx.x] =
        hg_lb_sax_lane(s_paa, threadIdx.x, a.bp);
  }
  if (!a.lb) return;
  for (int w = blockIdx.y * (kPrepThreads / 32) + warp; w < a.nleaves; w += (gridDim.y - 1) * (kPrepThreads / 32)) {
    const int off = a.seg_off[w], nseg = a.seg_off[w + 1] - off;
    float sum = 0.0f;
    int start = 0;
    for (int s = 0; s < nseg; ++s) {
      const int end = a.points[off + s];
      float m, sd;
      warp_mean_stdev(qs, start, end, &m, &sd);
      sum = __fadd_rn(sum, hg_eapca_term(m, sd, a.sk + 4 * (off + s), end - start));
      start = end;
    }
    if (lane == 0) a.lb[(uint64_t)slot * a.nleaves + w] = sum;
  }
}

// Mean and stdev of every query over every distinct leaf segment (leaves
// share most of their segments: a split refines its parent's), with the
// reference arithmetic of calculate_node_min_distance's calc_mean_stdev_SIMD:
// one block per query, a warp per segment (warp_mean_stdev for segments of 64
// points or more, else hg_mean_stdev on one lane).  out[q * nu + u].
__global__ void k_query_segstats(const float* __restrict__ Q, int L, int nq, const short* __restrict__ useg_start,
                                 const short* __restrict__ useg_end, int nu, float2* __restrict__ out) {
  extern __shared__ float qs[];
  const int q = blockIdx.x;
  if (q >= nq) return;
  for (int i = threadIdx.x; i < L; i += blockDim.x) qs[i] = Q[(uint64_t)q * L + i];
  __syncthreads();
  const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  for (int u = threadIdx.x >> 5; u < nu; u += nw) {
    const int start = useg_start[u], end = useg_end[u];
    float m, sd;
    if (end - start >= 64) {
      warp_mean_stdev(qs, start, end, &m, &sd);
    } else {
      hg_mean_stdev(qs, start, end, &m, &sd);  // every lane, the same values
    }
    if (lane == 0) out[(uint64_t)q * nu + u] = make_float2(m, sd);
  }
}

// Leaves each query of a batch must filter: a thread per (query, leaf) sums
// the LB_EAPCA terms of the leaf's segments in order (the plain path's
// k_query_prep arithmetic, segment statistics from k_query_segstats; the terms
// are >= 0, so the sum stops once it exceeds the limit) and keeps the leaf
// when
//     LB <= B_q (1 + 2^-10) + L 2^-20,
// B_q the query's bound (+inf keeps every leaf).  The plain path scans only
// leaves with LB <= its running bound <= B_q, so the kept leaves include
// every leaf it scans; the margins cover the rounding of B_q's product.
// Kept (leaf, query) pairs go to leaf_q[leaf * stride + i], counted in
// leaf_cnt[leaf].
// qlist (optional): the queries are qlist[0 .. *nq_dev) instead of 0 .. nq.
// A thread per (query, leaf) pair, grid-stride (a warp per pair, with the
// sum's order kept through shuffles, made the bound phase 0.33 ms longer per
// batch of 4,096 queries at 25M x 256).
__global__ void k_leaf_keep(const float2* __restrict__ segstats, int nu, int L, int nq,
                            const int* __restrict__ seg_off, const short* __restrict__ points,
                            const int* __restrict__ seg_uid, const float* __restrict__ sk,
                            const uint32_t* __restrict__ leaf_size, int nleaves, const float* __restrict__ bound,
                            uint32_t* leaf_cnt, uint32_t* leaf_q, uint32_t stride, const uint32_t* qlist,
                            const uint32_t* nq_dev) {
  const uint64_t n = (uint64_t)(nq_dev ? min((uint32_t)nq, *nq_dev) : (uint32_t)nq) * nleaves;
  const uint64_t nt = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t g = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; g < n; g += nt) {
    const int qi = (int)(g / nleaves), w = (int)(g % nleaves);
    const int q = qlist ? (int)qlist[qi] : qi;
    if (leaf_size[w] == 0) continue;
    const float B = bound[q];
    const float lim = B < __int_as_float(0x7f800000)
                          ? __fadd_ru(__fmul_ru(B, 1.0f + 0x1p-10f), __fmul_ru((float)L, 0x1p-20f))
                          : __int_as_float(0x7f800000);
    const int off = seg_off[w], nseg = seg_off[w + 1] - off;
    const float2* st = segstats + (uint64_t)q * nu;
    float sum = 0.0f;
    int start = 0;
    for (int s = 0; s < nseg; ++s) {
      const int end = points[off + s];
      const float2 ms = st[seg_uid[off + s]];
      sum = __fadd_rn(sum, hg_eapca_term(ms.x, ms.y, sk + 4 * (off + s), end - start));
      start = end;
      if (!(sum <= lim)) break;
    }
    if (sum <= lim) leaf_q[(uint64_t)w * stride + atomicAdd(&leaf_cnt[w], 1u)] = (uint32_t)q;
  }
}

// Candidate leaves: LB_EAPCA <= current bound, not the approximate leaf, not
// empty; ordered by LB with a stable LSD radix sort (4-bit digits, 8 passes)
// in one CTA; then the exclusive prefix of their tile counts.
constexpr int kSortThreads = 1024;
__device__ void select_sort(const SelectArgs& a, uint32_t slot, float B, uint32_t* sm) {
  const int nleaves = a.nleaves;
  const float* __restrict__ lb = a.lb + (uint64_t)slot * nleaves;
  const uint64_t* __restrict__ leaf_start = a.leaf_start;
  const uint32_t* __restrict__ leaf_size = a.leaf_size;
  int* cand = a.cand + (uint64_t)slot * (nleaves + 1);
  float* cand_lb = a.cand_lb + (uint64_t)slot * (nleaves + 1);
  uint32_t* unit_prefix = a.unit_prefix + (uint64_t)slot * (nleaves + 2);
  // keys and values (two buffers each) live in shared memory up to
  // kMaxLeavesSort leaves, else in gkeys (4 x nleaves words of global memory)
  uint32_t* gkeys = a.gkeys ? a.gkeys + (uint64_t)slot * 4 * nleaves : nullptr;
  uint32_t* cnt = sm;  // 16 x kSortThreads digit counts
  uint32_t* kbase = gkeys ? gkeys : sm + 16 * kSortThreads;
  const int cap = gkeys ? nleaves : kMaxLeavesSort;
  uint32_t* keys0 = kbase;
  uint32_t* vals0 = keys0 + cap;
  uint32_t* keys1 = vals0 + cap;
  uint32_t* vals1 = keys1 + cap;
  __shared__ uint32_t tmp[kSortThreads / 32 + 1];
  __shared__ uint32_t total;
  const int t = threadIdx.x;
  const int approx = a.approx_leaf[slot];
  // 1. select the non-empty leaves within the bound, the approximate leaf
  //    excepted (it was scanned first), order preserving
  const int per = (nleaves + kSortThreads - 1) / kSortThreads;
  const int b0 = min(nleaves, t * per), b1 = min(nleaves, b0 + per);
  uint32_t mine = 0;
  for (int i = b0; i < b1; ++i) {
    const float l = lb[i];
    if (leaf_size[i] > 0 && i != approx && !(l > B)) ++mine;
  }
  uint32_t pos = block_exclusive_scan<kSortThreads>(mine, tmp, &total);
  const int n = (int)total;
  for (int i = b0; i < b1; ++i) {
    const float l = lb[i];
    if (leaf_size[i] > 0 && i != approx && !(l > B)) {
      keys0[pos] = (l == l) ? __float_as_uint(l) : 0u;  // a NaN bound never prunes
      vals0[pos] = (uint32_t)i;
      ++pos;
    }
  }
  __syncthreads();
  // 2. sort by LB, unless the leaves may stay in file order (by_file, all of
  //    them within a finite bound, so none is met that ends the list: their
  //    LBs read 0).  Up to kSortThreads candidates (the usual case): one
  //    bitonic sort of (LB bits, leaf) keys; the leaves are in index order on
  //    input, so equal LBs end in the order the stable radix sort below gives
  //    them, which handles larger counts.
  const int per2 = (n + kSortThreads - 1) / kSortThreads;
  const int r0 = min(n, t * per2), r1 = min(n, r0 + per2);
  uint32_t *ki = keys0, *vi = vals0, *ko = keys1, *vo = vals1;
  const bool by_file = a.by_file && B < __int_as_float(0x7f800000);
  if (by_file) {
    for (int i = t; i < n; i += kSortThreads) keys0[i] = 0;
    __syncthreads();
  } else if (n <= kSortThreads) {
    unsigned long long* kv = reinterpret_cast<unsigned long long*>(keys1);  // 8-byte aligned, 2 x cap words (n <= 1024)
    int np = 2;
    while (np < n) np <<= 1;
    for (int i = t; i < np; i += kSortThreads)
      kv[i] = i < n ? (((unsigned long long)keys0[i] << 32) | vals0[i]) : ~0ull;
    __syncthreads();
    for (int size = 2; size <= np; size <<= 1)
      for (int stride = size >> 1; stride > 0; stride >>= 1) {
        for (int i = t; i < np / 2; i += kSortThreads) {
          const int pos = 2 * i - (i & (stride - 1));
          const int partner = pos + stride;
          const bool asc = (pos & size) == 0;
          const unsigned long long x = kv[pos], y = kv[partner];
          if ((x > y) == asc) {
            kv[pos] = y;
            kv[partner] = x;
          }
        }
        __syncthreads();
      }
    for (int i = t; i < n; i += kSortThreads) {
      keys0[i] = (uint32_t)(kv[i] >> 32);
      vals0[i] = (uint32_t)kv[i];
    }
    __syncthreads();
  }
  for (int pass = 0; !by_file && n > kSortThreads && pass < 8; ++pass) {
    const int shift = pass * 4;
    uint32_t c[16];
#pragma unroll
    for (int d = 0; d < 16; ++d) c[d] = 0;
    for (int i = r0; i < r1; ++i) ++c[(ki[i] >> shift) & 15];
    // flattened digit-major counts: index d * kSortThreads + t; scan them in
    // that order (thread t owns the 16 entries t*16 .. t*16+15 of the flat array)
#pragma unroll
    for (int d = 0; d < 16; ++d) cnt[d * kSortThreads + t] = c[d];
    __syncthreads();
    uint32_t s = 0;
    uint32_t loc[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      loc[j] = s;
      s += cnt[t * 16 + j];
    }
    const uint32_t base = block_exclusive_scan<kSortThreads>(s, tmp, nullptr);
#pragma unroll
    for (int j = 0; j < 16; ++j) cnt[t * 16 + j] = base + loc[j];
    __syncthreads();
    uint32_t off[16];
#pragma unroll
    for (int d = 0; d < 16; ++d) off[d] = cnt[d * kSortThreads + t];
    for (int i = r0; i < r1; ++i) {
      const int d = (ki[i] >> shift) & 15;
      const uint32_t p = off[d]++;
      ko[p] = ki[i];
      vo[p] = vi[i];
    }
    __syncthreads();
    uint32_t* x = ki;
    ki = ko;
    ko = x;
    x = vi;
    vi = vo;
    vo = x;
  }
  // 3. outputs and tile prefix
  uint32_t tiles = 0, rows = 0;
  for (int i = r0; i < r1; ++i) {
    const int leaf = (int)vi[i];
    rows += leaf_size[leaf];
    cand[i] = leaf;
    cand_lb[i] = __uint_as_float(ki[i]);
    tiles += tiles_of_leaf(leaf_start[leaf], leaf_size[leaf]);
  }
  uint32_t tp = block_exclusive_scan<kSortThreads>(tiles, tmp, &total);
  for (int i = r0; i < r1; ++i) {
    const int leaf = (int)vi[i];
    unit_prefix[i] = tp;
    tp += tiles_of_leaf(leaf_start[leaf], leaf_size[leaf]);
  }
  if (a.row_prefix) {
    uint32_t* row_prefix = a.row_prefix + (uint64_t)slot * (nleaves + 2);
    if (t == 0) unit_prefix[n] = total;
    uint32_t rp = block_exclusive_scan<kSortThreads>(rows, tmp, &total);
    for (int i = r0; i < r1; ++i) {
      row_prefix[i] = rp;
      rp += leaf_size[vi[i]];
    }
    if (t == 0) row_prefix[n] = total;
  } else if (t == 0) {
    unit_prefix[n] = total;
  }
  if (t == 0) {
    a.cand_count[slot] = n;
  }
}

__global__ void k_pscan_prep(uint32_t* bound, uint32_t* kslots, int* topk_count) {
  const int slot = blockIdx.x;
  for (int i = threadIdx.x; i < kMaxK; i += blockDim.x) kslots[slot * kMaxK + i] = 0x7f800000u;  // +inf
  if (threadIdx.x == 0) {
    bound[slot] = 0x7f800000u;
    topk_count[slot] = 0;
  }
}

// ---------------------------------------------------------------------------
// The leaf scan (exact_de_knn_search's refine loop, hercules_query_engine.c:
// 2391-2425, with the per-row LB_SAX test of the reference's SIMS path,
// :2183-2211) runs as two kernels: a streaming LB_SAX filter that turns the
// candidate leaves into a compact list of surviving rows, and a distance
// stream over that list.
// ---------------------------------------------------------------------------

// Stage 1.  Work: the candidate leaves (file order, or ascending LB_EAPCA:
// select_sort), cut into
// 32-row units (32-aligned rows; a unit's rows outside its leaf are skipped).
// One persistent block per SM owns a contiguous range of units, ending at the
// first leaf whose LB exceeds the bound (found by the producer warp while
// the consumers build the table).  Its producer lane bulk-copies the
// units' iSAX words (a leaf's units are contiguous in memory: one
// cp.async.bulk per leaf run, 512 bytes per unit) into kFiltStages stages of
// shared memory, each guarded by a full and an empty mbarrier; 20 consumer
// warps take 3 units of every stage each (lane = row), test the rows from
// shared memory and append the survivors with one atomicAdd per warp and
// stage.  Every wait is bounded: on timeout the block raises *err, the
// producer drains the copies it issued, and the call reports HG_ERR_TIMEOUT.
//
// The per-row test is a certified lower bound of the reference's LB_SAX
// (minidist_paa_to_isax_raw_SIMD, sax.c:310-479).  The query's 16 x 256
// table of per-segment terms (k_query_prep, reference arithmetic) is turned,
// per block, into 8-bit terms q = floor(term * 254 / T) (rounded down at
// every step, at most 255) against the pruning threshold
// T = (B (1 + 2^-10) + 1e-6) / (L / 16); a row is pruned when its 16 terms
// add up to at least 255, which implies (L / 16) * (sum of the terms) >=
// (255 / 254) (B (1 + 2^-10) + 1e-6): the reference's float LB_SAX exceeds
// the bound with room to spare for its rounding, so every row this test
// prunes is one the exact float test prunes too (never a true neighbour).
// The 8-bit table is laid out lane-private: byte b of word
// ((h * 256 + s) * 2 + g) * 32 + lane holds that lane's term of symbol s for
// segment t = 8 h + 4 g + b, so the byte of (t, s) sits at
// (t / 8) * 65536 + ((t / 4) & 1) * 128 + (t & 3) + 256 s + 4 lane: the 16
// data-dependent lookups of a row never conflict on a bank, and one byte
// permute of the row's word and 4 lane gives each lookup's address.
constexpr int kFiltConsumers = 20;                          // consumer warps
constexpr int kFilterThreads = 32 * (kFiltConsumers + 1);   // + the producer warp
constexpr int kUnitsPerWarp = 3;                            // units of a stage per consumer warp
constexpr int kStageUnits = kFiltConsumers * kUnitsPerWarp; // 60 units: 30 KB
constexpr int kFiltStages = 3;
constexpr uint32_t kUnitBytes = 32 * 16;
constexpr uint32_t kStageBytes = kStageUnits * kUnitBytes;
constexpr int kSaxTabWords = HG_PAA_SEGMENTS * HG_SAX_CARD / 4 * 32;  // 128 KB
constexpr uint32_t kFiltSmStage = kSaxTabWords * 4;                     // stages after the table
constexpr uint32_t kFiltSmBar = kFiltSmStage + kFiltStages * kStageBytes;  // 2 x kFiltStages mbarriers
constexpr uint32_t kFiltSmMeta = kFiltSmBar + 2 * kFiltStages * 8;  // end unit, abort flag, first candidate
constexpr uint64_t kFiltWaitNs = 2000000000ull;                           // 2 s per wait
size_t lbsax_filter_smem() { return kFiltSmMeta + 16; }

__device__ __forceinline__ uint32_t sax_qterm(float term, float scale) {
  const float p = __fmul_rd(term, scale);
  return p >= 255.0f ? 255u : (uint32_t)p;
}

__device__ __forceinline__ bool fl_try(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ uint64_t fl_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
// Bounded wait for the phase of `parity`: false when the block aborted or
// the wait ran out (then the block aborts and *err is raised).
__device__ __noinline__ bool fl_wait_slow(uint32_t bar, uint32_t parity, volatile int* abort_flag, int* err) {
  const uint64_t t0 = fl_ns();
  for (uint32_t i = 1;; ++i) {
    if (fl_try(bar, parity)) return true;
    if ((i & 63) == 0) {
      if (*abort_flag) return false;
      if (fl_ns() - t0 > kFiltWaitNs) {
        *abort_flag = 1;
        if (err) atomicExch(err, 1);
        return false;
      }
    }
  }
}

// the first test inline, the polling loop out of line
__device__ __forceinline__ bool fl_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag, int* err) {
  return fl_try(bar, parity) || fl_wait_slow(bar, parity, abort_flag, err);
}

// The launch's arguments moved to the block's query, and the units [ubase,
// ubase + total) of its candidates [clo, chi) (all of them by default).
__device__ __forceinline__ void filter_range(FilterArgs& a, int& ncand, int& clo, int& chi, uint32_t& ubase,
                                             uint32_t& total) {
  const uint32_t slot = blockIdx.x;
  a.cand += (uint64_t)slot * (a.nleaves + 1);
  a.cand_lb += (uint64_t)slot * (a.nleaves + 1);
  a.unit_prefix += (uint64_t)slot * (a.nleaves + 2);
  a.row_prefix += (uint64_t)slot * (a.nleaves + 2);
  a.sax_tab += (uint64_t)slot * (HG_PAA_SEGMENTS * HG_SAX_CARD);
  a.bound += slot;
  a.list += (uint64_t)slot * a.list_stride;
  a.list_count += 8 * slot;
  ncand = a.cand_count[slot];
  clo = min(a.cand_lo, ncand);
  chi = a.cand_hi > 0 ? min(a.cand_hi, ncand) : ncand;
  ubase = clo < chi ? a.unit_prefix[clo] : 0u;
  total = clo < chi ? a.unit_prefix[chi] - ubase : 0u;
}

// Stage 1 without LB_SAX: every row of the leaves within the bound, in LB
// order (a row's place in the list is its leaf's row prefix plus its place in
// the leaf).  A warp lists a contiguous range of units, at least kListUnits of
// them; the one that meets the last leaf within the bound writes the count.
// Bound by its stores, 4 bytes per row: 16 queries of 8M x 256, 56.5M rows,
// 57 us; the LB_SAX filter's kernel, which did this too, took 332 us (one block
// of 21 warps per SM, the words copied and not read, an atomicAdd per 96 rows),
// and its list, in no order, made the scan behind it slower (100 queries of
// 1M x 256: 5.79 ms per call, now 5.38; 12 of 100k x 16384 3.99, now 3.71).
constexpr int kListWarps = 8, kListUnits = 8;
__global__ void __launch_bounds__(32 * kListWarps) k_list_rows(FilterArgs a) {
  int ncand, clo, chi;
  uint32_t ubase, total;
  filter_range(a, ncand, clo, chi, ubase, total);
  const uint32_t lane = threadIdx.x & 31, w = blockIdx.y * kListWarps + (threadIdx.x >> 5);
  const uint32_t nwarps = gridDim.y * kListWarps;
  const uint32_t per_warp = max((uint32_t)kListUnits, (total + nwarps - 1) / nwarps);
  if ((uint64_t)w * per_warp >= total) return;
  const uint32_t u0 = ubase + w * per_warp, u1 = min(ubase + total, u0 + per_warp);
  const float B = __int_as_float((int)ld_volatile(a.bound));
  const uint32_t base = a.row_prefix[clo];
  uint32_t n_leaves = 0;
  for (int c = unit_candidate_warp(a.unit_prefix, ncand, clo, u0, (int)lane); c < chi; ++c) {
    const uint32_t first_unit = a.unit_prefix[c], next = a.unit_prefix[c + 1];
    if (first_unit >= u1 || a.cand_lb[c] > B) break;  // LBs ascend: no later leaf is within the bound
    const uint32_t from = max(u0, first_unit), to = min(u1, next);
    n_leaves += from == first_unit ? 1u : 0u;
    const int leaf = a.cand[c];
    const uint32_t lstart = (uint32_t)a.leaf_start[leaf], lend = lstart + a.leaf_size[leaf];
    uint32_t* out = a.list + (a.row_prefix[c] - base);
    const uint32_t row1 = min(lend, ((lstart >> 5) + (to - first_unit)) << 5);
#pragma unroll 4
    for (uint32_t r = (((lstart >> 5) + (from - first_unit)) << 5) + lane; r < row1; r += 32)
      if (r >= lstart) out[r - lstart] = r;
    if (to == next && (c + 1 == chi || a.cand_lb[c + 1] > B) && lane == 0) {
      const uint32_t count = a.row_prefix[c + 1] - base;
      *a.list_count = count;
      atomicAdd(&a.stats[0], (unsigned long long)count);
    }
  }
  if (lane == 0 && n_leaves) atomicAdd(&a.stats[3], (unsigned long long)n_leaves);
}

__global__ void __launch_bounds__(kFilterThreads, 1) k_lbsax_filter(FilterArgs a) {
  extern __shared__ __align__(16) unsigned char fsm[];
  uint32_t* qtab = reinterpret_cast<uint32_t*>(fsm);
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(fsm);
  auto full_bar = [&](int st) { return sbase + kFiltSmBar + 8u * st; };
  auto empty_bar = [&](int st) { return sbase + kFiltSmBar + 8u * (kFiltStages + st); };
  volatile uint32_t* s_uend = reinterpret_cast<volatile uint32_t*>(fsm + kFiltSmMeta);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(fsm + kFiltSmMeta + 4);
  int ncand, clo, chi;
  uint32_t ubase, total;
  filter_range(a, ncand, clo, chi, ubase, total);
  const float B = __int_as_float((int)ld_volatile(a.bound));
  // at least one full stage per block: fewer units leave blocks without a
  // range, which return before they build a table
  const uint32_t per_block = max((uint32_t)kStageUnits, (total + gridDim.y - 1) / gridDim.y);
  if ((uint64_t)blockIdx.y * per_block >= total) return;
  const uint32_t u0 = ubase + blockIdx.y * per_block;
  const uint32_t u1 = min(ubase + total, u0 + per_block);
  volatile int* s_c0 = reinterpret_cast<volatile int*>(fsm + kFiltSmMeta + 8);
  if (wib == kFiltConsumers) {
    // the producer warp finds the block's first candidate and where its
    // range ends -- at the first leaf whose LB exceeds the bound (LBs ascend
    // along the list, so every later unit is past it too) -- with 32-way
    // searches, sets up the barriers and hands both to the consumers
    // through named barrier 1, while they build the table
    int c0 = clo;
    uint32_t ue = u0;
    if (u0 < u1) {
      c0 = unit_candidate_warp(a.unit_prefix, ncand, clo, u0, lane);
      ue = u1;
      for (int cb = c0; cb < chi; cb += 32) {
        const int c = cb + lane;
        const bool in_range = c < chi && a.unit_prefix[c] < u1;
        const uint32_t past = __ballot_sync(HG_FULL, in_range && a.cand_lb[c] > B);
        if (past) {
          ue = max(u0, a.unit_prefix[cb + __ffs(past) - 1]);
          break;
        }
        if (!__all_sync(HG_FULL, in_range)) break;
      }
    }
    if (lane == 0) {
      *s_uend = ue;
      *s_c0 = c0;
      *abort_flag = 0;
      for (int st = 0; st < kFiltStages; ++st) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(full_bar(st)), "r"(1) : "memory");
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(empty_bar(st)), "r"(kFiltConsumers) : "memory");
      }
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();
    asm volatile("bar.arrive 1, %0;" ::"r"(kFilterThreads) : "memory");
  } else {
    const float Bs = __fadd_rn(__fmul_rn(B, 1.0009765625f), 1e-6f);
    const float T = __fdiv_ru(Bs, (float)(a.L / HG_PAA_SEGMENTS));
    const float scale = __fdiv_rd(254.0f, T);  // 0 when the bound is +inf: nothing is pruned
    for (int g = threadIdx.x; g < kSaxTabWords / 32; g += 32 * kFiltConsumers) {
      // the terms of symbol s for segments t0 .. t0 + 3
      const int sym = (g >> 1) & (HG_SAX_CARD - 1), t0 = 8 * (g >> 9) + 4 * (g & 1);
      const float* col = a.sax_tab + t0 * HG_SAX_CARD + sym;
      const uint32_t packed = sax_qterm(col[0], scale) | (sax_qterm(col[HG_SAX_CARD], scale) << 8) |
                              (sax_qterm(col[2 * HG_SAX_CARD], scale) << 16) |
                              (sax_qterm(col[3 * HG_SAX_CARD], scale) << 24);
#pragma unroll 8
      for (int r = 0; r < 32; ++r) qtab[g * 32 + ((r + lane) & 31)] = packed;
    }
  }
  if (wib != kFiltConsumers) asm volatile("bar.sync 1, %0;" ::"r"(kFilterThreads) : "memory");
  const uint32_t uend = *s_uend;
  const int c0 = *s_c0;
  const uint32_t nstages = (uend - u0 + kStageUnits - 1) / kStageUnits;  // 0 when u0 == uend
  if (wib == kFiltConsumers) {
    // ---------------- producer: bulk copies of whole units, leaf by leaf
    if (lane == 0 && nstages) {
      int c = c0;
      uint32_t k = 0;
      bool ok = true;
      for (; k < nstages; ++k) {
        const int st = (int)(k % kFiltStages);
        ok = fl_wait(empty_bar(st), ((k / kFiltStages) & 1) ^ 1, abort_flag, a.err);
        if (!ok) break;
        const uint32_t us = u0 + k * kStageUnits, ue = min(uend, us + kStageUnits);
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(full_bar(st)),
                     "r"((ue - us) * kUnitBytes)
                     : "memory");
        for (uint32_t u = us; u < ue;) {
          while (c + 1 < ncand && a.unit_prefix[c + 1] <= u) ++c;
          const uint32_t run_end = min(ue, c + 1 < ncand ? a.unit_prefix[c + 1] : ue);
          const uint64_t first_row = ((a.leaf_start[a.cand[c]] >> 5) + (u - a.unit_prefix[c])) << 5;
          const unsigned char* src = a.sax + first_row * 16;
          const uint32_t dst = sbase + kFiltSmStage + (uint32_t)st * kStageBytes + (u - us) * kUnitBytes;
          asm volatile(
              "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
              "l"(reinterpret_cast<uint64_t>(src)), "r"((run_end - u) * kUnitBytes), "r"(full_bar(st))
              : "memory");
          u = run_end;
        }
      }
      // leaving early: the copies in flight land before the block exits
      if (!ok) {
        const uint32_t first = k > (uint32_t)kFiltStages ? k - kFiltStages : 0u;
        for (uint32_t kk = first; kk < k; ++kk) {
          const uint64_t t0 = fl_ns();
          while (!fl_try(full_bar((int)(kk % kFiltStages)), (kk / kFiltStages) & 1) && fl_ns() - t0 < kFiltWaitNs) {
          }
        }
      }
    }
  } else {
    // ---------------- consumers: lane = row of a unit
    const unsigned char* tb = fsm;
    const uint32_t lanev = (uint32_t)(4 * lane);  // byte 0: 4 lane, bytes 1..3: zero
    const uint32_t lt = (1u << lane) - 1;
    int c = c0;  // the body moves it forward to each unit's candidate
    uint32_t next_c = c + 1 < ncand ? a.unit_prefix[c + 1] : 0xffffffffu;
    int cur = -1;
    uint32_t lstart = 0, lend = 0, first_unit = 0;
    uint32_t n_rows = 0, n_pass = 0, n_leaves = 0;  // lane 0's counts
    for (uint32_t k = 0; k < nstages; ++k) {
      const int st = (int)(k % kFiltStages);
      int got = 1;
      if (lane == 0) got = fl_wait(full_bar(st), (k / kFiltStages) & 1, abort_flag, a.err) ? 1 : 0;
      if (!__shfl_sync(HG_FULL, got, 0)) break;
      const uint32_t us = u0 + k * kStageUnits, ue = min(uend, us + kStageUnits);
      const uint4* stage = reinterpret_cast<const uint4*>(fsm + kFiltSmStage + st * kStageBytes);
      uint32_t m[kUnitsPerWarp], rr[kUnitsPerWarp];
      uint32_t cnt = 0;
#pragma unroll
      for (int i = 0; i < kUnitsPerWarp; ++i) {
        const uint32_t slot = (uint32_t)(wib * kUnitsPerWarp + i), unit = us + slot;
        m[i] = 0;
        rr[i] = 0;
        if (unit >= ue) continue;  // uniform over the warp
        while (unit >= next_c) {
          ++c;
          next_c = c + 1 < ncand ? a.unit_prefix[c + 1] : 0xffffffffu;
        }
        if (c != cur) {
          cur = c;
          const int leaf = a.cand[c];
          lstart = (uint32_t)a.leaf_start[leaf];
          lend = lstart + a.leaf_size[leaf];
          first_unit = a.unit_prefix[c];
        }
        const uint32_t tile_in = unit - first_unit;
        n_leaves += tile_in == 0 ? 1u : 0u;
        rr[i] = (((lstart >> 5) + tile_in) << 5) + lane;
        bool pass = rr[i] >= lstart && rr[i] < lend;
        n_rows += (uint32_t)__popc(__ballot_sync(HG_FULL, pass));
        if (pass) {
          // byte j of word q is the symbol s of segment t = 4 q + j; the
          // permute puts s in byte 1 and 4 lane in byte 0: 256 s + 4 lane,
          // the lookup's offset from segment t's fixed base
          const uint4 w = stage[slot * 32 + lane];
          const uint32_t ws[4] = {w.x, w.y, w.z, w.w};
          uint32_t sum = 0;
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const int tq = (q >> 1) * 65536 + (q & 1) * 128;
            sum += (uint32_t)tb[tq + __byte_perm(ws[q], lanev, 0x5504)] +
                   (uint32_t)tb[tq + 1 + __byte_perm(ws[q], lanev, 0x5514)] +
                   (uint32_t)tb[tq + 2 + __byte_perm(ws[q], lanev, 0x5524)] +
                   (uint32_t)tb[tq + 3 + __byte_perm(ws[q], lanev, 0x5534)];
          }
          pass = sum < 255u;
        }
        m[i] = __ballot_sync(HG_FULL, pass);
        cnt += (uint32_t)__popc(m[i]);
      }
      // the stage's words are read: hand it back to the producer
      __syncwarp();
      if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(empty_bar(st)) : "memory");
      n_pass += cnt;
      uint32_t pos = 0;
      if (lane == 0 && cnt) pos = atomicAdd(a.list_count, cnt);
      pos = __shfl_sync(HG_FULL, pos, 0);
#pragma unroll
      for (int i = 0; i < kUnitsPerWarp; ++i) {
        if ((m[i] >> lane) & 1u) a.list[pos + __popc(m[i] & lt)] = rr[i];
        pos += __popc(m[i]);
      }
    }
    // rows considered, pruned (considered minus survivors) and leaves visited
    if (lane == 0) {
      atomicAdd(&a.stats[0], (unsigned long long)n_rows);
      atomicAdd(&a.stats[2], (unsigned long long)(n_rows - n_pass));
      atomicAdd(&a.stats[3], (unsigned long long)n_leaves);
    }
  }
}

// Stage 2: the early-abandoning squared distance (ts_euclidean_distance_SIMD,
// ts.c:83-109) over a row list, or over a row range when there is no list.
//
// A warp works on 8 rows at a time, 4 lanes per row ("slot"; wider slots for
// long series).  Per step the lanes of a slot load kLines lines of their row
// (chunk ch + j of a line in lane j), each computes its 8-float chunk sums, and
// the slot adds them to the running distance in chunk order (shuffles) and
// tests the bound once (a strict test: a row whose distance equals the bound
// finishes, so ties keep the lowest id).  A slot whose row abandoned or
// finished takes the next row of its warp's batch: warp w of W owns the
// batches w, w + W, w + 2W, ... of the list (up to 32 entries each), and the
// next batch's entries are loaded while the current one is consumed.  Finished rows within the bound enter
// the warp's top-k list, which lowers the global bound (atomicMin) once it
// holds k distances.  The query lives in shared memory in blocks of 32
// chunks (40 float4 pairs each): chunk r of a block sits at pair r + r / 4,
// so the slots of a warp, which sit at different 4-chunk positions, read
// different banks.
__device__ __forceinline__ int q4_index(int chunk, int half) {
  const int r = chunk & 31;
  return ((chunk >> 5) * 40 + r + (r >> 2)) * 2 + half;
}
// bytes of that layout for a series of L floats
__host__ __device__ inline size_t q4_bytes(int L) { return (size_t)((L / 8 + 31) / 32) * 40 * 2 * 16; }
// What this block scans: the launch's arguments moved to its query and list,
// the rows' first index and count.  False when nothing falls to the block (its
// list is then empty).
template <int W>
__device__ __forceinline__ bool ed_range(EdArgs& a, uint64_t& first, uint32_t& total, uint32_t& bs) {
  const uint32_t qslot = blockIdx.x;  // the query of the group
  a.bound += qslot;
  a.kslots += (uint64_t)qslot * kMaxK;
  a.parts += ((uint64_t)qslot * a.parts_stride + blockIdx.y) * kWarpListCap;
  a.part_count += (uint64_t)qslot * a.parts_stride + blockIdx.y;
  a.q += (uint64_t)qslot * a.L;
  if (a.list) a.list += (uint64_t)qslot * a.list_stride;
  first = a.ident_first;
  if (a.gate && *a.gate == 0) {
    total = 0;  // a gated launch that did not pass
  } else if (a.list) {
    total = a.list_count[8 * qslot];
  } else if (a.ident_leaf) {
    const int leaf = a.ident_leaf[qslot];
    first = a.leaf_start[leaf];
    total = a.leaf_size[leaf];
  } else {
    total = (uint32_t)a.ident_count;
  }
  // warp w of the launch takes entries [(w + b nwarps) bs, +bs), b = 0, 1, ..:
  // bs spreads a short list over the warps, at least min_batch entries each
  const uint32_t nwarps = gridDim.y * W;
  const uint32_t per_warp = (uint32_t)(((uint64_t)total + nwarps - 1) / nwarps);
  bs = per_warp < a.min_batch ? a.min_batch : (per_warp > 32u ? 32u : per_warp);
  if ((uint64_t)blockIdx.y * W * bs < total) return true;
  if (threadIdx.x == 0) *a.part_count = 0;
  return false;
}

// The running bound of a scan.  A warp's own k-th distance is a poor bound: a
// warp sees a few hundred rows, and the least of 4,736 warps' 10th distances
// after 16 rows each is at the 17% quantile.  So the query also has k slots:
// a finished row's distance goes to slot hash(distance) with a minimum, equal
// distances share a slot, so k filled slots hold k distinct distances, and
// their maximum bounds the k-th distinct distance of all rows finished so far
// on the GPU (about three times its quantile).  Each block keeps a copy in
// shared memory; a warp exchanges it with the global slots when it kept a row
// and in every 16th turn (rarer with more warps per block and more than 32
// slots), its block mates in others: a word that every warp reads in every turn keeps its L2 slice busy
// longer than a scan of 2M rows takes.  Against bounds from the warps' own
// lists alone, one query: PSCAN of 2M x 256 329 -> 230 us, of 1M x 512 429 ->
// 269 us, the allocation-free scan of 1M x 256 200 -> 126 us.
struct EdShared {
  uint32_t bound;
  uint32_t slot[kMaxK];
};
__device__ __forceinline__ void ed_shared_init(const EdArgs& a, EdShared& sh, int threads) {
  for (int i = threadIdx.x; i < a.k; i += threads) sh.slot[i] = 0x7f800000u;
  if (threadIdx.x == 0) sh.bound = ld_volatile(a.bound);
}
__device__ __noinline__ void ed_exchange(uint32_t* gslot, uint32_t* gbound, int k, EdShared* sh) {
  const int lane = threadIdx.x & 31;
  const uint32_t gb = ld_volatile(gbound);
  uint32_t most = 0;
  for (int i = lane; i < k; i += 32) {
    const uint32_t g = ld_volatile(gslot + i), s = ld_volatile(&sh->slot[i]);
    if (s < g) atomicMin(gslot + i, s);
    else if (g < s) atomicMin(&sh->slot[i], g);
    most = max(most, min(g, s));
  }
  most = __reduce_max_sync(HG_FULL, most);
  if (lane == 0) {
    if (most < gb) atomicMin(gbound, most);
    atomicMin(&sh->bound, min(most, gb));
  }
  __syncwarp();
}
// after a turn's finished rows (take, dist) are in the list: the bound to go on with
__device__ __forceinline__ float ed_bound(const EdArgs& a, EdShared& sh, uint32_t turn, bool take, float dist, float B,
                                          float T) {
  if (take) {
    const uint32_t bits = __float_as_uint(dist);
    atomicMin(&sh.slot[__umulhi(bits * 2654435761u, (uint32_t)a.k)], bits);
  }
  if (__any_sync(HG_FULL, take) || ((turn + 2 * (threadIdx.x >> 5)) & (a.period - 1)) == 0) {
    __syncwarp();
    ed_exchange(a.kslots, a.bound, a.k, &sh);
  }
  return fminf(fminf(B, T), __uint_as_float(ld_volatile(&sh.bound)));
}

// The block's warp lists (each at most k entries) become one: the entries
// within the bound are packed to the front (read to registers, a barrier,
// written at the warp's offset), the next power of two of them sorted, the
// first k distinct distances kept; the merge then reads one part per block.
template <int W>
__device__ __forceinline__ void ed_finish(const EdArgs& a, unsigned long long* lists, unsigned long long* list, int cnt,
                                          uint32_t n_chunks, uint32_t n_done, uint32_t n_rows) {
  constexpr int kEdThreads = 32 * W;
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  cnt = warp_compact(list, cnt, a.k);
  uint32_t B = 0;
  if (lane == 0) {
    if (cnt == a.k) atomicMin(a.bound, (uint32_t)(list[a.k - 1] >> 32));
    B = ld_volatile(a.bound);
  }
  B = __shfl_sync(HG_FULL, B, 0);
  __shared__ int s_cnt[W];
  constexpr int kPer = kWarpListCap / 32;  // entries per lane of a full list
  unsigned long long mine[kPer];
  int within = 0;  // entries within the bound: a prefix of the sorted list
#pragma unroll
  for (int r = 0; r < kPer; ++r) {
    mine[r] = list[lane + 32 * r];
    within += __popc(__ballot_sync(HG_FULL, lane + 32 * r < cnt && (uint32_t)(mine[r] >> 32) <= B));
  }
  cnt = within;
  if (lane == 0) s_cnt[wib] = cnt;
  __syncthreads();
  int offset = 0, packed = 0;
#pragma unroll
  for (int w = 0; w < W; ++w) {
    offset += w < wib ? s_cnt[w] : 0;
    packed += s_cnt[w];
  }
  int nsort = 32;
  while (nsort < packed) nsort <<= 1;
  unsigned long long* flat = lists;
  __syncthreads();
#pragma unroll
  for (int r = 0; r < kPer; ++r)
    if (lane + 32 * r < cnt) flat[offset + lane + 32 * r] = mine[r];
  for (int i = packed + (int)threadIdx.x; i < nsort; i += kEdThreads) flat[i] = ~0ull;
  __syncthreads();
  for (int size = 2; size <= nsort; size <<= 1)
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      for (int i = threadIdx.x; i < nsort / 2; i += kEdThreads) {
        const int pos = 2 * i - (i & (stride - 1));
        const int partner = pos + stride;
        const bool asc = (pos & size) == 0;
        const unsigned long long x = flat[pos], y = flat[partner];
        if ((x > y) == asc) {
          flat[pos] = y;
          flat[partner] = x;
        }
      }
      __syncthreads();
    }
  if (wib == 0) {
    const int bc = warp_dedup_sorted(flat, packed, a.k, 0);
    for (int i = lane; i < bc; i += 32) a.parts[i] = flat[i];
    if (lane == 0) {
      *a.part_count = bc;
      if (bc == a.k) atomicMin(a.bound, (uint32_t)(flat[a.k - 1] >> 32));
    }
  }
  unsigned long long s_chunks = n_chunks, s_done = n_done, s_rows = n_rows;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    s_chunks += __shfl_xor_sync(HG_FULL, s_chunks, o);
    s_done += __shfl_xor_sync(HG_FULL, s_done, o);
    s_rows += __shfl_xor_sync(HG_FULL, s_rows, o);
  }
  if (lane == 0) {
    atomicAdd(&a.stats[1], s_chunks);
    atomicAdd(&a.stats[4], s_done);
    atomicAdd(&a.stats[5], s_rows);
  }
}

// kRowIds: the id of a row is its row index (a matrix without an id map).
// kSlot: lanes per row (a slot); kLines: 32-byte chunks per lane of a row in
// flight per step, so a slot reads kSlot * kLines * 32 bytes of its row per
// step.  Short series use 4-lane slots (8 rows per warp, 128-byte lines);
// long series, few candidate rows per query, use wider slots.
// kWarps: warps per block.  Eight, four blocks per SM, where the staged query
// leaves room for four blocks; else 32 warps that share one staged query, one
// block per SM (from about 7,900 points: at 16,384 two blocks of eight fitted,
// and 12 queries of 100k x 16384 took 1.18 instead of 1.12 ms).
// The allocation-free scan, which has room for 148 lists, uses 32 at any
// length (eight warps per SM: 325 us for 1M x 256, 32: 183 us).
template <int kSlot>
__host__ __device__ constexpr uint32_t slot_leaders() {
  return kSlot == 32 ? 0x1u : (kSlot == 16 ? 0x10001u : (kSlot == 8 ? 0x01010101u : 0x11111111u));
}
template <bool kRowIds, int kLines, int kSlot, int kWarps>
__global__ void __launch_bounds__(32 * kWarps, 32 / kWarps) k_ed_stream(EdArgs a) {
  constexpr int W = kWarps;
  extern __shared__ float4 ed_smem[];
  unsigned long long* lists = reinterpret_cast<unsigned long long*>(ed_smem);  // [W][kWarpListCap]
  float4* qs4 = ed_smem + W * kWarpListCap / 2;                                // the query, q4_bytes(L) bytes
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const int slot_lead = lane & ~(kSlot - 1), j = lane & (kSlot - 1);
  const int nch = a.L >> 3;
  uint64_t first;
  uint32_t total, bs;
  if (!kRowIds && kSlot >= 8 && a.few_rows && a.few_rows != UINT32_MAX) {
    // one of two launches over the same list, and the other one's list (looked
    // at here and not in ed_range, where it made this kernel spill)
    const uint32_t n = a.list_count[8 * blockIdx.x];
    if (kSlot == 32 ? n > a.few_rows : n <= a.few_rows) return;
  }
  if (!ed_range<W>(a, first, total, bs)) return;
  const uint32_t nwarps = gridDim.y * W;
  const uint32_t gw = blockIdx.y * W + wib;
  const uint32_t leaders = slot_leaders<kSlot>();
  unsigned long long* list = lists + wib * kWarpListCap;
  for (int i = lane; i < kWarpListCap; i += 32) list[i] = ~0ull;
  for (int i = threadIdx.x; i < (a.L >> 2); i += 32 * W)
    qs4[q4_index(i >> 1, i & 1)] = reinterpret_cast<const float4*>(a.q)[i];
  __shared__ EdShared sh;
  ed_shared_init(a, sh, 32 * W);
  __syncthreads();
  auto entry = [&](uint32_t batch) -> uint32_t {
    const uint64_t idx = (uint64_t)batch * bs + lane;
    if ((uint32_t)lane >= bs || idx >= total) return 0xffffffffu;
    return a.list ? a.list[idx] : (uint32_t)(first + idx);
  };
  auto count_of = [&](uint32_t batch) -> uint32_t {
    const uint64_t b0 = (uint64_t)batch * bs;
    return b0 < total ? (uint32_t)(total - b0 < bs ? total - b0 : bs) : 0u;
  };
  uint32_t batch = gw;
  uint32_t cur = entry(batch);  // lane i holds entry i of the current batch
  uint32_t cur_n = count_of(batch);
  uint32_t cur_used = 0;
  batch += nwarps;
  uint32_t nxt = entry(batch);
  uint32_t nxt_n = count_of(batch);

  int cnt = 0;
  float T = __int_as_float(0x7f800000);
  float B = __uint_as_float(sh.bound);
  const float F = a.has_floor ? a.floor : -1.0f;  // distances are >= 0
  bool valid = false;  // slot-uniform
  uint32_t row = 0;
  int ch = 0;  // a multiple of kStep: the query offsets below stay inside one 32-chunk group
  float dist = 0.0f;
  const float* x = nullptr;
  uint32_t n_chunks = 0, n_done = 0, n_rows = 0;  // this lane's (slot leaders only)
  constexpr int kStep = kSlot * kLines;  // chunks of a row per step
  static_assert(32 % kStep == 0, "a step stays inside one 32-chunk group of the staged query");
  // staged-query float4 index of chunk ch + kSlot l + j: base(ch) + qoff[l]
  int qoff[kLines];
#pragma unroll
  for (int l = 0; l < kLines; ++l) {
    const int o = kSlot * l + j;
    qoff[l] = 2 * (o + (o >> 2));
  }
  for (uint32_t turn = 0;; ++turn) {
    // refill the slots without a row
    uint32_t need = __ballot_sync(HG_FULL, !valid) & leaders;
    while (need) {
      if (cur_used == cur_n) {
        if (nxt_n == 0) break;
        cur = nxt;
        cur_n = nxt_n;
        cur_used = 0;
        batch += nwarps;
        nxt = entry(batch);  // loaded while the current batch is consumed
        nxt_n = count_of(batch);
      }
      const int take = min(__popc(need), (int)(cur_n - cur_used));
      const int r = __popc(need & ((1u << slot_lead) - 1));  // rank among the free slots
      const bool mine = ((need >> slot_lead) & 1u) && r < take;
      const uint32_t got = __shfl_sync(HG_FULL, cur, (cur_used + (mine ? r : 0)) & 31);
      if (mine) {
        row = got;
        valid = true;
        dist = 0.0f;
        ch = 0;
        x = a.rows + (uint64_t)row * a.L + 8 * j;
        if (j == 0) ++n_rows;
      }
      cur_used += take;
      need = __ballot_sync(HG_FULL, !valid) & leaders;
    }
    if (!__any_sync(HG_FULL, valid)) break;
    // kLines chunks of every owned row in flight: lane j computes chunks
    // ch + kSlot l + j (l < kLines); chunks past the row's end count as 0
    float xa[kLines][8];
    bool in[kLines];
#pragma unroll
    for (int l = 0; l < kLines; ++l) {
      in[l] = valid && ch + kSlot * l + j < nch;
      if (in[l]) {
        if constexpr (kRowIds || (kWarps != 32 && kSlot != 32)) {
          // a caller's matrix is aligned to 16 bytes; and 8-warp blocks over
          // medium lengths are up to 3% faster with these
          const float4* p = reinterpret_cast<const float4*>(x + 8 * kSlot * l);
          const float4 lo = __ldcs(p), hi = __ldcs(p + 1);
          xa[l][0] = lo.x; xa[l][1] = lo.y; xa[l][2] = lo.z; xa[l][3] = lo.w;
          xa[l][4] = hi.x; xa[l][5] = hi.y; xa[l][6] = hi.z; xa[l][7] = hi.w;
        } else {
          load_chunk(x + 8 * kSlot * l, xa[l]);
        }
      }
    }
    // a slot without a row (its ch may equal nch) reads the first chunks:
    // every index stays inside the staged query
    const int cq = valid ? ch : 0;
    const int qb = 2 * ((cq >> 5) * 40 + (cq & 31) + ((cq & 31) >> 2));
    float dl[kLines];
#pragma unroll
    for (int l = 0; l < kLines; ++l) {
      const float4 q0 = qs4[qb + qoff[l]], q1 = qs4[qb + qoff[l] + 1];
      const float qa[8] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
      const float d = hg_chunk_d2(qa, xa[l]);
      dl[l] = in[l] ? d : 0.0f;
    }
    // the slot adds the step's chunk sums in order (adding 0 leaves a sum
    // unchanged); one abandon test per step, since the step's lines are
    // already loaded
    float part[kStep];
    float acc = dist;
#pragma unroll
    for (int t = 0; t < kStep; ++t) {
      acc = __fadd_rn(acc, __shfl_sync(HG_FULL, dl[t / kSlot], slot_lead + (t % kSlot)));
      part[t] = acc;
    }
    bool finished = false;
    if (valid) {
      if (acc > B) {
        // abandoned: the reference reads up to the first chunk whose sum
        // exceeds the bound (the partial sums never decrease)
        if (j == 0) {
          int used = 1;
#pragma unroll
          for (int t = 0; t < kStep; ++t) used += part[t] <= B ? 1 : 0;
          n_chunks += (uint32_t)(ch + used);
        }
        valid = false;
      } else {
        dist = acc;
        ch += kStep;
        x += 8 * kStep;
        if (ch >= nch) {
          finished = true;
          valid = false;
          if (j == 0) {
            n_chunks += (uint32_t)nch;
            ++n_done;
          }
        }
      }
    }
    const bool take = finished && j == 0 && dist <= B && dist <= T && dist > F;
    warp_list_add<true>(list, cnt, T, a.k, a.bound, take, dist, take ? (kRowIds ? row : (uint32_t)a.ids[row]) : 0u);
    B = ed_bound(a, sh, turn, take, dist, B, T);
  }
  ed_finish<W>(a, lists, list, cnt, n_chunks, n_done, n_rows);
}

// The same for a group of queries over short series: a warp takes 32 / kSlot
// rows (kSlot lanes each) together and stays with them until the last has finished or
// abandoned, instead of giving a free slot the next row at every step.  Lanes
// idle more (a row of 256 points abandons after 1.5 to 2.7 of its 4 steps), but
// a step costs far fewer instructions (no refill; one place in the query for
// all slots, so its reads are broadcasts), which bind the scan once a group
// keeps every warp busy: 16 queries of 8M x 256, k = 100, 6.01 -> 5.66 ms per
// call, 100 of 1M x 256 2.91 -> 2.73, 16 of 1M x 1024 1.19 -> 1.08, 16 of 300k
// x 2048 0.85 -> 0.77.  A query alone waits for its loads instead, and the
// other kernel's slots never idle: allocation-free scan of 1M x 256 127 us
// there, 145 here.  (Loading the next rows' first step early spills at 64
// registers, 5 to 20% slower; through shared memory with cp.async it does not,
// and is 1 to 11% slower: issue, load pipe and DRAM are each half busy.)  Up to 256 points 16 rows of 128 bytes per step:
// half the chain of sums per row and less read past the abandoning chunk
// (PSCAN of 2M x 256, 4 queries 655 -> 555 us, of 2M x 96, 8 queries 740 -> 481,
// 16 queries of 8M x 256 5.37 -> 5.10 ms); longer rows differ more, so 8 of 256
// bytes (1M x 1024: 1.04 ms against 1.13).
template <int kSlot, int kLines>
__global__ void __launch_bounds__(32 * kEdWarps, kEdBlocksPerSm) k_ed_short(EdArgs a) {
  constexpr int W = kEdWarps, kStep = kSlot * kLines, kRows = 32 / kSlot;
  extern __shared__ float4 ed_smem[];
  unsigned long long* lists = reinterpret_cast<unsigned long long*>(ed_smem);  // [W][kWarpListCap]
  float4* qs = ed_smem + W * kWarpListCap / 2;                                 // the query, whole steps, zero beyond L
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const int slot = lane / kSlot, slot_lead = lane & ~(kSlot - 1), j = lane & (kSlot - 1);
  const int nch = a.L >> 3;
  uint64_t first;
  uint32_t total, bs;
  if (!ed_range<W>(a, first, total, bs)) return;
  unsigned long long* list = lists + wib * kWarpListCap;
  for (int i = lane; i < kWarpListCap; i += 32) list[i] = ~0ull;
  for (int i = threadIdx.x; i < 2 * ((nch + kStep - 1) / kStep) * kStep; i += 32 * W)
    qs[i] = i < 2 * nch ? reinterpret_cast<const float4*>(a.q)[i] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  __shared__ EdShared sh;
  ed_shared_init(a, sh, 32 * W);
  __syncthreads();
  const uint32_t nwarps = gridDim.y * W;
  uint32_t batch = blockIdx.y * W + wib;  // the batch of `cur`
  auto entry = [&](uint32_t b) -> uint32_t {
    const uint64_t idx = (uint64_t)b * bs + lane;
    if ((uint32_t)lane >= bs || idx >= total) return 0u;
    return a.list ? a.list[idx] : (uint32_t)(first + idx);
  };
  auto count_of = [&](uint32_t b) -> uint32_t {
    const uint64_t b0 = (uint64_t)b * bs;
    return b0 < total ? (uint32_t)(total - b0 < bs ? total - b0 : bs) : 0u;
  };
  uint32_t cur = entry(batch), cur_n = count_of(batch), used = 0;  // lane i holds entry i of the batch
  uint32_t nxt = entry(batch + nwarps), nxt_n = count_of(batch + nwarps);
  // the next kRows rows; false: none left
  uint32_t row = 0;
  bool alive = false;  // slot-uniform
  auto fetch = [&]() -> bool {
    if (used >= cur_n) {
      if (nxt_n == 0) return false;
      batch += nwarps;
      cur = nxt;
      cur_n = nxt_n;
      used = 0;
      nxt = entry(batch + nwarps);
      nxt_n = count_of(batch + nwarps);
    }
    row = __shfl_sync(HG_FULL, cur, (int)(used + slot) & 31);
    alive = used + slot < cur_n;
    used += kRows;
    return true;
  };
  int cnt = 0;
  float T = __int_as_float(0x7f800000);
  float B = __uint_as_float(sh.bound);
  const float F = a.has_floor ? a.floor : -1.0f;  // distances are >= 0
  uint32_t n_chunks = 0, n_done = 0, n_rows = 0;  // this lane's (slot leaders only)
  for (uint32_t turn = 0; fetch(); ++turn) {
    const float* x = a.rows + (uint64_t)row * a.L + 8 * j;
    if (alive && j == 0) ++n_rows;
    float dist = 0.0f;
    for (int ch = 0;;) {
      float xa[kLines][8];
      bool in[kLines];
#pragma unroll
      for (int l = 0; l < kLines; ++l) {
        in[l] = alive && ch + kSlot * l + j < nch;
        if (in[l]) load_chunk(x + 8 * (ch + kSlot * l), xa[l]);
      }
      float dl[kLines];
#pragma unroll
      for (int l = 0; l < kLines; ++l) {
        const float4 q0 = qs[2 * (ch + kSlot * l + j)], q1 = qs[2 * (ch + kSlot * l + j) + 1];
        const float qa[8] = {q0.x, q0.y, q0.z, q0.w, q1.x, q1.y, q1.z, q1.w};
        const float d = hg_chunk_d2(qa, xa[l]);
        dl[l] = in[l] ? d : 0.0f;  // adding 0 leaves a sum unchanged
      }
      float part[kStep];
      float acc = dist;
#pragma unroll
      for (int t = 0; t < kStep; ++t) {
        acc = __fadd_rn(acc, __shfl_sync(HG_FULL, dl[t / kSlot], slot_lead + (t % kSlot)));
        part[t] = acc;
      }
      const bool dead = alive && acc > B;
      if (dead && j == 0) {
        // the reference reads up to the first chunk whose sum exceeds the
        // bound (the partial sums never decrease)
        uint32_t u = 1;
#pragma unroll
        for (int t = 0; t < kStep; ++t) u += part[t] <= B ? 1u : 0u;
        n_chunks += (uint32_t)ch + u;
      }
      alive = alive && !dead;
      dist = acc;
      ch += kStep;
      if (ch >= nch || !__any_sync(HG_FULL, alive)) break;
    }
    const bool lead = alive && j == 0;
    if (lead) {
      n_chunks += (uint32_t)nch;
      ++n_done;
    }
    const bool take = lead && dist <= B && dist <= T && dist > F;
    warp_list_add<true>(list, cnt, T, a.k, a.bound, take, dist, take ? (uint32_t)a.ids[row] : 0u);
    B = ed_bound(a, sh, turn, take, dist, B, T);
  }
  ed_finish<W>(a, lists, list, cnt, n_chunks, n_done, n_rows);
}

// Merges the per-block lists and the current top-k into the k smallest
// distinct distances, lowest id per distance; returns the bound after it.
// Only entries <= the bound can belong to the answer, and the lists are
// sorted, so a warp per list reads a prefix of each, 32 entries at a time,
// four lists in flight.  All of them are gathered in one go if they fit in
// buf; if not (large k, many lists), 32 lists are merged alone, which lowers
// the bound, and the rest is tried again.  (A thread per list with its reads
// one after the other: 8 - 25 us per merge at k = 10, and about 150 us at
// k = 100 with 592 lists.)
constexpr int kMergeThreads = 1024;
__device__ float merge_parts(const MergeArgs& a, uint32_t slot, unsigned long long* buf /* kMergeCap */) {
  __shared__ int s_n, s_best;
  const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
  constexpr int W = kMergeThreads / 32;
  static_assert(kMaxK + W * kMaxK <= kMergeCap, "the lists of one round fit");
  const unsigned long long* parts = a.parts + (uint64_t)slot * a.parts_stride * kWarpListCap;
  const int* part_count = a.part_count + (uint64_t)slot * a.parts_stride;
  unsigned long long* topk = a.topk + (uint64_t)slot * kMaxK;
  const int k = a.k;
  uint32_t B = ld_volatile(a.bound + slot);
  const int n0 = a.topk_count[slot];
  for (int i = t; i < n0; i += kMergeThreads) buf[i] = topk[i];
  if (t == 0) s_best = n0;
  __syncthreads();
  for (int p_lo = 0;;) {
    const int nbest = s_best;
    // [p_lo, p_hi): every list left, or after an overflow the next 32
    int p_hi = a.nparts;
    for (;;) {
      if (t == 0) s_n = nbest;
      __syncthreads();
      for (int pb = p_lo + wid; pb < p_hi; pb += 4 * W) {
        int cnt[4];
        unsigned long long v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) cnt[u] = pb + u * W < p_hi ? part_count[pb + u * W] : 0;
#pragma unroll
        for (int u = 0; u < 4; ++u)
          v[u] = lane < cnt[u] ? parts[(uint64_t)(pb + u * W) * kWarpListCap + lane] : ~0ull;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          unsigned long long x = v[u];
          for (int base = 0; base < cnt[u]; base += 32) {
            if (base) x = base + lane < cnt[u] ? parts[(uint64_t)(pb + u * W) * kWarpListCap + base + lane] : ~0ull;
            const bool take = base + lane < cnt[u] && (uint32_t)(x >> 32) <= B;
            const uint32_t m = __ballot_sync(HG_FULL, take);
            int pos = 0;
            if (lane == 0 && m) pos = atomicAdd(&s_n, __popc(m));
            pos = __shfl_sync(HG_FULL, pos, 0) + __popc(m & ((1u << lane) - 1));
            if (take && pos < kMergeCap) buf[pos] = x;
            if (m != HG_FULL) break;
          }
        }
      }
      __syncthreads();
      if (s_n <= kMergeCap) break;
      p_hi = min(a.nparts, p_lo + W);
      __syncthreads();
    }
    const int n = s_n;
    if (n > nbest) {
      int nsort = 32;
      while (nsort < n) nsort <<= 1;
      for (int i = n + t; i < nsort; i += kMergeThreads) buf[i] = ~0ull;
      __syncthreads();
      for (int size = 2; size <= nsort; size <<= 1)
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
          for (int i = t; i < nsort / 2; i += kMergeThreads) {
            const int pos = 2 * i - (i & (stride - 1));
            const int partner = pos + stride;
            const bool asc = (pos & size) == 0;
            const unsigned long long x = buf[pos], y = buf[partner];
            if ((x > y) == asc) {
              buf[pos] = y;
              buf[partner] = x;
            }
          }
          __syncthreads();
        }
      if (wid == 0) {
        const int best = warp_dedup_sorted(buf, n, k, 0);
        if (lane == 0) s_best = best;
      }
      __syncthreads();
    }
    if (s_best == k) B = min(B, (uint32_t)(buf[k - 1] >> 32));
    p_lo = p_hi;
    if (p_lo >= a.nparts) break;
  }
  const int cnt = s_best;
  for (int i = t; i < cnt; i += kMergeThreads) topk[i] = buf[i];
  if (t == 0) {
    a.topk_count[slot] = cnt;
    a.bound[slot] = B;
  }
  if (a.dist_out || a.id_out) {
    const uint64_t out_at = a.out_row ? (uint64_t)a.out_row[slot] * a.out_stride : (uint64_t)slot * k;
    for (int i = t; i < k; i += kMergeThreads) {
      const unsigned long long v = i < cnt ? buf[i] : ~0ull;
      if (a.dist_out)
        a.dist_out[out_at + i] = i < cnt ? __uint_as_float((uint32_t)(v >> 32)) : __int_as_float(0x7f800000);
      if (a.id_out) a.id_out[out_at + i] = i < cnt ? (int64_t)(uint32_t)v : -1;
    }
  }
  return __uint_as_float(B);
}

__global__ void __launch_bounds__(kMergeThreads) k_merge(MergeArgs a) {
  extern __shared__ unsigned long long merge_buf[];  // kMergeCap
  merge_parts(a, blockIdx.x, merge_buf);
}

// The merge of the approximate leaf's lists and, against the bound it gives,
// the candidate leaves: one block per query, the two steps one after the
// other in the same shared memory.
__global__ void __launch_bounds__(kMergeThreads) k_merge_select(MergeArgs a, SelectArgs sel) {
  extern __shared__ unsigned long long merge_buf[];
  static_assert(kMergeThreads == kSortThreads, "one block does both");
  const float B = merge_parts(a, blockIdx.x, merge_buf);
  __syncthreads();
  select_sort(sel, blockIdx.x, B, reinterpret_cast<uint32_t*>(merge_buf));
}

__global__ void k_emit(const unsigned long long* topk, const int* topk_count, int k, float* dist_out,
                       int64_t* id_out) {
  const int i = threadIdx.x + blockIdx.x * blockDim.x;
  if (i >= k) return;
  const int n = *topk_count;
  if (i < n) {
    const unsigned long long v = topk[i];
    if (dist_out) dist_out[i] = __uint_as_float((uint32_t)(v >> 32));
    if (id_out) id_out[i] = (int64_t)(uint32_t)v;
  } else {
    if (dist_out) dist_out[i] = __int_as_float(0x7f800000);
    if (id_out) id_out[i] = -1;
  }
}

// ---------------------------------------------------------------------------
// data generation
// ---------------------------------------------------------------------------

__global__ void k_generate_walks(uint64_t seed, uint64_t first, uint64_t n, int L, float* out, int unit) {
  const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  // each thread writes its own row; the L2 merges the partial sectors
  if (unit) gaussian_unit(seed, first + i, L, out + i * (uint64_t)L);
  else random_walk(seed, first + i, L, out + i * (uint64_t)L);
}

// data == nullptr: the base row is regenerated from data_seed into the
// query's own output row (the collection need not be resident), then the
// noise is added in place.
__global__ void k_generate_queries(uint64_t seed, const float* data, uint64_t n, int L, int nq,
                                   const double* sigma2, float* out, uint64_t* base_ids, int unit,
                                   uint64_t data_seed) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= nq) return;
  const uint64_t b = pick_row(seed, (uint64_t)j, n);
  if (base_ids) base_ids[j] = b;
  float* o = out + (uint64_t)j * L;
  const float* base = data + b * (uint64_t)L;
  if (!data) {
    if (unit) gaussian_unit(data_seed, b, L, o);
    else random_walk(data_seed, b, L, o);
    base = o;
  }
  noisy_query(seed, (uint64_t)j, base, L, sigma2[j], o, unit);
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------

static inline unsigned blocks_for(uint64_t n, int t) { return (unsigned)((n + t - 1) / t); }

int sm_count(int device) {
  int sms = 148;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  return sms;
}

cudaError_t launch_route_rows(const float* X, int L, uint64_t first, uint32_t count, Tree t, int* node_of,
                              cudaStream_t s) {
  if (!count) return cudaSuccess;
  if (L <= kStagedL) {
    static SmemLimit attr;
    const cudaError_t ea = attr.ensure((const void*)k_route_staged, (int)staged_bytes(kStagedL));
    if (ea != cudaSuccess) return ea;
    k_route_staged<<<blocks_for(count, kStagedRows), 32, staged_bytes(L), s>>>(X, L, first, count, t, node_of);
  } else {
    k_route_long<<<blocks_for((uint64_t)count * 32, 256), 256, 0, s>>>(X, L, first, count, t, node_of);
  }
  return cudaGetLastError();
}

cudaError_t launch_collect_members(const int* node_of, uint64_t end, const int* slot_of, const uint64_t* start,
                                   const uint32_t* last, uint64_t members, uint32_t* list, uint32_t* counts,
                                   uint32_t* later, int* keys, int nsegs, cudaStream_t s) {
  const unsigned want = blocks_for(end ? end : 1, 4 * 256);
  k_collect_members<<<want < 148 * 8 ? want : 148 * 8, 256, 0, s>>>(node_of, end, slot_of, start, last, members, list,
                                                                    counts, later, keys, nsegs);
  return cudaGetLastError();
}

cudaError_t launch_sketch(const SketchArgs& a, cudaStream_t s) {
  const int groups = a.ngroups, segs = a.max_segs;
  const uint32_t size = a.max_size;
  if (!groups || !segs || !size) return cudaSuccess;
  const bool staged = a.L <= kStagedL;
  // parts per group: the rows of one tile (8 (row, segment) pairs) at least,
  // and enough blocks in all for every SM
  const uint64_t most = staged ? blocks_for(size, kStagedRows) : blocks_for((uint64_t)size * segs, kSketchThreads / 32);
  const uint64_t fill = (148 * 8 + groups - 1) / groups;
  const unsigned parts = (unsigned)(most < fill ? most : fill);
  if (staged) {
    const size_t smem = staged_bytes(a.L) + sizeof(int) * 4 * segs;
    static SmemLimit attr;
    const cudaError_t ea = attr.ensure((const void*)k_sketch_staged, 200 * 1024);
    if (ea != cudaSuccess) return ea;
    k_sketch_staged<<<dim3(groups, parts), kSketchThreads, smem, s>>>(a);
  } else {
    static SmemLimit attr;
    const cudaError_t ea = attr.ensure((const void*)k_sketch_long, 200 * 1024);
    if (ea != cudaSuccess) return ea;
    k_sketch_long<<<dim3(groups, parts), kSketchThreads, sizeof(int) * 4 * segs, s>>>(a);
  }
  return cudaGetLastError();
}

cudaError_t launch_split_members(const float* X, int L, int* node_of, const uint32_t* list, uint64_t members,
                                 const uint32_t* later, uint64_t later_max, const int* slot_of, const SplitPolicy* splits,
                                 uint32_t* n_left, cudaStream_t s) {
  const uint64_t rows = members + later_max;
  if (!rows) return cudaSuccess;
  const unsigned want = blocks_for(rows * 32, 256);
  k_split_members<<<want < 148 * 32 ? want : 148 * 32, 256, 0, s>>>(X, L, node_of, list, members, later, slot_of, splits,
                                                                  n_left);
  return cudaGetLastError();
}

cudaError_t launch_widen_ids(const uint32_t* perm, uint64_t n, int64_t* ids, cudaStream_t s) {
  if (!n) return cudaSuccess;
  k_widen_ids<<<blocks_for(n, 256), 256, 0, s>>>(perm, n, ids);
  return cudaGetLastError();
}

cudaError_t launch_gather_rows(const float* X, int L, const uint32_t* perm, uint64_t n, float* rows,
                               cudaStream_t s) {
  const uint64_t threads = n * (L / 4);
  if (!threads) return cudaSuccess;
  k_gather_rows<<<blocks_for(threads, 256), 256, 0, s>>>(X, L, perm, n, rows);
  return cudaGetLastError();
}

cudaError_t launch_sax_rows(const float* rows, int L, uint64_t n, const float* bp, uint8_t* sax,
                            cudaStream_t s) {
  if (!n) return cudaSuccess;
  k_sax_rows<<<blocks_for(n * HG_PAA_SEGMENTS, 256), 256, 0, s>>>(rows, L, n, bp, sax);
  return cudaGetLastError();
}

cudaError_t launch_query_prep(const PrepArgs& a, int slots, cudaStream_t s) {
  static SmemLimit attr;
  const cudaError_t ea = attr.ensure((const void*)k_query_prep, 65536);
  if (ea != cudaSuccess) return ea;
  unsigned blocks = a.lb ? blocks_for((uint64_t)a.nleaves * 32, kPrepThreads) : 0;
  if (a.sax_tab && blocks < HG_PAA_SEGMENTS) blocks = HG_PAA_SEGMENTS;
  if (blocks > 4096) blocks = 4096;  // a warp takes several leaves from 32,768 on (grid.y ends at 65,535)
  k_query_prep<<<dim3(slots, blocks + 1), kPrepThreads, sizeof(float) * a.L, s>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_route_queries(const float* Q, int nq, int L, Tree t, int* leaf_out, cudaStream_t s,
                                 uint32_t* zero_a, uint32_t na, uint32_t* zero_b, uint32_t nb,
                                 unsigned long long* stamp) {
  if (!nq) return cudaSuccess;
  k_route_queries<<<blocks_for((uint64_t)nq * 32, 128), 128, 0, s>>>(Q, nq, L, t, leaf_out, zero_a, na, zero_b, nb, stamp);
  return cudaGetLastError();
}

cudaError_t launch_leaf_keep(const float* Q, int L, int nq, const short* useg_start, const short* useg_end, int nu,
                             float2* segstats, const int* seg_off, const short* points, const int* seg_uid,
                             const float* sk, const uint32_t* leaf_size, int nleaves, const float* bound,
                             uint32_t* leaf_cnt, uint32_t* leaf_q, uint32_t stride, cudaStream_t s) {
  if (nq <= 0 || nleaves <= 0) return cudaSuccess;
  static SmemLimit attr;
  const cudaError_t ea = attr.ensure((const void*)k_query_segstats, 65536);
  if (ea != cudaSuccess) return ea;
  k_query_segstats<<<nq, 256, sizeof(float) * L, s>>>(Q, L, nq, useg_start, useg_end, nu, segstats);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  return launch_leaf_keep_list(segstats, nu, L, nq, seg_off, points, seg_uid, sk, leaf_size, nleaves, bound,
                               leaf_cnt, leaf_q, stride, nullptr, nullptr, s);
}

cudaError_t launch_leaf_keep_list(const float2* segstats, int nu, int L, int nq, const int* seg_off,
                                  const short* points, const int* seg_uid, const float* sk, const uint32_t* leaf_size,
                                  int nleaves, const float* bound, uint32_t* leaf_cnt, uint32_t* leaf_q,
                                  uint32_t stride, const uint32_t* qlist, const uint32_t* nq_dev, cudaStream_t s) {
  if (nq <= 0 || nleaves <= 0) return cudaSuccess;
  // grid-stride over the (query, leaf) pairs: at most 64 blocks of 256 threads per SM
  int dev = 0;
  const cudaError_t ed = cudaGetDevice(&dev);
  if (ed != cudaSuccess) return ed;
  const uint64_t want = blocks_for((uint64_t)nq * nleaves, 256);
  const uint64_t cap = 64ull * (uint64_t)sm_count(dev);
  k_leaf_keep<<<(unsigned)(want < cap ? want : cap), 256, 0, s>>>(
      segstats, nu, L, nq, seg_off, points, seg_uid, sk, leaf_size, nleaves, bound, leaf_cnt, leaf_q, stride, qlist,
      nq_dev);
  return cudaGetLastError();
}

__global__ void k_leaf_gate(float lb, float eps1, const uint32_t* stale, int* flag, unsigned long long* scanned) {
  const float kth = __uint_as_float(*stale);
  const int pass = lb <= __fdiv_rn(kth, eps1) ? 1 : 0;
  *flag = pass;
  if (pass) ++*scanned;
}
__global__ void k_stale_copy(const int* flag, const uint32_t* bound, uint32_t* stale) {
  if (*flag) *stale = *bound;
}
cudaError_t launch_leaf_gate(float lb, float eps1, const uint32_t* stale, int* flag, unsigned long long* scanned,
                             cudaStream_t s) {
  k_leaf_gate<<<1, 1, 0, s>>>(lb, eps1, stale, flag, scanned);
  return cudaGetLastError();
}
cudaError_t launch_stale_copy(const int* flag, const uint32_t* bound, uint32_t* stale, cudaStream_t s) {
  k_stale_copy<<<1, 1, 0, s>>>(flag, bound, stale);
  return cudaGetLastError();
}

static size_t select_smem(bool global_keys) {
  return sizeof(uint32_t) * 16 * kSortThreads + (global_keys ? 0 : sizeof(uint32_t) * 4 * kMaxLeavesSort);
}
constexpr size_t kMergeSmem = sizeof(unsigned long long) * kMergeCap;

cudaError_t launch_merge(const MergeArgs& a, int slots, cudaStream_t s) {
  static SmemLimit attr;
  const cudaError_t ea = attr.ensure((const void*)k_merge, (int)kMergeSmem);
  if (ea != cudaSuccess) return ea;
  k_merge<<<slots, kMergeThreads, kMergeSmem, s>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_merge_select(const MergeArgs& a, const SelectArgs& sel, int slots, cudaStream_t s) {
  const bool global_keys = sel.nleaves > kMaxLeavesSort;
  if (global_keys && !sel.gkeys) return cudaErrorInvalidValue;
  static SmemLimit attr;
  const cudaError_t ea = attr.ensure((const void*)k_merge_select, (int)select_smem(false));
  if (ea != cudaSuccess) return ea;
  SelectArgs b = sel;
  if (!global_keys) b.gkeys = nullptr;
  const size_t ss = select_smem(global_keys);
  k_merge_select<<<slots, kMergeThreads, ss > kMergeSmem ? ss : kMergeSmem, s>>>(a, b);
  return cudaGetLastError();
}

cudaError_t launch_pscan_prep(uint32_t* bound, uint32_t* kslots, int* topk_count, int slots, cudaStream_t s) {
  k_pscan_prep<<<slots, 128, 0, s>>>(bound, kslots, topk_count);
  return cudaGetLastError();
}

cudaError_t launch_list_rows(const FilterArgs& a, int slots, int blocks, cudaStream_t s) {
  k_list_rows<<<dim3(slots, blocks), 32 * kListWarps, 0, s>>>(a);
  return cudaGetLastError();
}
cudaError_t launch_lbsax_filter(const FilterArgs& a, int slots, int blocks, cudaStream_t s) {
  static SmemLimit attr;
  const cudaError_t ea = attr.ensure((const void*)k_lbsax_filter, (int)lbsax_filter_smem());
  if (ea != cudaSuccess) return ea;
  k_lbsax_filter<<<dim3(slots, blocks), kFilterThreads, lbsax_filter_smem(), s>>>(a);
  return cudaGetLastError();
}

static size_t ed_smem_bytes(int L, int warps) { return (size_t)warps * kWarpListCap * 8 + q4_bytes(L); }
// 32-warp blocks: where fewer than four 8-warp blocks fit on an SM
static bool ed_wide(int L) { return kEdBlocksPerSm * (ed_smem_bytes(L, kEdWarps) + 1024) > (size_t)227 * 1024; }
constexpr int kEdShortL = 2048;  // k_ed_short up to this length, for groups

template <class K>
static cudaError_t launch_ed(K kernel, SmemLimit& attr, const EdArgs& args, int warps, int slots, int blocks,
                             cudaStream_t s) {
  const cudaError_t ea = attr.ensure((const void*)kernel, (int)ed_smem_bytes(16384, warps));
  if (ea != cudaSuccess) return ea;
  EdArgs a = args;
  a.period = 2 * (uint32_t)warps;
  for (int k = 32; k < a.k; k *= 2) a.period *= 2;
  kernel<<<dim3(slots, blocks), 32 * warps, ed_smem_bytes(a.L, warps), s>>>(a);
  return cudaGetLastError();
}
// Groups over series of at most kEdShortL points: k_ed_short (longer rows of a
// warp differ too much in where they abandon).  Long series (L >= 4096): few
// candidate rows per query, each long, so more lanes per row keep more of each
// row in flight -- all 32 where there are fewer rows than warps (one query over
// a leaf of a thousand rows of 64 KB reads each row in 128 dependent steps with
// 8 lanes: 528 us, 348 us with 32; with rows for every warp 8 lanes are faster,
// PSCAN of 60k x 16384 619 us against 1,007).  Where the device alone knows how
// many rows there are, both are launched and one of them returns at once.
cudaError_t launch_ed_stream(const EdArgs& a, int slots, int blocks, cudaStream_t s) {
  static SmemLimit wide, lng, mid, shrt, shrt2, few_wide, few_lng;
  if (a.few_rows) {
    EdArgs f = a;
    f.min_batch = 1;
    const cudaError_t e = ed_wide(a.L) ? launch_ed(k_ed_stream<false, 1, 32, 32>, few_wide, f, 32, slots, blocks, s)
                                       : launch_ed(k_ed_stream<false, 1, 32, kEdWarps>, few_lng, f, kEdWarps, slots, blocks, s);
    if (e != cudaSuccess || a.few_rows == UINT32_MAX) return e;
  }
  if (slots > 1 && a.L <= 256) return launch_ed(k_ed_short<2, 2>, shrt, a, kEdWarps, slots, blocks, s);
  if (slots > 1 && a.L <= kEdShortL) return launch_ed(k_ed_short<4, 2>, shrt2, a, kEdWarps, slots, blocks, s);
  if (ed_wide(a.L)) return launch_ed(k_ed_stream<false, 2, 8, 32>, wide, a, 32, slots, blocks, s);
  if (a.L >= 4096) return launch_ed(k_ed_stream<false, 2, 8, kEdWarps>, lng, a, kEdWarps, slots, blocks, s);
  return launch_ed(k_ed_stream<false, 2, 4, kEdWarps>, mid, a, kEdWarps, slots, blocks, s);
}
cudaError_t launch_ed_stream_row_ids(const EdArgs& a, int slots, int blocks, cudaStream_t s) {
  static SmemLimit lng, mid;
  if (a.L >= 4096) return launch_ed(k_ed_stream<true, 2, 8, 32>, lng, a, 32, slots, blocks, s);
  return launch_ed(k_ed_stream<true, 2, 4, 32>, mid, a, 32, slots, blocks, s);
}
int ed_blocks_per_sm(int L) { return ed_wide(L) ? 1 : kEdBlocksPerSm; }

cudaError_t launch_emit(const unsigned long long* topk, const int* topk_count, int k, float* dist_out,
                        int64_t* id_out, cudaStream_t s) {
  k_emit<<<blocks_for(k, 128), 128, 0, s>>>(topk, topk_count, k, dist_out, id_out);
  return cudaGetLastError();
}

cudaError_t launch_generate_walks(uint64_t seed, uint64_t first, uint64_t n, int L, float* out,
                                  cudaStream_t s, int unit) {
  if (!n) return cudaSuccess;
  k_generate_walks<<<blocks_for(n, 128), 128, 0, s>>>(seed, first, n, L, out, unit);
  return cudaGetLastError();
}

cudaError_t launch_generate_queries(uint64_t seed, const float* data, uint64_t n, int L, int nq,
                                    const double* sigma2, float* out, uint64_t* base_ids, cudaStream_t s, int unit,
                                    uint64_t data_seed) {
  if (!nq) return cudaSuccess;
  k_generate_queries<<<blocks_for(nq, 64), 64, 0, s>>>(seed, data, n, L, nq, sigma2, out, base_ids, unit,
                                                       data_seed);
  return cudaGetLastError();
}

}  // namespace hg
