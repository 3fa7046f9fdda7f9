// cf_cells.cu — the data term, cell by cell: J^T W J / J^T W r (6x6 BSR)
// without atomics, from correspondences sorted by their set of nodes.
//
// The skinning nodes of a correspondence do not change over the GN
// iterations, and on a surface few node sets occur: about 6 per node, with 25
// correspondences each at 150 correspondences per node.  A run of at most 64
// correspondences of one node set is a task.
//
// Once per solve:
//   key_count     per correspondence its key (its distinct nodes, ascending,
//                 as 16-bit local ids) and per sort CTA a histogram of the
//                 keys' first nodes                       (cf_kernels.cu)
//   bin_scan, bin_scatter   stable counting sort by that node  (cf_kernels.cu)
//   bucket_sort   a CTA per node sorts its bucket by the rest of the key and
//                 marks the tasks
//   permute       the correspondences in that order as four float4 streams
//   node lists    per node the tasks that contain it, in position order
// Every GN iteration:
//   cells_kernel  a warp takes 32 sorted correspondences at a time, skins
//                 them, forms their residuals and weights, and sums per task
//                 the 21 products of (u, n) (u, n)^T for the 10 pairs of its
//                 nodes, and the 4 right-hand sides: one record per task
//   gather_kernel two or four warps per block row add the records of the tasks that
//                 contain its node, in position order (Kahan on the diagonal),
//                 expand the upper blocks, add the ARAP terms and the damping
// The products are summed once per node set rather than once per (row, block)
// entry, of which a correspondence has ten, and the gather reads a record per
// task instead of every correspondence of a row.  Per GN iteration on B200 (data
// term + assembly, event times; before: one record per correspondence, gathered
// entry by entry): 2048 nodes, 306k correspondences 37 + 23 us (before 20 + 56),
// 8192 nodes, 1.2M 103 + 62 (46 + 192), 64 problems, 33M 3.1 + 1.57 ms (1.7 + 7.1);
// three CTAs per SM at 80 registers spill (4.0 ms);
// the sort costs 98 us against 80 at 306k and 7 ms against 10 at 33M.  Sets that occur
// once each (no surface has them) leave nothing to sum per set: random ones take
// 530 us a solve at 64 nodes and 20k correspondences (before: 307), 1010 at 2048
// and 300k (687).
// Restates kernels/solver_kernels.cu:52-352 (data term, ARAP, damping).
#include <algorithm>

#include "cf_device.cuh"
#include "cf_internal.h"

namespace cf {

namespace {

constexpr int kWarps = kThreads / 32;
constexpr unsigned kNone = 0xffffu;
constexpr int kSortThreads = 256;
constexpr int kSortMax = 2 * kSortChunk;  // positions of a bucket's first chunk at most
constexpr int kTaskMax = 64;              // correspondences of a task at most

__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
  unsigned long long d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ unsigned long long pack2(float x, float y) {
  unsigned long long d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(x), "f"(y));
  return d;
}
__device__ __forceinline__ float2 unpack2(unsigned long long v) {
  float2 f;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(v));
  return f;
}

// index of (p, q) in the packed upper triangle of a symmetric 3x3
__host__ __device__ constexpr int sym3(int p, int q) {
  return p <= q ? p * 3 - p * (p - 1) / 2 + (q - p) : q * 3 - q * (q - 1) / 2 + (p - q);
}
// where the sums of the pair (a, b), a <= b, of a task's nodes start in its
// record: pairs in the order 00 01 02 03 11 12 13 22 23 33, each 21 sums, the
// diagonal ones followed by the 6 right-hand sides of their node
__host__ __device__ __forceinline__ constexpr int pair_at(int a, int b) {
  return a * 90 - a * (a - 1) / 2 * 21 + (b > a ? 27 + 21 * (b - a - 1) : 0);
}
static_assert(pair_at(0, 1) == 27 && pair_at(1, 1) == 90 && pair_at(2, 2) == 159 && pair_at(3, 3) == 207, "layout");

// A task's sums.  With g = fw w_a w_b, u = (src - x) x n and the normal n, per
// pair (a, b) the 21 sums
//   [0, 6)   S_uu = sum g u u^T (upper triangle: 00 01 02 11 12 22)
//   [6, 15)  S_un = sum g u n^T (row-major)
//   [15, 21) S_nn = sum g n n^T (upper triangle)
// and per node a the 6 sums -sum fw w_a r (u, n).  x is the position of the
// pair's lower node (of a for the right-hand sides).
constexpr int kSums = 21;
static_assert(pair_at(3, 3) + 27 <= kRecFloats, "record layout");

// ----------------------------------------------------------------------------
// sort within a node's bucket
// ----------------------------------------------------------------------------
// Blocks [0, N): node b's first chunk, up to kSortMax positions.  Blocks from
// N on: the chunks of kSortChunk positions at multiples of kSortChunk inside
// buckets that are longer (a bucket of at most kSortChunk is never cut; a cut
// only splits a node set into two tasks).  Bound by the chain of the largest
// bucket's sort (few nodes: 12.7 us per launch at 256 nodes, 15 with every step
// through shared memory; 128 threads instead of 256: 17) and by shared memory
// (33M correspondences: 1.8 ms, 2.3).
__global__ void __launch_bounds__(kSortThreads) bucket_sort_kernel(Table tb, Work w, int N) {
  after_previous();
  __shared__ unsigned long long key[kSortMax];
  __shared__ int cidx[kSortMax];
  const int tid = threadIdx.x;
  int node, q0, q1;
  if ((int)blockIdx.x < N) {
    node = blockIdx.x;
    q0 = w.inc_start[node];
    q1 = min(w.inc_start[node + 1], (q0 + kSortMax) & ~(kSortChunk - 1));
  } else {
    q0 = ((int)blockIdx.x - N + 1) * kSortChunk;
    if (q0 >= w.inc_start[N]) return;
    int lo = 0, hi = N - 1;  // the last node whose bucket starts at or before q0
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (w.inc_start[mid] <= q0) lo = mid; else hi = mid - 1;
    }
    node = lo;
    if (q0 < ((w.inc_start[node] + kSortMax) & ~(kSortChunk - 1))) return;  // in the first chunk
    q1 = min(w.inc_start[node + 1], q0 + kSortChunk);
  }
  const int n = q1 - q0;
  if (n <= 0) return;
  const int node_off = tb.desc[tb.node_prob[node]].node_off;
  int np2 = 32;
  while (np2 < n) np2 <<= 1;
  for (int i = tid; i < np2; i += kSortThreads) {
    unsigned long long k = ~0ull;
    if (i < n) {
      const int c = w.order[q0 + i];
      cidx[i] = c;
      const uint2 kk = w.key[c];
      k = ((unsigned long long)(kk.x >> 16) << 48) | ((unsigned long long)(kk.y & 0xffffu) << 32) |
          ((unsigned long long)(kk.y >> 16) << 16) | (unsigned)i;
    }
    key[i] = k;
  }
  __syncthreads();
  // bitonic; the steps within 32 positions by shuffles, so only those across
  // them pass through shared memory and a barrier
  const int lane = tid & 31;
  auto within = [&](int from, int to) {  // stages from..to of each 32 positions, their steps below 32
    for (int g = tid & ~31; g < np2; g += kSortThreads) {
      unsigned long long x = key[g + lane];
      for (int k = from; k <= to; k <<= 1) {
        const bool up = ((g + lane) & k) == 0;
        for (int j = min(k >> 1, 16); j > 0; j >>= 1) {
          const unsigned long long y = __shfl_xor_sync(0xffffffffu, x, j);
          if ((y < x) == (((lane & j) == 0) == up)) x = y;
        }
      }
      key[g + lane] = x;
    }
    __syncthreads();
  };
  within(2, 32);
  for (int k = 64; k <= np2; k <<= 1) {
    for (int j = k >> 1; j >= 32; j >>= 1) {
      for (int t = tid; t < np2 / 2; t += kSortThreads) {
        const int a = ((t & ~(j - 1)) << 1) | (t & (j - 1)), b = a | j;
        const unsigned long long x = key[a], y = key[b];
        if ((x > y) == ((a & k) == 0)) {
          key[a] = y;
          key[b] = x;
        }
      }
      __syncthreads();
    }
    within(k, k);
  }
  for (int i = tid; i < n; i += kSortThreads) {
    w.task[q0 + i] = 0;
    w.sorted[q0 + i] = cidx[(int)(key[i] & 0xffffu)];
  }
  __syncthreads();
  // the first position of each run of equal node sets cuts it into tasks
  for (int i = tid; i < n; i += kSortThreads) {
    const unsigned long long k = key[i], k48 = k >> 16;
    if (i > 0 && (key[i - 1] >> 16) == k48) continue;
    int b = i + 1, e = n;
    while (b < e) {
      const int mid = (b + e) >> 1;
      if ((key[mid] >> 16) == k48) b = mid + 1; else e = mid;
    }
    const unsigned u1 = (unsigned)(k >> 48), u2 = (unsigned)(k >> 32) & 0xffffu, u3 = (unsigned)(k >> 16) & 0xffffu;
    const bool none = u1 == kNone - 1;  // no valid node at all
    int4 ids;
    ids.x = none ? -1 : node;
    ids.y = none || u1 == kNone ? -1 : (int)u1 + node_off;
    ids.z = u2 == kNone ? -1 : (int)u2 + node_off;
    ids.w = u3 == kNone ? -1 : (int)u3 + node_off;
    const int tasks = (b - i + kTaskMax - 1) / kTaskMax;
    for (int t = 0, at = i; t < tasks; t++, at += kTaskMax) {
      w.task[q0 + at] = (unsigned char)min(kTaskMax, b - at);
      w.cell_ids[q0 + at] = ids;
    }
    if (ids.x >= 0) atomicAdd(w.cl_total + ids.x, tasks);
    if (ids.y >= 0) atomicAdd(w.cl_total + ids.y, tasks);
    if (ids.z >= 0) atomicAdd(w.cl_total + ids.z, tasks);
    if (ids.w >= 0) atomicAdd(w.cl_total + ids.w, tasks);
  }
}

// A warp per 32 sorted positions: their correspondences' words by consecutive
// lanes, through shared memory, all loads in flight; written as the four
// streams.  Bound by the gather of 76 + 12 B per correspondence.  The tasks
// that start here enter their nodes' lists (in any order; list_sort follows).
// A list entry: the task's first position << 2 | its size if below kRecMin
// (its correspondences are read one by one), else 0 (it has a record).
constexpr int kPermThreads = 128;
__global__ void __launch_bounds__(kPermThreads) permute_kernel(Table tb, Work w) {
  after_previous();
  __shared__ float stage[kPermThreads / 32][32 * 23];
  const int lane = lane_id(), wid = threadIdx.x >> 5;
  const int q0 = (blockIdx.x * (kPermThreads / 32) + wid) * 32;
  const int total = w.inc_start[tb.N];
  if (q0 >= total) return;
  const int m = min(32, total - q0);
  const int c = lane < m ? w.sorted[q0 + lane] : 0;
  const int size = lane < m ? w.task[q0 + lane] : 0;
  if (size) {
    const int4 ids = w.cell_ids[q0 + lane];
    const int e = ((q0 + lane) << 2) | (size < kRecMin ? size : 0);
    if (ids.x >= 0) w.clist[atomicAdd(w.cl_cur + ids.x, 1)] = e;
    if (ids.y >= 0) w.clist[atomicAdd(w.cl_cur + ids.y, 1)] = e;
    if (ids.z >= 0) w.clist[atomicAdd(w.cl_cur + ids.z, 1)] = e;
    if (ids.w >= 0) w.clist[atomicAdd(w.cl_cur + ids.w, 1)] = e;
  }
  // the problem of each correspondence (one for the warp, but at a boundary)
  int prob = 0;
  if (tb.P > 1) {
    int lo = 0, hi = tb.P - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (tb.desc[mid].corr_off <= c) lo = mid; else hi = mid - 1;
    }
    prob = lo;
  }
  const ProbDesc& d = tb.desc[prob];
  const unsigned long long rec = reinterpret_cast<unsigned long long>(d.corrs + (c - d.corr_off));
  const unsigned long long can = d.canon ? reinterpret_cast<unsigned long long>(d.canon + 3 * (size_t)(c - d.corr_off)) : 0ull;
  const uint2 kk = lane < m ? w.key[c] : make_uint2(~0u, ~0u);
  float* st = stage[wid];
  {
    float v[22];
#pragma unroll
    for (int h = 0; h < 19; h++) {
      const int f = 32 * h + lane, e = f / 19;
      const unsigned long long base = __shfl_sync(0xffffffffu, rec, e);
      v[h] = f < 19 * m ? __ldg(reinterpret_cast<const float*>(base) + (f - 19 * e)) : 0.f;
    }
#pragma unroll
    for (int h = 0; h < 3; h++) {
      const int f = 32 * h + lane, e = f / 3;
      const unsigned long long base = __shfl_sync(0xffffffffu, can, e);
      v[19 + h] = f < 3 * m && base ? __ldg(reinterpret_cast<const float*>(base) + (f - 3 * e)) : 0.f;
    }
#pragma unroll
    for (int h = 0; h < 19; h++) {
      const int f = 32 * h + lane, e = f / 19;
      st[e * 23 + f - 19 * e] = v[h];
    }
#pragma unroll
    for (int h = 0; h < 3; h++) {
      const int f = 32 * h + lane, e = f / 3;
      st[e * 23 + 19 + f - 3 * e] = v[19 + h];
    }
  }
  __syncwarp();
  if (lane >= m) return;
  const float* r = st + lane * 23;
  // Per slot, which of the key's nodes it names (3 bits; 7: none), and the sum
  // of each node's weights.  A node that a later slot names again (codes 4..6,
  // which node in bits 12 + 2 s, bit 20: there are such) is blended again there,
  // with that slot's weight, which goes to one of the entries past the last node.
  const unsigned u0 = kk.x & 0xffffu, u1 = kk.x >> 16, u2 = kk.y & 0xffffu, u3 = kk.y >> 16;
  float uw[4] = {0.f, 0.f, 0.f, 0.f};
  unsigned perm = 0, seen = 0, spare = 1u + (u1 != kNone) + (u2 != kNone) + (u3 != kNone);
#pragma unroll
  for (int s = 0; s < kK; s++) {
    const int id = __float_as_int(r[9 + s]);
    const float ws = r[13 + s];
    unsigned p = 7u;
    if (id >= 0 && id < d.N && !(ws < 1e-8f)) {
      const unsigned at = (unsigned)id == u0 ? 0u : (unsigned)id == u1 ? 1u : (unsigned)id == u2 ? 2u : 3u;
      p = at;
      const bool again = (seen >> at) & 1u;
      if (again) {
        perm |= 1u << 20 | at << (12 + 2 * s);
        p = 3u + spare;
      }
      seen |= 1u << at;
#pragma unroll
      for (unsigned a = 0; a < 4; a++) {
        uw[a] += a == at ? ws : 0.f;
        if (again && a == spare) uw[a] = ws;
      }
      spare += again ? 1u : 0u;
    }
    perm |= p << (3 * s);
  }
  const bool canon = d.canon != nullptr;
  const int q = q0 + lane;
  w.sp_src[q] = make_float4(canon ? r[19] : r[0], canon ? r[20] : r[1], canon ? r[21] : r[2], r[17]);
  w.sp_dst[q] = make_float4(r[3], r[4], r[5], __uint_as_float(perm));
  w.sp_nrm[q] = make_float4(r[6], r[7], r[8], 0.f);
  w.sp_uw[q] = make_float4(uw[0], uw[1], uw[2], uw[3]);
}

// ----------------------------------------------------------------------------
// node lists
// ----------------------------------------------------------------------------
// What the gather needs of a list entry e of node r: where the run of r's sums
// starts in the task's record, r's place a among the task's nodes | raw
// correspondences << 2, and the off-diagonal upper block of row r that each of
// the nodes after a belongs to, 21 bits each (kNoBlock: none; find_block < 0
// drops the pair, as in kernels/solver_kernels.cu:123-125).
constexpr unsigned kNoBlock = 0x1fffffu;
__device__ __forceinline__ uint4 list_desc(const Work& w, const Pattern& pt, int r, int e) {
  const int4 ids = __ldg(w.cell_ids + (e >> 2));
  const int a = ids.x == r ? 0 : ids.y == r ? 1 : ids.z == r ? 2 : 3;
  const int4* meta = pt.upper_meta + pt.ustart[r] + 1;
  const int nu = pt.ustart[r + 1] - pt.ustart[r] - 1;
  unsigned long long kb = 0;
#pragma unroll
  for (int b = 0; b < 3; b++) {
    const int c = a + 1 + b < 4 ? sel4i(ids, a + 1 + b) : -1;
    unsigned at = kNoBlock;
    if (c >= 0) {
      int lo = 0, hi = nu;  // columns ascend
      while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (__ldg(&meta[mid].z) < c) lo = mid + 1; else hi = mid;
      }
      if (lo < nu && __ldg(&meta[lo].z) == c) at = (unsigned)lo;
    }
    kb |= (unsigned long long)at << (21 * b);
  }
  const unsigned run = (unsigned)((e >> 2) + kRecMin - 1) / kRecMin * kRecFloats + pair_at(a, a);
  return make_uint4((e & 3) ? (unsigned)(e >> 2) : run, (unsigned)a | (unsigned)(e & 3) << 2, (unsigned)kb,
                    (unsigned)(kb >> 32));
}

// Puts each node's list in position order (its entries came in any order; the
// gather's sums follow it) and describes its entries.  A warp per node up to
// 64 tasks, by rank; the CTA together for the others, one after another, so a CTA
// has no more nodes (`per`, at most one per warp) than about 1024 CTAs need: 64 nodes
// with 1250 tasks each take 29 us, 205 with eight to a CTA.
constexpr int kListSmem = 4096;
__global__ void __launch_bounds__(kThreads) list_sort_kernel(Work w, Pattern pt, int N, int per) {
  after_previous();
  __shared__ int big[kWarps];
  __shared__ int buf[kListSmem];
  const int lane = lane_id(), wid = threadIdx.x >> 5;
  const int node = blockIdx.x * per + wid;
  int n = 0, b0 = 0;
  if (wid < per && node < N) {
    b0 = w.cl_start[node];
    n = w.cl_start[node + 1] - b0;
  }
  if (n > 0 && n <= 64) {
    int* list = w.clist + b0;
    const int x = lane < n ? list[lane] : 0x7fffffff, y = lane + 32 < n ? list[lane + 32] : 0x7fffffff;
    int rx = 0, ry = 0;
    for (int k = 0; k < min(n, 32); k++) {
      const int v = __shfl_sync(0xffffffffu, x, k);
      rx += v < x;
      ry += v < y;
    }
    for (int k = 32; k < n; k++) {
      const int v = __shfl_sync(0xffffffffu, y, k - 32);
      rx += v < x;
      ry += v < y;
    }
    __syncwarp();
    if (lane < n) {
      list[rx] = x;
      w.cdesc[b0 + rx] = list_desc(w, pt, node, x);
    }
    if (lane + 32 < n) {
      list[ry] = y;
      w.cdesc[b0 + ry] = list_desc(w, pt, node, y);
    }
  }
  if (lane == 0) big[wid] = n > 64 ? node : -1;
  __syncthreads();
  for (int v = 0; v < per; v++) {
    const int nd = big[v];
    if (nd < 0) continue;
    const int b = w.cl_start[nd], m = w.cl_start[nd + 1] - b;
    int* g = w.clist + b;
    int* a = m <= kListSmem ? buf : g;
    if (m <= kListSmem) {
      for (int i = threadIdx.x; i < m; i += kThreads) buf[i] = g[i];
      __syncthreads();
    }
    int np2 = 64;
    while (np2 < m) np2 <<= 1;
    // bitonic over np2 slots of which those from m on hold +inf and stay put:
    // every comparator is written ascending (the first step of a stage mirrors)
    for (int k = 2; k <= np2; k <<= 1)
      for (int j = k >> 1; j > 0; j >>= 1) {
        const bool mirror = j == (k >> 1);
        for (int t = threadIdx.x; t < np2 / 2; t += kThreads) {
          const int lo = ((t & ~(j - 1)) << 1) | (t & (j - 1));
          const int hi = mirror ? (lo | (k - 1)) - (lo & (k - 1)) : lo | j;
          if (hi < m) {
            const int x = a[lo], y = a[hi];
            if (x > y) {
              a[lo] = y;
              a[hi] = x;
            }
          }
        }
        __syncthreads();
      }
    for (int i = threadIdx.x; i < m; i += kThreads) {
      const int x = a[i];
      if (a == buf) g[i] = x;
      w.cdesc[b + i] = list_desc(w, pt, nd, x);
    }
    __syncthreads();
  }
}

// ----------------------------------------------------------------------------
// ARAP edges
// ----------------------------------------------------------------------------
struct EdgeArgs {
  const int* edge_ijk;
  int n_edges;
  const cf_deform_node* nodes;
  const cf_dual_quat* T;
  float lambda, arap_sgn;
  float4* out;     // [kEdgeTerms4 * n_edges]
  double* energy;  // [n_edges]
  int edge_ctas;   // the launch's first CTAs
  int stats;       // per task the residual statistics of the features
};

__device__ __forceinline__ int tri6(int p, int q) { return p * 6 - p * (p - 1) / 2 + (q - p); }

// Every ARAP edge (i, j) at the current
// transforms (kernels/solver_kernels.cu:202-352: strain and Huber weight,
// residual r, Jacobians J_i, J_j of both endpoints), written as its complete
// contributions for the assembly: the diagonal blocks of i and j (upper
// triangle el J J^T and rhs -+el J r, 27 + pad floats each), the
// off-diagonal block -el J_i J_j^T (36 floats) and the energy el |r|^2 (FP64).
__device__ void edge_terms_cta(const EdgeArgs& ea, int cta) {
  const int ed = cta * kThreads + threadIdx.x;
  if (ed >= ea.n_edges) return;
  const Edge ev = eval_edge(ea.nodes, ea.T, ea.edge_ijk[3 * ed], ea.edge_ijk[3 * ed + 1], ea.edge_ijk[3 * ed + 2],
                            ea.lambda);
  float Ji[6][3], Jj[6][3];
  arap_jac(ev.qi, ea.arap_sgn, Ji);
  arap_jac(ev.qj, ea.arap_sgn, Jj);
  const float rr[3] = {ev.r.x, ev.r.y, ev.r.z};
  float4* out = ea.out + (size_t)kEdgeTerms4 * ed;
  // one output vector at a time: the Jacobians stay in registers, the terms do not
#pragma unroll
  for (int h = 0; h < 2; h++) {
    float dv[28];
#pragma unroll
    for (int p = 0; p < 6; p++) {
      const float* P = h ? Jj[p] : Ji[p];
#pragma unroll
      for (int q = p; q < 6; q++) {
        const float* Q = h ? Jj[q] : Ji[q];
        float t = 0.f;
        t += P[0] * Q[0];
        t += P[1] * Q[1];
        t += P[2] * Q[2];
        dv[tri6(p, q)] = ev.el * t;
      }
      float t = 0.f;
      t += P[0] * rr[0];
      t += P[1] * rr[1];
      t += P[2] * rr[2];
      dv[21 + p] = (h ? ev.el : -ev.el) * t;
    }
    dv[27] = 0.f;
#pragma unroll
    for (int k = 0; k < 7; k++)
      out[7 * h + k] = make_float4(dv[4 * k], dv[4 * k + 1], dv[4 * k + 2], dv[4 * k + 3]);
  }
  float o[36];
#pragma unroll
  for (int p = 0; p < 6; p++)
#pragma unroll
    for (int q = 0; q < 6; q++) {
      float t = 0.f;
      t += Ji[p][0] * Jj[q][0];
      t += Ji[p][1] * Jj[q][1];
      t += Ji[p][2] * Jj[q][2];
      o[p * 6 + q] = -ev.el * t;
    }
#pragma unroll
  for (int k = 0; k < 9; k++) out[14 + k] = make_float4(o[4 * k], o[4 * k + 1], o[4 * k + 2], o[4 * k + 3]);
  ea.energy[ed] =
      ev.el > 0.f ? (double)ev.el * ((double)rr[0] * rr[0] + (double)rr[1] * rr[1] + (double)rr[2] * rr[2]) : 0.0;
}

// ----------------------------------------------------------------------------
// energies
// ----------------------------------------------------------------------------
// Sum of p[0..n) by `stride` threads starting at `t`, in a fixed order per
// thread, with 8 loads in flight at a time.
__device__ __forceinline__ double strided_sum(const double* p, int n, int t, int stride) {
  double v = 0.0;
  for (int k0 = t; k0 < n; k0 += 8 * stride) {
    double x[8];
#pragma unroll
    for (int b = 0; b < 8; b++) x[b] = k0 + b * stride < n ? __ldcg(p + k0 + b * stride) : 0.0;
#pragma unroll
    for (int b = 0; b < 8; b++)
      if (k0 + b * stride < n) v += x[b];
  }
  return v;
}

// A problem's energy into its statistics: the sum of its n partials, by one
// warp.  slot < 0: an energy that the learned solve's gate compares; kNoSlot: for nobody.
__device__ __forceinline__ void reduce_energy(const Work& w, const double* part, int n, int prob, int slot) {
  double v = strided_sum(part, n, threadIdx.x & 31, 32);
  v = warp_sum_d(v);
  if ((threadIdx.x & 31) == 0 && slot != kNoSlot) {
    if (slot >= 0) {
      w.stats[prob].energy[slot] = v;
      if (!isfinite(v)) atomicOr(w.err, kErrNonFinite);
    } else {
      w.stats[prob].gate[-slot - 1] = v;
    }
  }
}
__global__ void energy_reduce_kernel(Table tb, Work w, int slot) {
  after_previous();
  const ProbDesc d = tb.desc[blockIdx.x];
  reduce_energy(w, w.e_data_part + d.e_cta0, d.e_ctas, blockIdx.x, slot);
}

// ----------------------------------------------------------------------------
// cells
// ----------------------------------------------------------------------------
// Lane v < 21: the two of (u, n) whose product sum v adds; lanes 21..26: the
// component of the right-hand side.
__device__ __forceinline__ void product_of(int v, int& i, int& j) {
  if (v < 6) {
    i = v < 3 ? 0 : v < 5 ? 1 : 2;
    j = v < 3 ? v : v < 5 ? v - 2 : 2;
  } else if (v < 15) {
    i = (v - 6) / 3;
    j = 3 + (v - 6) % 3;
  } else if (v < kSums) {
    i = v < 18 ? 3 : v < 20 ? 4 : 5;
    j = v < 18 ? v - 12 : v < 20 ? v - 14 : 5;
  } else {
    i = v < 27 ? v - kSums : 0;
    j = 0;
  }
}
// Per correspondence: 10 weights g, 4 right-hand factors at 12, the 21
// products of (u, n) at 16 and (u, n) itself at 38.
constexpr int kStageWords = 44;
constexpr int kSumStride = 22;           // a pair's sums while the task is closed
constexpr int kRhsAt = 10 * kSumStride;  // then [4][6] right-hand sides
constexpr int kUnAt = kRhsAt + 24;       // and [6][9] moved S_un
struct WarpMem {
  float stage[32 * kStageWords];
  float sum[kUnAt + 56];  // (two of padding: 16-byte rows)
  float e[32][12];  // at the first lane of each task: x_0 - x_a of its other nodes
};
static_assert(sizeof(WarpMem) % 16 == 0, "16-byte rows");
constexpr int kCellsSmem = kWarps * (int)sizeof(WarpMem);

// blend_warp (cf_device.cuh) over the nodes of the task, in the order of the
// correspondence's slots; the four nodes' loads are issued together.  A node
// that two slots name enters at both places: the sign that it gets at the second
// depends on what was blended in between.
__device__ __forceinline__ float3 blend_cell(float3 p, unsigned perm, const float4& uw, const int4& ids,
                                             const cf_dual_quat* plain) {
  float4 br = make_float4(0.f, 0.f, 0.f, 0.f), bd = br;
  float wsum = 0.f;
  auto add = [&](const DQ& q, float w) {
    wsum += w;
    const float s = qdot(q.r, br) < 0.f ? -w : w;
    br.x += s * q.r.x; br.y += s * q.r.y; br.z += s * q.r.z; br.w += s * q.r.w;
    bd.x += s * q.d.x; bd.y += s * q.d.y; bd.z += s * q.d.z; bd.w += s * q.d.w;
  };
  if (perm >> 20) {  // slot by slot; uw has the sum of a node's weights, so the first slot's is what the others leave
#pragma unroll 1
    for (int k = 0; k < kK; k++) {
      const int c = (perm >> (3 * k)) & 7, a = c < 4 ? c : (perm >> (12 + 2 * k)) & 3;
      if (c == 7) continue;
      float w = sel4(uw, c < 4 ? c : c - 3);
      if (c < 4)
#pragma unroll 1
        for (int j = k + 1; j < kK; j++) {
          const int cj = (perm >> (3 * j)) & 7;
          if (cj >= 4 && cj < 7 && (int)((perm >> (12 + 2 * j)) & 3) == a) w -= sel4(uw, cj - 3);
        }
      add(load_dq(plain + sel4i(ids, a)), w);
    }
  } else {
    DQ q[kK];
    float wt[kK];
#pragma unroll
    for (int k = 0; k < kK; k++) {
      const int a = (perm >> (3 * k)) & 7;
      q[k].r = q[k].d = make_float4(0.f, 0.f, 0.f, 0.f);
      wt[k] = 0.f;
      if (a < 4) {
        q[k] = load_dq(plain + sel4i(ids, a));
        wt[k] = sel4(uw, a);
      }
    }
#pragma unroll
    for (int k = 0; k < kK; k++) add(q[k], wt[k]);
  }
  if (wsum < 1e-8f) return p;
  DQ b;
  b.r = br;
  b.d = bd;
  return dq_transform_point(dq_normalize(b), p);
}

// Closes a task: the half-warps' sums together, moved to each pair's lower
// node, into the task's record.  u_a = u + e x n with e = x_0 - x_a, so with
// E = [e]_x (row p: -e(p2) at column p1, e(p1) at column p2)
//   S_un' = S_un + E S_nn,  S_uu' = S_uu + S_un E^T + E S_un'^T,
// and a right-hand side's u part gains E times its n part.
__device__ __forceinline__ void close_task(const unsigned long long (&acc)[10], WarpMem& m, const float* e,
                                           float* rec, int lane, int p, int r) {
  const int hl = lane & 15, half = lane >> 4;
  float* S = m.sum;
  // half 0 keeps the weights 0..3 and 8 (of its two columns), half 1 4..7 and 9
  float v[10];
#pragma unroll
  for (int t = 0; t < 2; t++) {
    const float2 a0 = unpack2(acc[5 * t]), a1 = unpack2(acc[5 * t + 1]), a2 = unpack2(acc[5 * t + 2]),
                 a3 = unpack2(acc[5 * t + 3]), a4 = unpack2(acc[5 * t + 4]);
    const float lo[5] = {a0.x, a0.y, a1.x, a1.y, a4.x}, hi[5] = {a2.x, a2.y, a3.x, a3.y, a4.y};
#pragma unroll
    for (int k = 0; k < 5; k++) {
      const float send = half ? lo[k] : hi[k], keep = half ? hi[k] : lo[k];
      v[5 * t + k] = keep + __shfl_xor_sync(0xffffffffu, send, 16);
    }
  }
  if (hl < 11) {
#pragma unroll
    for (int k = 0; k < 4; k++)
      *reinterpret_cast<float2*>(S + (4 * half + k) * kSumStride + 2 * hl) = make_float2(v[k], v[5 + k]);
    *reinterpret_cast<float2*>(S + (8 + half) * kSumStride + 2 * hl) = make_float2(v[4], v[9]);
  } else if (hl < 14 && !half) {
#pragma unroll
    for (int k = 0; k < 4; k++)
      *reinterpret_cast<float2*>(S + kRhsAt + 6 * k + 2 * (hl - 11)) = make_float2(v[k], v[5 + k]);
  }
  __syncwarp();
  const int p1 = p == 2 ? 0 : p + 1, p2 = p == 0 ? 2 : p - 1;
  float c1[3], c2[3];
#pragma unroll
  for (int a = 0; a < 3; a++) {
    c1[a] = -e[3 * a + p2];
    c2[a] = e[3 * a + p1];
  }
  constexpr int kLow[6] = {0, 0, 0, 1, 1, 2};  // a - 1 of the pairs 11 12 13 22 23 33
  if (lane < kSums) {
#pragma unroll
    for (int k = 0; k < 10; k++) v[k] = S[k * kSumStride + lane];
  } else if (lane < 27) {
#pragma unroll
    for (int k = 0; k < 4; k++) v[k] = S[kRhsAt + 6 * k + lane - kSums];
  }
  if (lane >= 6 && lane < 15) {
    const int i1 = 15 + sym3(p1, r), i2 = 15 + sym3(p2, r);
#pragma unroll
    for (int k = 0; k < 6; k++) {
      const float* P = S + (4 + k) * kSumStride;
      v[4 + k] += c1[kLow[k]] * P[i1] + c2[kLow[k]] * P[i2];
      S[kUnAt + k * 9 + lane - 6] = v[4 + k];
    }
  } else if (lane >= kSums && lane < kSums + 3) {
#pragma unroll
    for (int a = 0; a < 3; a++) {
      const float* P = S + kRhsAt + 6 * (a + 1) + 3;
      v[a + 1] += c1[a] * P[p1] + c2[a] * P[p2];
    }
  }
  __syncwarp();
  if (lane < 6) {
    const int r1 = r == 2 ? 0 : r + 1, r2 = r == 0 ? 2 : r - 1;
#pragma unroll
    for (int k = 0; k < 6; k++) {
      const float d1 = -e[3 * kLow[k] + r2], d2 = e[3 * kLow[k] + r1];
      const float *P = S + (4 + k) * kSumStride + 6 + 3 * p, *Q = S + kUnAt + k * 9 + 3 * r;
      v[4 + k] += d1 * P[r1] + d2 * P[r2] + c1[kLow[k]] * Q[p1] + c2[kLow[k]] * Q[p2];
    }
  }
  rec += lane;
  if (lane < kSums) {
    int k = 0;
#pragma unroll
    for (int a = 0; a < 4; a++)
#pragma unroll
      for (int b = a; b < 4; b++) rec[pair_at(a, b)] = v[k++];
  } else if (lane < 27) {
#pragma unroll
    for (int a = 0; a < 4; a++) rec[pair_at(a, a)] = v[a];
  }
  __syncwarp();
}

// Warp `gw` of the problem's e_ctas * 8 takes the tasks that start in an equal
// share of its sorted positions, 32 positions at a time: a lane per position
// first (skinning, residual, weights, the 21 products, into shared memory),
// then per task the half-warps over its even and odd correspondences, a lane
// owning two of the products and their sums for the 10 pairs.  Sums of a task
// that goes on in the next 32 positions stay in registers.  kAcc: the records
// (and the raw records of small tasks); otherwise the energy alone, with the
// problem's ARAP edges.
template <bool kSkin, bool kAcc>
__global__ void __launch_bounds__(kThreads, kAcc ? 2 : 3) cells_kernel(Table tb, Work w, Pattern pt, EdgeArgs ea, int slot) {
  extern __shared__ __align__(16) unsigned char cells_smem[];
  __shared__ double red[kWarps];
  if (kAcc && (int)blockIdx.x < ea.edge_ctas) {
    after_previous();
    edge_terms_cta(ea, blockIdx.x);
    return;
  }
  const int lane = lane_id(), wid = threadIdx.x >> 5;
  const int cta = kAcc ? blockIdx.x - ea.edge_ctas : blockIdx.x;
  // (a single problem's share needs no table: one load instead of three in a row)
  int prob = 0, lc = cta, e_ctas = kAcc ? tb.n_e : (int)gridDim.x, n0 = 0, n1 = tb.N;
  if (tb.P > 1) {
    prob = tb.e_prob[cta];
    const ProbDesc& d = tb.desc[prob];
    lc = cta - d.e_cta0;
    e_ctas = d.e_ctas;
    n0 = d.node_off;
    n1 = n0 + d.N;
  }
  const int s0 = n0 ? w.inc_start[n0] : 0;
  const long long mp = w.inc_start[n1] - s0;
  const int gw = lc * kWarps + wid, gt = e_ctas * kWarps;
  const int qa = s0 + (int)(mp * gw / gt), qb = s0 + (int)(mp * (gw + 1) / gt);
  WarpMem& m = reinterpret_cast<WarpMem*>(cells_smem)[wid];
  double energy = 0.0;
  int li, lj;
  product_of(lane, li, lj);
  // the lane's row p and column r of S_uu or S_un, or its row of a right-hand side
  const int p = lane < 15 ? li : lane >= kSums && lane < kSums + 3 ? lane - kSums : 0;
  const int r = lane < 15 ? lj % 3 : 0;
  const int hl = lane & 15, half = lane >> 4;
  const float* colp = m.stage + half * kStageWords + (hl < 11 ? 16 + 2 * hl : hl < 14 ? 38 + 2 * (hl - 11) : 16);
  const float* wgtp = m.stage + half * kStageWords + (hl < 11 ? 0 : 12);
  unsigned long long acc[10];
#pragma unroll
  for (int k = 0; k < 10; k++) acc[k] = 0ull;
  // One window ahead: its streams and its tasks' nodes are loaded while the
  // products of the current one are summed, and the task sizes one window
  // before that.  Loads that are used once go past L1, which keeps the nodes.
  auto sizes = [&](int q) { return q + lane < qb ? (int)__ldcg(w.task + q + lane) : 0; };
  int open = -1, osize = 0, left = 0;  // the task that goes on from the window before: start, size, what is left
  // the share's first task (the positions before it belong to the warp before)
  int w0 = qa, size = sizes(w0), size1 = sizes(w0 + 32);
  for (unsigned starts = 0; w0 < qb; w0 += 32) {
    starts = __ballot_sync(0xffffffffu, size > 0);
    if (starts) {
      const int f = __ffs(starts) - 1, from = (lane + f) & 31;
      const int x = __shfl_sync(0xffffffffu, size, from), y = __shfl_sync(0xffffffffu, size1, from);
      size = lane + f < 32 ? x : y;
      w0 += f;
      size1 = sizes(w0 + 32);
      break;
    }
    size = size1;
    size1 = sizes(w0 + 64);
  }
  unsigned heads;
  int hd, hs, hq;
  bool on;
  float4 sv, dv, nv, uw;
  int4 ids;
  float rs = 0.f, rm = 0.f, rc = 0.f;
  // the window at q0 of the given task sizes: each lane's task, and its loads
  auto enter = [&](int q0, int sz) {
    heads = __ballot_sync(0xffffffffu, sz > 0);
    const unsigned upto = heads & (0xffffffffu >> (31 - lane));
    hd = upto ? 31 - __clz(upto) : -1;  // the lane whose position starts this one's task
    hs = __shfl_sync(0xffffffffu, sz, max(hd, 0));
    on = hd >= 0 ? lane < hd + hs : lane < left;
    hq = hd >= 0 ? q0 + hd : open;
    hs = hd >= 0 ? hs : osize;
    if (on) {
      sv = __ldcg(w.sp_src + q0 + lane);
      dv = __ldcg(w.sp_dst + q0 + lane);
      nv = __ldcg(w.sp_nrm + q0 + lane);
      uw = __ldcg(w.sp_uw + q0 + lane);
      ids = __ldg(w.cell_ids + hq);
    }
  };
  enter(w0, size);
  // read already: the sorted streams, task sizes and nodes (bucket_sort and permute;
  // list_sort lies between); from here on the transforms, positions and records
  after_previous();
  for (; w0 < qb || left > 0; w0 += 32) {
    const int q = w0 + lane;
    float3 src = f3(0.f, 0.f, 0.f);
    float4 x0 = make_float4(0.f, 0.f, 0.f, 0.f);
    float res = 0.f, fw = 0.f;
    if (on) {
      if (kAcc && ids.x >= 0) x0 = __ldg(w.npos + ids.x);
      src = f3(sv.x, sv.y, sv.z);
      if (kSkin) src = blend_cell(src, __float_as_uint(dv.w), uw, ids, w.plain);
      // kernels/solver_kernels.cu:76-85
      res = nv.x * (src.x - dv.x) + nv.y * (src.y - dv.y) + nv.z * (src.z - dv.z);
      fw = fmaxf(sv.w, 0.f) * huber_w(res, 0.2f);
      if (!(fw > 1e-8f)) fw = 0.f;
      else energy += (double)fw * (double)res * (double)res;
    }
    const unsigned heads0 = heads;
    const int open0 = open, osize0 = osize, left0 = left, size0 = size;
    {  // what goes on into the next window
      const int end = heads ? 31 - __clz(heads) : 0;
      const int es = __shfl_sync(0xffffffffu, size, end);
      left = heads ? max(0, end + es - 32) : max(0, left - 32);
      open = heads ? w0 + end : open;
      osize = heads ? es : osize;
    }
    const bool rec_task = hs >= kRecMin, first_lane = lane == max(hd, 0);
    if (!kAcc) {
      if (ea.stats) {  // the features' residual statistics of each task: sum, maximum, count of |r|
        int first = 0, last = left0, start = open0;
        for (unsigned todo = heads0; last > first || todo;) {
          if (last <= first) {
            first = __ffs(todo) - 1;
            todo &= todo - 1;
            last = first + __shfl_sync(0xffffffffu, size0, first);
            start = w0 + first;
          }
          const bool mine = lane >= first && lane < last && fw > 0.f;
          float t = mine ? fabsf(res) : 0.f;
          rs += warp_sum_f(t);
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) t = fmaxf(t, __shfl_xor_sync(0xffffffffu, t, o));
          rm = fmaxf(rm, t);
          rc += (float)__popc(__ballot_sync(0xffffffffu, mine));
          if (last > 32) break;  // goes on in the next window
          if (lane == 0) w.cstat[start] = make_float4(rs, rm, rc, 0.f);
          rs = rm = rc = 0.f;
          first = last = 0;
        }
      }
      size = size1;
      enter(w0 + 32, size);
      size1 = sizes(w0 + 64);
      continue;
    }
    if (on) {
      if (rec_task) {
        float3 u = f3(0.f, 0.f, 0.f), nn = u;
        if (fw > 0.f) {
          nn = f3(nv.x, nv.y, nv.z);
          u = cross3(f3(src.x - x0.x, src.y - x0.y, src.z - x0.z), nn);
        }
        const float wa = uw.x > 1e-8f ? uw.x : 0.f, wb = uw.y > 1e-8f ? uw.y : 0.f, wc = uw.z > 1e-8f ? uw.z : 0.f,
                    wd = uw.w > 1e-8f ? uw.w : 0.f;
        const float ga = fw * wa, gb = fw * wb, gc = fw * wc, gd = fw * wd;
        const float t = fw > 0.f ? -res : 0.f;
        float4* s4 = reinterpret_cast<float4*>(m.stage + lane * kStageWords);
        s4[0] = make_float4(ga * wa, ga * wb, ga * wc, ga * wd);
        s4[1] = make_float4(gb * wb, gb * wc, gb * wd, gc * wc);
        s4[2] = make_float4(gc * wd, gd * wd, 0.f, 0.f);
        s4[3] = make_float4(ga * t, gb * t, gc * t, gd * t);
        s4[4] = make_float4(u.x * u.x, u.x * u.y, u.x * u.z, u.y * u.y);
        s4[5] = make_float4(u.y * u.z, u.z * u.z, u.x * nn.x, u.x * nn.y);
        s4[6] = make_float4(u.x * nn.z, u.y * nn.x, u.y * nn.y, u.y * nn.z);
        s4[7] = make_float4(u.z * nn.x, u.z * nn.y, u.z * nn.z, nn.x * nn.x);
        s4[8] = make_float4(nn.x * nn.y, nn.x * nn.z, nn.y * nn.y, nn.y * nn.z);
        s4[9] = make_float4(nn.z * nn.z, 0.f, u.x, u.y);
        s4[10] = make_float4(u.z, nn.x, nn.y, nn.z);
        if (first_lane) {
          float4 x[3];
#pragma unroll
          for (int a = 0; a < 3; a++) {
            const int id = sel4i(ids, a + 1);
            x[a] = id >= 0 ? __ldg(w.npos + id) : x0;
          }
#pragma unroll
          for (int a = 0; a < 3; a++) {
            m.e[lane][3 * a] = x0.x - x[a].x;
            m.e[lane][3 * a + 1] = x0.y - x[a].y;
            m.e[lane][3 * a + 2] = x0.z - x[a].z;
          }
        }
      } else {
        w.raw[q] = make_float4(src.x, src.y, src.z, fw);
        w.sp_nrm[q].w = res;
      }
    }
    // the next window's loads
    size = size1;
    enter(w0 + 32, size);
    size1 = sizes(w0 + 64);
    __syncwarp();
    // the tasks one by one: first the one that goes on, then those that start here
    unsigned todo = heads0;
    int first = 0, last = left0, start = open0, full = osize0;  // lanes [first, last) (last may lie past the 32)
    if (left0 <= 0 && todo) {
      const int t = __ffs(todo) - 1;
      todo &= todo - 1;
      first = t;
      full = __shfl_sync(0xffffffffu, size0, t);
      last = t + full;
      start = w0 + t;
    }
    while (last > first) {
      const int n = min(last, 32) - first;
      const bool has_rec = full >= kRecMin;
      if (has_rec) {
        const float *cp = colp + first * kStageWords, *wp = wgtp + first * kStageWords;
        const float* wq = m.stage + (first + half) * kStageWords;
        int j = half;
#pragma unroll 4  // (2: 3.21 ms against 3.10 at 33M correspondences; 8: the same as 4)
        for (; j < (n & ~1); j += 2, cp += 2 * kStageWords, wp += 2 * kStageWords, wq += 2 * kStageWords) {
          const float2 L = *reinterpret_cast<const float2*>(cp);
          const ulonglong2 g01 = *reinterpret_cast<const ulonglong2*>(wp);
          const ulonglong2 g23 = *reinterpret_cast<const ulonglong2*>(wq + 4);
          const unsigned long long g4 = *reinterpret_cast<const unsigned long long*>(wq + 8);
          const unsigned long long A = pack2(L.x, L.x), B = pack2(L.y, L.y);
          acc[0] = fma2(A, g01.x, acc[0]);
          acc[1] = fma2(A, g01.y, acc[1]);
          acc[2] = fma2(A, g23.x, acc[2]);
          acc[3] = fma2(A, g23.y, acc[3]);
          acc[4] = fma2(A, g4, acc[4]);
          acc[5] = fma2(B, g01.x, acc[5]);
          acc[6] = fma2(B, g01.y, acc[6]);
          acc[7] = fma2(B, g23.x, acc[7]);
          acc[8] = fma2(B, g23.y, acc[8]);
          acc[9] = fma2(B, g4, acc[9]);
        }
        if ((n & 1) && !half) {
          const float2 L = *reinterpret_cast<const float2*>(cp);
          const ulonglong2 g01 = *reinterpret_cast<const ulonglong2*>(wp);
          const ulonglong2 g23 = *reinterpret_cast<const ulonglong2*>(wq + 4);
          const unsigned long long g4 = *reinterpret_cast<const unsigned long long*>(wq + 8);
          const unsigned long long A = pack2(L.x, L.x), B = pack2(L.y, L.y);
          acc[0] = fma2(A, g01.x, acc[0]);
          acc[1] = fma2(A, g01.y, acc[1]);
          acc[2] = fma2(A, g23.x, acc[2]);
          acc[3] = fma2(A, g23.y, acc[3]);
          acc[4] = fma2(A, g4, acc[4]);
          acc[5] = fma2(B, g01.x, acc[5]);
          acc[6] = fma2(B, g01.y, acc[6]);
          acc[7] = fma2(B, g23.x, acc[7]);
          acc[8] = fma2(B, g23.y, acc[8]);
          acc[9] = fma2(B, g4, acc[9]);
        }
        __syncwarp();
        if (last <= 32) {
          close_task(acc, m, m.e[first], w.rec + (size_t)((start + kRecMin - 1) / kRecMin) * kRecFloats, lane, p, r);
#pragma unroll
          for (int k = 0; k < 10; k++) acc[k] = 0ull;
        }
      }
      const bool more = last < 32 && todo;
      first = last = 0;
      if (more) {
        const int t = __ffs(todo) - 1;
        todo &= todo - 1;
        first = t;
        full = __shfl_sync(0xffffffffu, size0, t);
        last = t + full;
        start = w0 + t;
      }
    }
    __syncwarp();
  }
  if (!kAcc) {
    const int e0 = pt.prob_edge_off[prob], ne = pt.prob_edge_off[prob + 1] - e0;
    const int per = (ne + e_ctas - 1) / e_ctas;
    const int ea0 = e0 + min(ne, lc * per), eb = e0 + min(ne, lc * per + per);
    for (int ed = ea0 + threadIdx.x; ed < eb; ed += kThreads) {
      const Edge ev = eval_edge(ea.nodes, ea.T, pt.edge_ijk[3 * ed], pt.edge_ijk[3 * ed + 1], pt.edge_ijk[3 * ed + 2],
                                ea.lambda);
      if (ev.el > 0.f)
        energy += (double)ev.el * ((double)ev.r.x * ev.r.x + (double)ev.r.y * ev.r.y + (double)ev.r.z * ev.r.z);
    }
  }
  energy = warp_sum_d(energy);
  if (lane == 0) red[wid] = energy;
  __syncthreads();
  if (threadIdx.x == 0) {
    double v = 0.0;
#pragma unroll
    for (int k = 0; k < kWarps; k++) v += red[k];
    w.e_data_part[cta] = v;
  }
  if (!kAcc && tb.P == 1) {  // the last CTA to finish adds the partials, in their order
    __shared__ bool final_cta;
    if (threadIdx.x == 0) {
      __threadfence();
      final_cta = atomicAdd(w.done, 1u) == gridDim.x - 1u;
    }
    __syncthreads();
    if (final_cta && wid == 0) {
      __threadfence();
      reduce_energy(w, w.e_data_part, (int)gridDim.x, 0, slot);
      if (lane == 0) *w.done = 0u;
    }
  }
}

// ----------------------------------------------------------------------------
// gather
// ----------------------------------------------------------------------------
// A CTA of kRowWarps warps per block row r.  A task that contains r as its
// node a holds the sums of the pairs (a, a..3), and a's right-hand side, as one
// run of 90 - 21 a floats: three coalesced loads.  Each warp takes a share of
// the row's list, four runs in flight; it sums the diagonal block and right-hand
// side in registers (lanes 0..26, Kahan) and the off-diagonal blocks in shared
// memory, kRowBlocks of them at a time.  Then the warps' sums are added in warp
// order.  With d = x_c - x_r and D = [d]_x, the column node's u_c = u - D n, so
// a block is
//   [[S_uu + S_un D, S_un], [S_un^T + S_nn D, S_nn]]
// (kernels/solver_kernels.cu:113-137 regrouped; D = 0 on the diagonal).
// What bounds it is the chain of dependent loads (row -> list -> nodes ->
// records) while rows are few, and instruction issue when they are many; the
// warps of a row follow from that (rule at launch_assemble).
constexpr int kRowBlocks = 16;  // off-diagonal upper blocks of a row per pass (a surface's rows have about 5)
template <int kRowWarps>
struct RowMem {
  float sum[kRowWarps][kRowBlocks][kSums];
  float diag[kRowWarps][2][28];
  int4 meta[kRowBlocks];        // of the pass's blocks: row, position, column, position of the transpose
  float4 d[kRowBlocks];         // x_c - x_r
  int4 task[kRowWarps][32];     // run start, its floats, the blocks of its pairs, the row's node of the task
  int edge[kRowBlocks + 4];     // the blocks' first ARAP edges
  // (u, n), g w_a, -g r, g w_b of the three nodes after a (g = fw w_a), the blocks of its pairs
  float raw[kRowWarps][32][12];
};
// (18 CTAs of two warps per SM need 56 registers: 255k rows take 1.52 ms, with 64 1.66)
template <int kRowWarps>
__global__ void __launch_bounds__(32 * kRowWarps, kRowWarps == 2 ? 18 : 8) gather_kernel(Work w, Pattern pt, float lambda_damping) {
  constexpr int kRowThreads = 32 * kRowWarps;
  __shared__ __align__(16) RowMem<kRowWarps> m;
  const int tid = threadIdx.x, lane = lane_id(), wid = tid >> 5;
  const int r = blockIdx.x;
  const int u0 = __ldg(pt.ustart + r), nu = __ldg(pt.ustart + r + 1) - u0 - 1;  // off-diagonal upper blocks
  const int l0 = w.cl_start[r], nl = w.cl_start[r + 1] - l0;
  const bool diag_warp = wid == kRowWarps - 1;
  int a0 = 0, a1 = 0, inc = 1;  // the row's ARAP edges, a lane each (the diagonal's warp)
  if (diag_warp) {
    a0 = __ldg(pt.arap_row_ptr + r);
    a1 = __ldg(pt.arap_row_ptr + r + 1);
  }
  const int b0 = l0 + nl * wid / kRowWarps, b1 = l0 + nl * (wid + 1) / kRowWarps;
  const float4 xr = __ldg(w.npos + r);
  int li, lj;
  product_of(lane, li, lj);
  // the pair and sum of the lane's three floats of a run (pair 0: diagonal)
  const int pr0 = lane < 27 ? 0 : 1, at0 = lane < 27 ? lane : lane - 27;
  const int pr1 = lane < 16 ? 1 : 2, at1 = lane < 16 ? lane + 5 : lane - 16;
  const int pr2 = lane < 5 ? 2 : 3, at2 = lane < 5 ? lane + 16 : lane - 5;
  float tot = 0.f, comp = 0.f;
  for (int k0 = 0; k0 == 0 || k0 < nu; k0 += kRowBlocks) {
    const int kn = min(kRowBlocks, nu - k0);
    // the warp's first tasks, while the blocks' data arrive
    uint4 ds = make_uint4(0u, 0u, ~0u, ~0u);
    if (b0 + lane < b1) ds = __ldg(w.cdesc + b0 + lane);
    if (k0 == 0 && a0 + lane < a1) inc = __ldg(pt.arap_row_inc + a0 + lane);
    if (k0 > 0) __syncthreads();
    if (tid < kn) {
      const int4 mt = __ldg(pt.upper_meta + u0 + 1 + k0 + tid);
      const float4 xc = __ldg(w.npos + mt.z);
      m.meta[tid] = mt;
      m.d[tid] = make_float4(xc.x - xr.x, xc.y - xr.y, xc.z - xr.z, 0.f);
    }
    if (tid >= 32 && tid - 32 <= kn) m.edge[tid - 32] = __ldg(pt.arap_blk_ptr + u0 + 1 + k0 + tid - 32);
    for (int i = lane; i < kn * kSums; i += 32) (&m.sum[wid][0][0])[i] = 0.f;
    __syncthreads();
    if (k0 == 0) {
      after_previous();  // (so far the pattern and the lists of list_sort; the data term lies between)
      if (r == 0)  // the barriers of the PCG that follows
        for (int i = tid; i < pt.P; i += kRowThreads) w.barrier[i] = 0u;
    }
    float(*sum)[kSums] = m.sum[wid];
    for (int i0 = b0; i0 < b1; i0 += 32) {
      // a lane per task: the run, and the pass's blocks of the nodes after the row's
      if (i0 > b0) ds = i0 + lane < b1 ? __ldg(w.cdesc + i0 + lane) : make_uint4(0u, 0u, ~0u, ~0u);
      const int cnt = min(32, b1 - i0);
      const int a = ds.y & 3, nraw = ds.y >> 2;
      const unsigned long long kk = (unsigned long long)ds.w << 32 | ds.z;
      unsigned kb = 0;  // byte b: the block of pair (a, a + 1 + b), 0xff: none in this pass
#pragma unroll
      for (int b = 0; b < 3; b++) {
        const unsigned at = (unsigned)(kk >> (21 * b)) & kNoBlock, rel = at - (unsigned)k0;
        kb |= (at != kNoBlock && rel < (unsigned)kn ? rel : 0xffu) << (8 * b);
      }
      m.task[wid][lane] = make_int4((int)ds.x, lane < cnt && !nraw ? 90 - 21 * a : 0, (int)kb, a);
      __syncwarp();
      constexpr int kFly = 4;
      const int runs = __any_sync(0xffffffffu, lane < cnt && !nraw) ? cnt : 0;
      for (int t = 0; t < runs; t += kFly) {
        float x[kFly][3];
        unsigned k3[kFly];
#pragma unroll
        for (int h = 0; h < kFly; h++) {
          const int4 tk = m.task[wid][min(t + h, 31)];
          const int n = t + h < cnt ? tk.y : 0;
          const float* run = w.rec + (unsigned)tk.x + lane;
          k3[h] = n ? (unsigned)tk.z : 0xffffffu;
          x[h][0] = lane < n ? __ldcg(run) : 0.f;
          x[h][1] = lane + 32 < n ? __ldcg(run + 32) : 0.f;
          x[h][2] = lane + 64 < n ? __ldcg(run + 64) : 0.f;
        }
#pragma unroll
        for (int h = 0; h < kFly; h++) {
          if (pr0 == 0) {
            if (k0 == 0) kahan_add(tot, comp, x[h][0]);
          } else if ((k3[h] & 0xffu) != 0xffu) {
            sum[k3[h] & 0xffu][at0] += x[h][0];
          }
          const unsigned q1 = (k3[h] >> (8 * (pr1 - 1))) & 0xffu, q2 = (k3[h] >> (8 * (pr2 - 1))) & 0xffu;
          if (q1 != 0xffu) sum[q1][at1] += x[h][1];
          if (q2 != 0xffu && at2 < kSums) sum[q2][at2] += x[h][2];
          __syncwarp();
        }
      }
      // tasks without a record: their correspondences, a lane each, into
      // shared memory side by side, then added one by one, two's operands read together
      constexpr int kRawFly = 2;
      for (int j = 0; j < kRecMin - 1; j++) {
        const unsigned on = __ballot_sync(0xffffffffu, j < nraw);
        if (!on) break;
        const int n = __popc(on);
        if ((on >> lane) & 1u) {
          const int q = (int)ds.x + j;
          const float4 sf = __ldcg(w.raw + q), nr = __ldcg(w.sp_nrm + q), uw = __ldg(w.sp_uw + q);
          const float wa = sel4(uw, a) > 1e-8f ? sel4(uw, a) : 0.f;
          const float g = sf.w * wa;
          float3 u = f3(0.f, 0.f, 0.f), nn = u;
          if (g != 0.f) {
            nn = f3(nr.x, nr.y, nr.z);
            u = cross3(f3(sf.x - xr.x, sf.y - xr.y, sf.z - xr.z), nn);
          }
          float gb[3];
#pragma unroll
          for (int b = 0; b < 3; b++) {
            const float wb = sel4(uw, min(a + 1 + b, 3));
            gb[b] = a + 1 + b < 4 && wb > 1e-8f ? g * wb : 0.f;
          }
          float4* o = reinterpret_cast<float4*>(m.raw[wid][__popc(on & lanemask_lt())]);
          o[0] = make_float4(u.x, u.y, u.z, nn.x);
          o[1] = make_float4(nn.y, nn.z, g * wa, g != 0.f ? -g * nr.w : 0.f);
          o[2] = make_float4(gb[0], gb[1], gb[2], __int_as_float((int)kb));
        }
        if (lane >= n && lane < ((n + kRawFly - 1) & ~(kRawFly - 1))) {  // whole rounds: zeros, of no block
          float4* o = reinterpret_cast<float4*>(m.raw[wid][lane]);
          o[0] = o[1] = make_float4(0.f, 0.f, 0.f, 0.f);
          o[2] = make_float4(0.f, 0.f, 0.f, __int_as_float(0xffffff));
        }
        __syncwarp();
        for (int t = 0; t < n; t += kRawFly) {
          float y[kRawFly], L[kRawFly];
          float2 f[kRawFly];
          float4 e[kRawFly];
#pragma unroll
          for (int h = 0; h < kRawFly; h++) {
            const float* o = m.raw[wid][t + h];
            y[h] = o[li];
            L[h] = o[lj];
            f[h] = *reinterpret_cast<const float2*>(o + 6);
            e[h] = *reinterpret_cast<const float4*>(o + 8);
          }
#pragma unroll
          for (int h = 0; h < kRawFly; h++) {
            L[h] *= y[h];
            if (k0 == 0 && lane < 27) kahan_add(tot, comp, lane < kSums ? f[h].x * L[h] : f[h].y * y[h]);
            const unsigned k3 = (unsigned)__float_as_int(e[h].w);
            if (lane < kSums && k3 != 0xffffffu) {
              const float gb[3] = {e[h].x, e[h].y, e[h].z};
#pragma unroll
              for (int b = 0; b < 3; b++) {
                const unsigned kk = (k3 >> (8 * b)) & 0xffu;
                if (kk != 0xffu) sum[kk][lane] += gb[b] * L[h];
              }
            }
          }
        }
        __syncwarp();
      }
    }
    if (k0 == 0 && lane < 27) {
      m.diag[wid][0][lane] = tot;
      m.diag[wid][1][lane] = comp;
    }
    __syncthreads();
    // the warps' sums in warp order, then the pass's off-diagonal blocks, value by value
    for (int i = tid; i < kn * kSums; i += kRowThreads) {
      float t = (&m.sum[0][0][0])[i];
#pragma unroll
      for (int v = 1; v < kRowWarps; v++) t += (&m.sum[v][0][0])[i];
      (&m.sum[0][0][0])[i] = t;
    }
    __syncthreads();
    for (int i = tid; i < 36 * kn; i += kRowThreads) {
      const int kb = i / 36, v = i - 36 * kb, p = v / 6, q = v - 6 * p;
      const float* S = m.sum[0][kb];
      const int4 mt = m.meta[kb];
      // ARAP edges (r, c) visited from r (solver_kernels.cu:315-324); a block has one or two
      float arap = 0.f;
      for (int e2 = m.edge[kb]; e2 < m.edge[kb + 1]; e2++)
        arap += __ldcg(reinterpret_cast<const float*>(pt.edge_terms +
                                                      (size_t)kEdgeTerms4 * __ldg(pt.arap_blk_edge + e2) + 14) + v);
      float t;
      if (q >= 3) {
        t = p < 3 ? S[6 + 3 * p + (q - 3)] : S[15 + sym3(p - 3, q - 3)];  // S_un, S_nn
      } else {
        // (S_uu + S_un D)(p, q) or (S_un^T + S_nn D)(p - 3, q); column q of D = d x e_q
        const float4 d = m.d[kb];
        const float d0 = q == 0 ? 0.f : q == 1 ? -d.z : d.y, d1 = q == 0 ? d.z : q == 1 ? 0.f : -d.x,
                    d2 = q == 0 ? -d.y : q == 1 ? d.x : 0.f;
        if (p < 3) {
          t = S[sym3(p, q)] + S[6 + 3 * p] * d0 + S[6 + 3 * p + 1] * d1 + S[6 + 3 * p + 2] * d2;
        } else {
          const int pp = p - 3;
          t = S[6 + 3 * q + pp] + S[15 + sym3(pp, 0)] * d0 + S[15 + sym3(pp, 1)] * d1 + S[15 + sym3(pp, 2)] * d2;
        }
      }
      t += arap;
      pt.values[(size_t)mt.y * 36 + v] = t;
      pt.values[(size_t)mt.w * 36 + q * 6 + p] = t;
    }
  }
  if (!diag_warp) return;
  // the diagonal block: upper triangle tri6(p, q) (21) and the right-hand side (6)
  const int pos = __ldg(pt.diag_pos + r);
  if (lane < 27) {
    float t = 0.f, c = 0.f;
#pragma unroll
    for (int v = 0; v < kRowWarps; v++) {
      kahan_add(t, c, m.diag[v][0][lane]);
      kahan_add(t, c, -m.diag[v][1][lane]);
    }
    m.diag[0][0][lane] = t - c;
  }
  __syncwarp();
  const float* S = m.diag[0][0];
  int p = 0, q = 0;
  float v = 0.f, vc = 0.f;
  if (lane < kSums) {
    p = lane < 6 ? 0 : lane < 11 ? 1 : lane < 15 ? 2 : lane < 18 ? 3 : lane < 20 ? 4 : 5;
    q = lane - tri6(p, p) + p;
    v = p < 3 ? (q < 3 ? S[sym3(p, q)] : S[6 + 3 * p + (q - 3)]) : S[15 + sym3(p - 3, q - 3)];
  } else if (lane < 27) {
    v = S[lane];
  }
  // ARAP edges incident to r (kernels/solver_kernels.cu:293-313, 337-350), and the energy of those it owns
  double en = 0.0;
  for (int i0 = a0; i0 < a1; i0 += 32) {
    if (i0 > a0) inc = i0 + lane < a1 ? __ldg(pt.arap_row_inc + i0 + lane) : 1;
    if (!(inc & 1)) en += pt.edge_energy[inc >> 1];
    const int cnt = min(32, a1 - i0);
    for (int t0 = 0; t0 < cnt; t0 += 8) {
      float x[8];
#pragma unroll
      for (int h = 0; h < 8; h++) {
        const int iv = __shfl_sync(0xffffffffu, inc, min(t0 + h, 31));
        x[h] = t0 + h < cnt && lane < 27 ? __ldcg(reinterpret_cast<const float*>(
                                               pt.edge_terms + (size_t)kEdgeTerms4 * (iv >> 1) + 7 * (iv & 1)) + lane)
                                         : 0.f;
      }
#pragma unroll
      for (int h = 0; h < 8; h++)
        if (t0 + h < cnt) kahan_add(v, vc, x[h]);
    }
  }
  v -= vc;
  if (lane < kSums) {
    // damping on the diagonal entries (solver_kernels.cu:183-193)
    if (p == q) v = v + lambda_damping * fmaxf(fabsf(v), p < 3 ? 1e-3f : 1e-2f);
    float* out = pt.values + (size_t)pos * 36;
    out[p * 6 + q] = v;
    out[q * 6 + p] = v;
  } else if (lane < 27) {
    w.rhs[r * 6 + (lane - kSums)] = v;
  }
  en = warp_sum_d(en);
  if (lane == 0) w.e_arap_part[r] = en;
}

EdgeArgs edge_args(const Pattern& p, const SolveArgs& a, const cf_dual_quat* T, bool stats) {
  EdgeArgs ea;
  ea.edge_ijk = p.edge_ijk;
  ea.n_edges = p.n_edges;
  ea.nodes = a.nodes;
  ea.T = T;
  ea.lambda = a.lambda_smooth;
  ea.arap_sgn = a.arap_consistent ? -1.f : 1.f;
  ea.out = p.edge_terms;
  ea.energy = p.edge_energy;
  ea.edge_ctas = (p.n_edges + kThreads - 1) / kThreads;
  ea.stats = stats ? 1 : 0;
  return ea;
}

}  // namespace

cudaError_t launch_bucket_sort(const Work& w, const Table& tb, cudaStream_t s) {
  if (tb.N <= 0) return cudaSuccess;
  launch_next(bucket_sort_kernel, tb.N + tb.M / kSortChunk, kSortThreads, 0, s, tb, w, tb.N);
  return cudaGetLastError();
}

cudaError_t launch_node_lists(const Work& w, const Table& tb, const Pattern& p, cudaStream_t s) {
  if (tb.N <= 0 || tb.M <= 0) return cudaSuccess;
  launch_next(permute_kernel, (tb.M + kPermThreads - 1) / kPermThreads, kPermThreads, 0, s, tb, w);
  const int per = std::min(kWarps, std::max(1, (tb.N + 512) / 1024));
  launch_next(list_sort_kernel, (tb.N + per - 1) / per, kThreads, 0, s, w, p, tb.N, per);
  return cudaGetLastError();
}

cudaError_t launch_residual(const Work& w, const Table& tb, const Pattern& p, const SolveArgs& a,
                            const cf_dual_quat* T, bool skin, cudaStream_t s) {
  const EdgeArgs ea = edge_args(p, a, T, false);
  const int grid = tb.n_e + ea.edge_ctas;
  if (grid <= 0) return cudaSuccess;
  auto kern = skin ? cells_kernel<true, true> : cells_kernel<false, true>;
  const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kCellsSmem);
  if (e != cudaSuccess) return e;
  launch_next(kern, grid, kThreads, kCellsSmem, s, tb, w, p, ea, 0);
  return cudaGetLastError();
}

// Per problem the energy into statistics slot `slot` (reduce_energy).
cudaError_t launch_final_energy(const Work& w, const Pattern& p, const SolveArgs& a, int slot, cudaStream_t s,
                                bool stats) {
  const Table& tb = a.tb;
  if (tb.n_e <= 0) return cudaSuccess;
  // the energy alone needs no records and fits three CTAs per SM (1.2M
  // correspondences: 39 us, 47 with the two of the data term)
  launch_next(cells_kernel<true, false>, tb.P > 1 ? tb.n_e : 3 * 148, kThreads, 0, s, tb, w, p,
              edge_args(p, a, a.transforms, stats), slot);
  if (tb.P > 1) launch_next(energy_reduce_kernel, tb.P, 32, 0, s, tb, w, slot);
  return cudaGetLastError();
}

cudaError_t launch_assemble(const Work& w, const Pattern& p, const SolveArgs& a, cudaStream_t s) {
  if (p.N <= 0) return cudaSuccess;
  // Warps per row: four while all rows are resident with them (the chain of a
  // row is then four times shorter; 256 rows: 14.8 us against 18.9), two beyond
  // (less work per row; 2048 rows: 23 us against 26, 255k rows: 1.61 against 2.12 ms).
  if (p.N <= 1024)
    launch_next(gather_kernel<4>, p.N, 128, 0, s, w, p, a.lambda_damping);
  else
    launch_next(gather_kernel<2>, p.N, 64, 0, s, w, p, a.lambda_damping);
  return cudaGetLastError();
}

}  // namespace cf
