// cf_kernels.cu — sm_100a kernels of the warp-field Gauss-Newton solve.
//
// Per solve (the correspondences' node ids are fixed for all GN iterations) a
// stable counting sort by node; what follows it is in cf_cells.cu:
//   key_count     per correspondence its node set's key, per-CTA histograms
//   bin_scan_*    deterministic exclusive offsets (node, CTA)
//   bin_scatter   the correspondences in order of their first node
// The scan also resets the solve's statistics and makes each node's plain DQ
// (once per node, not per point; the PCG's node update keeps it current).
// Every kernel works on a table of problems (ProbDesc): a single solve is a
// batch of one; a batched solve concatenates its problems' correspondences
// and nodes, and each sort / energy CTA belongs to exactly one problem.
// The PCG kernels live in cf_pcg_grid.cu (grid-wide cooperative) and
// cf_pcg_cluster.cu (one thread-block cluster).
// The reference (CUDAFusion kernels/solver_kernels.cu) assembles with float
// atomicAdd and runs PCG as ~10 synchronised launches per iteration.
#include <cooperative_groups.h>

#include "cf_device.cuh"
#include "cf_internal.h"

namespace cf {

namespace {

constexpr int kWords = 19;  // sizeof(cf_correspondence) / 4
static_assert(sizeof(cf_correspondence) == 76, "Correspondence layout");
static_assert(sizeof(cf_deform_node) == 96, "DeformNode layout");
static_assert(sizeof(cf_dual_quat) == 32, "DualQuat layout");

// ----------------------------------------------------------------------------
// keys + count
// ----------------------------------------------------------------------------
// A correspondence's key: its distinct valid nodes (id in range, weight not
// below 1e-8) in ascending order as four 16-bit local ids, 0xffff past the
// last.  One that weighs but has no valid node sorts with node 0 under a
// second word of 0xfffe; one that does not weigh (invalid, or a weight that is
// not positive) has all bits set and is left out of the sort.
constexpr unsigned kNone = 0xffffu;
__device__ __forceinline__ int key_node(unsigned lo) {
  const unsigned a = lo & 0xffffu;
  return a != kNone ? (int)a : (lo >> 16) == kNone - 1 ? 0 : -1;
}

__global__ void __launch_bounds__(kThreads) key_count_kernel(Table tb, Work w) {
  after_previous();
  extern __shared__ int hist[];
  __shared__ __align__(16) uint32_t stage2[2][kThreads * kWords];  // double-buffered tiles of records
  const int tid = threadIdx.x;
  const ProbDesc d = tb.desc[tb.bin_prob[blockIdx.x]];
  const int N = d.N, lc = blockIdx.x - d.bin_cta0;
  for (int i = tid; i < N; i += kThreads) hist[i] = 0;
  const cf_correspondence* corrs = d.corrs;
  const bool al16 = ((reinterpret_cast<uintptr_t>(corrs) & 15u) == 0);
  const int cb = lc * d.chunk;
  const int ce = min(d.M, cb + d.chunk);
  // the next tile's records are in flight (cp.async) while this one is read
  auto issue = [&](int t0, int b) {
    const int nt = min(kThreads, ce - t0), nw = nt * kWords;
    const uint32_t* src = reinterpret_cast<const uint32_t*>(corrs) + (size_t)t0 * kWords;
    uint32_t* buf = stage2[b];
    if (al16 && (nw & 3) == 0) {
      for (int i = tid; i < (nw >> 2); i += kThreads) cp_async16(buf + 4 * i, src + 4 * i);
    } else {
      for (int i = tid; i < nw; i += kThreads) cp_async4(buf + i, src + i);
    }
    cp_async_commit();
  };
  if (cb < ce) issue(cb, 0);
  __syncthreads();
  for (int t0 = cb, it = 0; t0 < ce; t0 += kThreads, it++) {
    const int n = min(kThreads, ce - t0);
    const uint32_t* stage = stage2[it & 1];
    if (t0 + kThreads < ce) {
      issue(t0 + kThreads, (it & 1) ^ 1);
      cp_async_wait<1>();
    } else {
      cp_async_wait<0>();
    }
    __syncthreads();
    if (tid < n) {
      const uint32_t* rec = stage + tid * kWords;
      const bool on = (rec[18] & 0xffu) != 0 && __uint_as_float(rec[17]) > 0.f;
      unsigned k[kK];
#pragma unroll
      for (int s = 0; s < kK; s++) {
        const int id = (int)rec[9 + s];
        k[s] = id >= 0 && id < N && !(__uint_as_float(rec[13 + s]) < 1e-8f) ? (unsigned)id : kNone;
      }
      auto order = [](unsigned& x, unsigned& y) {
        const unsigned lo = min(x, y), hi = max(x, y);
        x = lo;
        y = hi;
      };
      order(k[0], k[1]); order(k[2], k[3]); order(k[0], k[2]); order(k[1], k[3]); order(k[1], k[2]);
      if (k[0] == k[1]) k[1] = kNone;
      if (k[2] == k[1] || k[2] == k[0]) k[2] = kNone;
      if (k[3] == k[2] || k[3] == k[1] || k[3] == k[0]) k[3] = kNone;
      order(k[1], k[2]); order(k[2], k[3]); order(k[1], k[2]);
      if (k[0] == kNone) k[1] = kNone - 1;
      if (!on) k[0] = k[1] = k[2] = k[3] = kNone;
      const uint2 key = make_uint2(k[0] | (k[1] << 16), k[2] | (k[3] << 16));
      w.key[d.corr_off + t0 + tid] = key;
      const int node = key_node(key.x);
      if (node >= 0) atomicAdd(&hist[node], 1);
    }
    __syncthreads();
  }
  int* out = w.cnt + d.cnt_off + (size_t)lc * N;
  for (int i = tid; i < N; i += kThreads) out[i] = hist[i];
}

// Statistics and error word of the solve that begins.
__device__ __forceinline__ void reset_state(const Table& tb, const Work& w, int reset_stats) {
  int* st = reinterpret_cast<int*>(w.stats);
  if (reset_stats)
    for (int i = threadIdx.x; i < tb.P * (int)(sizeof(DevStats) / sizeof(int)); i += kThreads) st[i] = 0;
  if (threadIdx.x == 0) *w.err = 0;
}
// A node's position and, at the solve's start, its plain DQ.
__device__ __forceinline__ void setup_node(const Table& tb, const Work& w, int n) {
  const ProbDesc& d = tb.desc[tb.node_prob[n]];
  const int l = n - d.node_off;
  const float3 x = node_pos(d.nodes, l);
  w.npos[n] = make_float4(x.x, x.y, x.z, 0.f);
  store_dq(w.plain + n, dq_centered(load_dq_cg(d.T + l), x));
}

// Per node: exclusive prefix of its counts over its problem's sort CTAs (in
// place); node_total[n] = sum.  32 nodes per CTA, lane = node (coalesced
// over the sort-CTA index k); the k range is split over the 8 warps: segment
// sums with all loads in flight, a prefix over the warps, then each warp
// rewrites its segment.
//
// The launch also resets the solve's statistics and sets up its nodes.
__global__ void __launch_bounds__(kThreads) bin_scan_nodes_kernel(Table tb, Work w, int reset_stats) {
  after_previous();
  __shared__ int seg[kThreads / 32][32];
  if (blockIdx.x == 0) reset_state(tb, w, reset_stats);
  const int lane = lane_id(), wid = threadIdx.x >> 5;
  const int n = blockIdx.x * 32 + lane;
  int bc = 0, stride = 0;
  int* p = nullptr;
  if (n < tb.N) {
    const ProbDesc& d = tb.desc[tb.node_prob[n]];
    bc = d.bin_ctas;
    stride = d.N;
    p = w.cnt + d.cnt_off + (n - d.node_off);
  }
  const int per = (bc + kThreads / 32 - 1) / (kThreads / 32);
  const int k0 = min(bc, wid * per), k1 = min(bc, k0 + per);
  int s = 0;
  for (int k = k0; k < k1; k += 8) {
    int v[8];
#pragma unroll
    for (int b = 0; b < 8; b++) v[b] = (k + b < k1) ? p[(size_t)(k + b) * stride] : 0;
#pragma unroll
    for (int b = 0; b < 8; b++) s += v[b];
  }
  seg[wid][lane] = s;
  __syncthreads();
  int run = 0;
  for (int v = 0; v < wid; v++) run += seg[v][lane];
  if (wid == kThreads / 32 - 1 && n < tb.N) {
    w.node_total[n] = run + s;
    w.cl_total[n] = 0;  // the tasks per node are counted after the sort
    setup_node(tb, w, n);
  }
  for (int k = k0; k < k1; k += 8) {
    int v[8];
#pragma unroll
    for (int b = 0; b < 8; b++) v[b] = (k + b < k1) ? p[(size_t)(k + b) * stride] : 0;
#pragma unroll
    for (int b = 0; b < 8; b++)
      if (k + b < k1) {
        p[(size_t)(k + b) * stride] = run;
        run += v[b];
      }
  }
}

// the node set-up alone, for a table without correspondences
__global__ void __launch_bounds__(kThreads) node_setup_kernel(Table tb, Work w, int reset_stats) {
  after_previous();
  if (blockIdx.x == 0) reset_state(tb, w, reset_stats);
  const int n = blockIdx.x * kThreads + threadIdx.x;
  if (n < tb.N) setup_node(tb, w, n);
}

// start = exclusive scan of total (one CTA of 1024 threads, 4096 nodes per
// round, the next round's totals in flight); cursor, when given, a copy of it.
__global__ void __launch_bounds__(1024) scan_kernel(const int* total, int* __restrict__ start,
                                                    int* __restrict__ cursor, int N) {
  after_previous();
  __shared__ int wsum[32];
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  auto load = [&](int i0) {
    int4 v = make_int4(0, 0, 0, 0);
    const int i = i0 + 4 * tid;
    if (i + 3 < N) return __ldcg(reinterpret_cast<const int4*>(total + i));
    if (i < N) v.x = __ldcg(total + i);
    if (i + 1 < N) v.y = __ldcg(total + i + 1);
    if (i + 2 < N) v.z = __ldcg(total + i + 2);
    return v;
  };
  int carry = 0;
  int4 v = load(0);
  for (int i0 = 0; i0 < N; i0 += 4096) {
    const int4 nx = load(i0 + 4096);
    const int sum = v.x + v.y + v.z + v.w;
    int incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += t;
    }
    if (lane == 31) wsum[wid] = incl;
    __syncthreads();
    int ws = wsum[lane], wi = ws;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, wi, o);
      if (lane >= o) wi += t;
    }
    const int before = __shfl_sync(0xffffffffu, wi - ws, wid), all = __shfl_sync(0xffffffffu, wi, 31);
    int run = carry + before + incl - sum;
    const int o[4] = {run, run + v.x, run + v.x + v.y, run + v.x + v.y + v.z};
    const int i = i0 + 4 * tid;
#pragma unroll
    for (int k = 0; k < 4; k++)
      if (i + k < N) {
        start[i + k] = o[k];
        if (cursor) cursor[i + k] = o[k];
      }
    carry += all;
    v = nx;
    __syncthreads();
  }
  if (tid == 0) start[N] = carry;
}

// Stable scatter of the correspondences by their key's first node: order
// within a node = (tile, correspondence).
__global__ void __launch_bounds__(kThreads) bin_scatter_kernel(Table tb, Work w) {
  after_previous();
  extern __shared__ int cursor[];
  __shared__ int wkey[kThreads / 32][32];
  __shared__ int wcnt[kThreads / 32][32];
  __shared__ int wlen[kThreads / 32];
  const int tid = threadIdx.x, lane = lane_id(), warp = tid >> 5;
  const ProbDesc d = tb.desc[tb.bin_prob[blockIdx.x]];
  const int N = d.N, lc = blockIdx.x - d.bin_cta0;
  const int* base = w.cnt + d.cnt_off + (size_t)lc * N;
  for (int i = tid; i < N; i += kThreads) cursor[i] = w.inc_start[d.node_off + i] + base[i];
  const int cb = d.corr_off + lc * d.chunk;
  const int ce = d.corr_off + min(d.M, lc * d.chunk + d.chunk);
  __syncthreads();
  for (int t0 = cb; t0 < ce; t0 += kThreads) {
    const int c = t0 + tid;
    const int key = c < ce ? key_node(w.key[c].x) : -1;
    const unsigned peers = __match_any_sync(0xffffffffu, key);
    const int rank = __popc(peers & lanemask_lt());
    const bool leader = (__ffs(peers) - 1) == lane;
    const bool last = (31 - __clz(peers)) == lane;
    const unsigned lead_mask = __ballot_sync(0xffffffffu, leader && key >= 0);
    if (leader && key >= 0) {
      const int slot = __popc(lead_mask & lanemask_lt());
      wkey[warp][slot] = key;
      wcnt[warp][slot] = __popc(peers);
    }
    if (lane == 0) wlen[warp] = __popc(lead_mask);
    __syncthreads();
    int pos = 0;
    bool is_last = false;
    if (key >= 0) {
      int prefix = 0;
      for (int v = 0; v < warp; v++)
        for (int s = 0; s < wlen[v]; s++)
          if (wkey[v][s] == key) prefix += wcnt[v][s];
      is_last = last;
      if (is_last)
        for (int v = warp + 1; v < kThreads / 32 && is_last; v++)
          for (int s = 0; s < wlen[v]; s++)
            if (wkey[v][s] == key) is_last = false;
      pos = cursor[key] + prefix + rank;
      w.order[pos] = c;
    }
    __syncthreads();
    if (is_last) cursor[key] = pos + 1;
    __syncthreads();
  }
}

// The same with per-warp cursors (problems of at most about 10k nodes): the
// sort CTA's correspondences are split into 8 contiguous warp ranges; order
// within a node = (warp range, correspondence).  Pass 1 counts per (warp,
// node) in 16-bit shared counters, pass 2 turns them into offsets below the
// CTA's base, pass 3 writes; no CTA barrier inside a pass.
constexpr int kScatterWarps = kThreads / 32;
constexpr int kWarpScatterSmem = 200 * 1024;
__global__ void __launch_bounds__(kThreads) bin_scatter_warp_kernel(Table tb, Work w) {
  after_previous();
  extern __shared__ int sbase[];  // [N] CTA base of each node, then [8][N] 16-bit warp offsets
  const int tid = threadIdx.x, lane = lane_id(), warp = tid >> 5;
  const ProbDesc d = tb.desc[tb.bin_prob[blockIdx.x]];
  const int N = d.N, lc = blockIdx.x - d.bin_cta0;
  unsigned short* wcnt = reinterpret_cast<unsigned short*>(sbase + N);
  unsigned short* mine = wcnt + (size_t)warp * N;
  const int* base = w.cnt + d.cnt_off + (size_t)lc * N;
  for (int i = tid; i < N; i += kThreads) sbase[i] = w.inc_start[d.node_off + i] + base[i];
  for (int i = tid; i < kScatterWarps * N; i += kThreads) wcnt[i] = 0;
  const int cb = d.corr_off + lc * d.chunk;
  const int ce = d.corr_off + min(d.M, lc * d.chunk + d.chunk);
  const int per = (ce - cb + kScatterWarps - 1) / kScatterWarps;
  const int wb = min(ce, cb + warp * per), we_ = min(ce, wb + per);
  __syncthreads();
  // pass 1: counts per (warp, node)
  for (int t0 = wb; t0 < we_; t0 += 32) {
    const int c = t0 + lane;
    const int key = c < we_ ? key_node(w.key[c].x) : -1;
    const unsigned peers = __match_any_sync(0xffffffffu, key);
    if (key >= 0 && (__ffs(peers) - 1) == lane) mine[key] += (unsigned short)__popc(peers);
    __syncwarp();
  }
  __syncthreads();
  // pass 2: per node, the warps' offsets below the CTA base
  for (int i = tid; i < N; i += kThreads) {
    unsigned run = 0;
#pragma unroll
    for (int v = 0; v < kScatterWarps; v++) {
      const unsigned t = wcnt[(size_t)v * N + i];
      wcnt[(size_t)v * N + i] = (unsigned short)run;
      run += t;
    }
  }
  __syncthreads();
  // pass 3: the writes, in the order of pass 1
  for (int t0 = wb; t0 < we_; t0 += 32) {
    const int c = t0 + lane;
    const int key = c < we_ ? key_node(w.key[c].x) : -1;
    const unsigned peers = __match_any_sync(0xffffffffu, key);
    if (key >= 0) w.order[sbase[key] + mine[key] + __popc(peers & lanemask_lt())] = c;
    __syncwarp();
    if (key >= 0 && (__ffs(peers) - 1) == lane) mine[key] += (unsigned short)__popc(peers);
    __syncwarp();
  }
}

// ----------------------------------------------------------------------------
// per-iteration kernels
// ----------------------------------------------------------------------------
// Batched solves: each problem's nodes (neighbour ids made global) and
// transforms into the concatenated arrays.
__global__ void batch_gather_kernel(Table tb, Work w) {
  after_previous();
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= tb.N) return;
  const ProbDesc d = tb.desc[tb.node_prob[n]];
  const int l = n - d.node_off;
  cf_deform_node nd = d.nodes[l];
  const int nn = min(max(nd.num_neighbors, 0), CF_K_GRAPH);
#pragma unroll
  for (int k = 0; k < CF_K_GRAPH; k++) {
    const int j = nd.neighbors[k];
    nd.neighbors[k] = (k < nn && j >= 0 && j < d.N) ? j + d.node_off : -1;
  }
  w.nodes_cat[n] = nd;
  store_dq(w.T_cat + n, load_dq_cg(d.T + l));
}

__global__ void batch_scatter_kernel(Table tb, Work w) {
  after_previous();
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= tb.N) return;
  const ProbDesc d = tb.desc[tb.node_prob[n]];
  store_dq(d.T + (n - d.node_off), load_dq_cg(w.T_cat + n));
}

// WarpField::apply_twist_increment (src/warp_field.cu:250-291).
__global__ void apply_twist_kernel(cf_dual_quat* __restrict__ T, const float* dx, int N, float max_rot,
                                   float max_trans, float scale) {
  after_previous();
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  float d[6];
#pragma unroll
  for (int k = 0; k < 6; k++) d[k] = dx[i * 6 + k];
  store_dq(T + i, twist_update(load_dq_cg(T + i), d, max_rot, max_trans, scale));
}

// warp_point per point (se3_math.cuh:450-510), centring each node DQ on the fly.
__global__ void skin_points_kernel(const float* pts, const int* ids,
                                   const float* ws, int M, const cf_deform_node* nodes,
                                   const cf_dual_quat* T, int N, float* out) {
  after_previous();
  int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= M) return;
  const float3 o = skin_point_centered(f3(pts[3 * c], pts[3 * c + 1], pts[3 * c + 2]), ids + 4 * c, ws + 4 * c,
                                       nodes, T, N);
  out[3 * c] = o.x;
  out[3 * c + 1] = o.y;
  out[3 * c + 2] = o.z;
}

inline int cdiv(int a, int b) { return (a + b - 1) / b; }

}  // namespace

// ----------------------------------------------------------------------------
// launchers
// ----------------------------------------------------------------------------
cudaError_t launch_key_count(const Work& w, const Table& tb, cudaStream_t s) {
  if (tb.n_bin <= 0) return cudaSuccess;
  const int smem = tb.max_N * (int)sizeof(int);
  cudaError_t e = cudaFuncSetAttribute(key_count_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return e;
  launch_next(key_count_kernel, tb.n_bin, kThreads, smem, s, tb, w);
  return cudaGetLastError();
}

cudaError_t launch_bin_scan(const Work& w, const Table& tb, bool reset_stats, cudaStream_t s) {
  if (tb.N <= 0) return cudaSuccess;
  launch_next(bin_scan_nodes_kernel, cdiv(tb.N, 32), kThreads, 0, s, tb, w, reset_stats ? 1 : 0);
  launch_next(scan_kernel, 1, 1024, 0, s, w.node_total, w.inc_start, nullptr, tb.N);
  return cudaGetLastError();
}

cudaError_t launch_node_setup(const Work& w, const Table& tb, bool reset_stats, cudaStream_t s) {
  if (tb.N <= 0) return cudaSuccess;
  launch_next(node_setup_kernel, cdiv(tb.N, kThreads), kThreads, 0, s, tb, w, reset_stats ? 1 : 0);
  return cudaGetLastError();
}

cudaError_t launch_list_scan(const Work& w, const Table& tb, cudaStream_t s) {
  if (tb.N <= 0) return cudaSuccess;
  launch_next(scan_kernel, 1, 1024, 0, s, w.cl_total, w.cl_start, w.cl_cur, tb.N);
  return cudaGetLastError();
}

cudaError_t launch_bin_scatter(const Work& w, const Table& tb, cudaStream_t s) {
  if (tb.n_bin <= 0) return cudaSuccess;
  // per-warp cursors: 20 B of shared memory per node, counts below 2^16
  const int wsmem = tb.max_N * (int)(sizeof(int) + kScatterWarps * sizeof(unsigned short));
  if (wsmem <= kWarpScatterSmem && tb.max_chunk < 65536) {
    cudaError_t e = cudaFuncSetAttribute(bin_scatter_warp_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         kWarpScatterSmem);
    if (e != cudaSuccess) return e;
    launch_next(bin_scatter_warp_kernel, tb.n_bin, kThreads, wsmem, s, tb, w);
    return cudaGetLastError();
  }
  const int smem = tb.max_N * (int)sizeof(int);
  cudaError_t e = cudaFuncSetAttribute(bin_scatter_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return e;
  launch_next(bin_scatter_kernel, tb.n_bin, kThreads, smem, s, tb, w);
  return cudaGetLastError();
}

cudaError_t launch_batch_gather(const Work& w, const Table& tb, cudaStream_t s) {
  if (tb.N <= 0) return cudaSuccess;
  launch_next(batch_gather_kernel, cdiv(tb.N, 128), 128, 0, s, tb, w);
  return cudaGetLastError();
}

cudaError_t launch_batch_scatter(const Work& w, const Table& tb, cudaStream_t s) {
  if (tb.N <= 0) return cudaSuccess;
  launch_next(batch_scatter_kernel, cdiv(tb.N, 128), 128, 0, s, tb, w);
  return cudaGetLastError();
}

cudaError_t launch_apply_twist(cf_dual_quat* T, const float* dx, int N, float max_rot, float max_trans,
                               float scale, cudaStream_t s) {
  if (N <= 0) return cudaSuccess;
  launch_next(apply_twist_kernel, cdiv(N, 128), 128, 0, s, T, dx, N, max_rot, max_trans, scale);
  return cudaGetLastError();
}

cudaError_t launch_skin_points(const float* pts, const int* ids, const float* ws, int M,
                               const cf_deform_node* nodes, const cf_dual_quat* T, int N, float* out,
                               cudaStream_t s) {
  if (M <= 0) return cudaSuccess;
  launch_next(skin_points_kernel, cdiv(M, 256), 256, 0, s, pts, ids, ws, M, nodes, T, N, out);
  return cudaGetLastError();
}

}  // namespace cf
