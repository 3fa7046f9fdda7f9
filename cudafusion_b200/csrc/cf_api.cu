// cf_api.cu — C ABI of the warp-field solve (include/cudafusion_b200.h).
//
// Host-side responsibilities: argument checks and status codes, the block
// pattern (built on the host from the node graph like the reference,
// kernels/solver_kernels.cu:498-541), the PCG row partition, and the launch
// sequence.  Every device computation happens in cf_kernels.cu.
#include <algorithm>
#include <map>
#include <mutex>
#include <set>
#include <string>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "cf_internal.h"

using namespace cf;

// Phase slots of the profiler (cf_gn_profile_*).  The nodes are set up by the
// scan's launch; node_plain is that alone, where there are no correspondences.
enum ProfSlot {
  kProfPack = 0, kProfBinScan, kProfScatter, kProfSort, kProfNodePlain, kProfResidual, kProfAssemble,
  kProfPcg, kProfEnergy, kProfTwist, kProfLists, kProfOther
};
constexpr int kProfLearned = kProfTwist;  // the learned start: features, network, apply, gate
static const char* kProfNames[CF_PROF_SLOTS] = {"key_count", "bin_scan", "bin_scatter", "bucket_sort",
                                                "node_plain", "residual", "assemble", "pcg",
                                                "final_energy", "apply_twist", "node_lists", "other"};

struct ProfEvent {
  int slot;
  cudaEvent_t a, b;
};

struct cf_gn {
  cf_gn_params params;
  int max_nodes = 0, max_corrs = 0;
  int device = 0, sms = 0;
  int arap_consistent = 0;
  int pcg_ctas_override = 0;
  int pcg_mode = 0;  // 0 auto, 1 grid-wide cooperative, 2 single cluster
  int pcg_pipelined = 0;
  int phase_timers = 0;
  unsigned spin_limit = 1u << 22;
  int stream_tile = 256;
  unsigned bar_extra = 0;
  Work w;
  Pattern p;
  bool pattern_valid = false;
  std::vector<int> h_row_ptr, h_col_idx;
  std::vector<int> pattern_key;  // problem sizes the pattern was built for
  unsigned pattern_version = 0;  // bumped by every pattern build
  // the captured launch sequence of the last solve and the arguments it was captured with
  int use_graph = 1;
  std::vector<unsigned char> graph_key;
  cudaGraphExec_t graph_exec = nullptr;
  long long graph_launches = 0;
  bool graph_key_failed = false;
  int graph_last = 0;  // the last solve ran as a graph
  // learned solve: the network and the transform history of the call being enqueued
  Mpnn* learn_net = nullptr;
  const cf_dual_quat* learn_hist = nullptr;
  DevStats* h_stats = nullptr;   // pinned, [kMaxProblems]
  // problem table: host copies (to skip unchanged uploads) and device arrays
  std::vector<ProbDesc> h_desc;
  std::vector<int> h_bin_prob, h_e_prob, h_node_prob;
  Table tb;
  int last_gn = 0;
  long long launches = 0;
  bool profile = false;
  std::vector<ProfEvent> prof_pool;  // events created once, reused
  size_t prof_used = 0;
  double prof_ms[CF_PROF_SLOTS] = {0};
  int prof_n[CF_PROF_SLOTS] = {0};
};

namespace {

thread_local char g_last_error[256] = {0};

cf_status from_cuda(cudaError_t e) {
  if (e == cudaSuccess) return CF_OK;
  snprintf(g_last_error, sizeof(g_last_error), "%s", cudaGetErrorString(e));
  if (e == cudaErrorMemoryAllocation) return CF_ERR_OOM;
  if (e == cudaErrorNoDevice || e == cudaErrorInsufficientDriver) return CF_ERR_NO_DEVICE;
  return CF_ERR_CUDA;
}

#define CF_TRY(expr)                        \
  do {                                      \
    cudaError_t e_ = (expr);                \
    if (e_ != cudaSuccess) return from_cuda(e_); \
  } while (0)

template <typename T>
cudaError_t dalloc(T** p, size_t n) {
  *p = nullptr;
  if (n == 0) n = 1;
  return cudaMalloc((void**)p, n * sizeof(T));
}

template <typename T>
void dfree(T*& p) {
  if (p) cudaFree((void*)p);
  p = nullptr;
}

void free_pattern(Pattern& p) {
  dfree(p.row_ptr); dfree(p.col_idx); dfree(p.diag_pos);
  dfree(p.upper_meta); dfree(p.arap_row_ptr); dfree(p.arap_row_inc);
  dfree(p.arap_blk_ptr); dfree(p.arap_blk_edge); dfree(p.edge_ijk); dfree(p.values);
  dfree(p.pcg_row_begin);
  dfree(p.clu_row_begin); dfree(p.ustart); dfree(p.clu_vidx); dfree(p.clu_halo);
  dfree(p.clu_halo_ptr); dfree(p.g_vidx); dfree(p.g_halo_ptr); dfree(p.g_halo_col);
  dfree(p.pcg_cta_off); dfree(p.pcg_prob); dfree(p.prob_edge_off);
  dfree(p.st_tile_ptr); dfree(p.st_tile_row); dfree(p.st_tile_cols); dfree(p.edge_terms); dfree(p.edge_energy);
  p = Pattern();
}

void free_work(Work& w) {
  dfree(w.key); dfree(w.order); dfree(w.sorted); dfree(w.npos); dfree(w.sp_src); dfree(w.sp_dst); dfree(w.sp_nrm); dfree(w.sp_uw); dfree(w.task);
  dfree(w.cell_ids); dfree(w.rec); dfree(w.raw); dfree(w.cstat); dfree(w.cl_total); dfree(w.cl_start);
  dfree(w.cl_cur); dfree(w.clist); dfree(w.cdesc); dfree(w.cnt); dfree(w.node_total); dfree(w.inc_start); dfree(w.rhs); dfree(w.plain); dfree(w.x); dfree(w.z); dfree(w.p0); dfree(w.p1);
  dfree(w.partials); dfree(w.barrier); dfree(w.dots); dfree(w.err); dfree(w.done); dfree(w.e_data_part); dfree(w.e_arap_part); dfree(w.stats); dfree(w.timers);
  dfree(w.nodes_cat); dfree(w.T_cat); dfree(w.r); dfree(w.ap); dfree(w.zp); dfree(w.minv32);
  w.cnt_cap = 0;
}

void free_table(Table& t) {
  dfree(t.desc); dfree(t.bin_prob); dfree(t.e_prob); dfree(t.node_prob);
  t = Table();
}

cudaError_t alloc_work(Work& w, int max_nodes, int max_corrs, int bin_ctas_max) {
  w.max_nodes = max_nodes;
  w.max_corrs = max_corrs;
  w.bin_ctas_max = bin_ctas_max;
  size_t M = (size_t)max_corrs, N = (size_t)max_nodes;
  cudaError_t e;
#define A_(ptr, n) if ((e = dalloc(&(ptr), (n))) != cudaSuccess) return e
  A_(w.key, M); A_(w.order, M); A_(w.sorted, M); A_(w.npos, N); A_(w.sp_src, M); A_(w.sp_dst, M); A_(w.sp_nrm, M); A_(w.sp_uw, M);
  A_(w.task, M); A_(w.cell_ids, M); A_(w.rec, (M / kRecMin + 2) * kRecFloats); A_(w.raw, M); A_(w.cstat, M);
  A_(w.node_total, N); A_(w.inc_start, N + 1);
  A_(w.cl_total, N); A_(w.cl_start, N + 1); A_(w.cl_cur, N); A_(w.clist, 4 * M); A_(w.cdesc, 4 * M);
  A_(w.rhs, 6 * N); A_(w.plain, N); A_(w.x, 6 * N); A_(w.z, 6 * N); A_(w.p0, 6 * N); A_(w.p1, 6 * N);
  A_(w.partials, (size_t)2 * 3 * kMaxPcgCtas); A_(w.barrier, (size_t)kMaxPcgCtas); A_(w.dots, (size_t)kMaxPcgCtas * 48); A_(w.err, 1);
  A_(w.e_data_part, (size_t)(kMaxEnergyCtas + kMaxProblems)); A_(w.e_arap_part, N); A_(w.stats, (size_t)kMaxProblems);
  A_(w.timers, (size_t)kTimerSlots); A_(w.done, 1);
#undef A_
  if ((e = cudaMemset(w.dots, 0, sizeof(unsigned long long) * (size_t)kMaxPcgCtas * 48)) != cudaSuccess) return e;
  return cudaMemset(w.done, 0, sizeof(unsigned));
}

int cdiv(int a, int b) { return (a + b - 1) / b; }

// Brackets one launch (or a short launch sequence) of phase `slot` with
// events when profiling is on; counts kernel launches always.
struct Timed {
  cf_gn* h;
  cudaStream_t s;
  ProfEvent* ev = nullptr;
  Timed(cf_gn* h_, cudaStream_t s_, int slot, int nkernels) : h(h_), s(s_) {
    h->launches += nkernels;
    if (!h->profile) return;
    if (h->prof_used == h->prof_pool.size()) {
      ProfEvent pe;
      pe.slot = slot;
      cudaEventCreate(&pe.a);
      cudaEventCreate(&pe.b);
      h->prof_pool.push_back(pe);
    }
    ev = &h->prof_pool[h->prof_used++];
    ev->slot = slot;
    h->prof_n[slot] += nkernels;
    cudaEventRecord(ev->a, s);
  }
  ~Timed() {
    if (ev) cudaEventRecord(ev->b, s);
  }
};

// Folds recorded event pairs into the per-slot totals (synchronises).
void prof_collect(cf_gn* h) {
  for (size_t i = 0; i < h->prof_used; i++) {
    ProfEvent& pe = h->prof_pool[i];
    cudaEventSynchronize(pe.b);
    float ms = 0.f;
    if (cudaEventElapsedTime(&ms, pe.a, pe.b) == cudaSuccess) h->prof_ms[pe.slot] += ms;
  }
  h->prof_used = 0;
}

template <typename T>
cudaError_t upload_if_changed(T* d, std::vector<T>& cache, const std::vector<T>& v, cudaStream_t s) {
  if (v.size() == cache.size() && (v.empty() || memcmp(v.data(), cache.data(), v.size() * sizeof(T)) == 0))
    return cudaSuccess;
  cache = v;
  // pageable source: the copy is staged before the call returns, so the
  // cache may change afterwards
  return v.empty() ? cudaSuccess : cudaMemcpyAsync(d, cache.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice, s);
}

// Lays out the sort and energy CTAs of the problems `in` (corrs, canon,
// nodes, T, M, N and the clamps filled in by the caller) and uploads the
// table when it changed.  single: one problem with the single-solve grid
// sizes.
cf_status prepare_table(cf_gn* h, std::vector<ProbDesc> in, bool single, cudaStream_t s) {
  Work& w = h->w;
  Table& t = h->tb;
  const int P = (int)in.size();
  if (P < 1 || P > kMaxProblems) return CF_ERR_CAPACITY;
  long long Mt = 0, Nt = 0;
  int maxN = 0;
  for (auto& d : in) {
    if (d.N > kMaxProblemNodes) return CF_ERR_CAPACITY;
    Mt += d.M;
    Nt += d.N;
    maxN = std::max(maxN, d.N);
  }
  if (Nt > w.max_nodes || Mt > w.max_corrs) return CF_ERR_CAPACITY;
  // sort CTAs: two per SM for a single solve; a batch gets at least one per
  // kSortCorrs correspondences, shared out in proportion to the problems' sizes
  const int B = single ? w.bin_ctas_max
                       : (int)std::max<long long>(w.bin_ctas_max, std::min<long long>(kMaxSortCtas, (Mt + kSortCorrs - 1) / kSortCorrs));
  const long long e_total = std::min<long long>(kMaxEnergyCtas, std::max<long long>(kEnergyCtas, Mt / kEnergyMinPerCta));
  std::vector<int> bin_prob, e_prob;
  long long cnt = 0;
  int corr_off = 0, node_off = 0;
  for (int p = 0; p < P; p++) {
    ProbDesc& d = in[p];
    d.corr_off = corr_off;
    d.node_off = node_off;
    int bc = 0, chunk = 0;
    if (d.M > 0) {
      bc = single ? std::min(B, std::max(1, cdiv(d.M, kThreads)))
                  : std::min(cdiv(d.M, kThreads), std::max(1, (int)((double)B * d.M / (double)Mt + 0.5)));
      chunk = cdiv(cdiv(d.M, bc), kThreads) * kThreads;
      bc = cdiv(d.M, chunk);
    }
    d.bin_cta0 = (int)bin_prob.size();
    d.bin_ctas = bc;
    d.chunk = chunk;
    d.cnt_off = cnt;
    cnt += (long long)bc * d.N;
    bin_prob.insert(bin_prob.end(), bc, p);
    const int ec = single ? kEnergyCtas
                          : std::max(1, (int)((double)e_total * d.M / (double)std::max(1LL, Mt) + 0.5));
    d.e_cta0 = (int)e_prob.size();
    d.e_ctas = ec;
    e_prob.insert(e_prob.end(), ec, p);
    corr_off += d.M;
    node_off += d.N;
  }
  if ((int)e_prob.size() > kMaxEnergyCtas + kMaxProblems) return CF_ERR_CAPACITY;
  if (cnt > w.cnt_cap) {
    dfree(w.cnt);
    w.cnt_cap = 0;
    CF_TRY(dalloc(&w.cnt, (size_t)cnt));
    w.cnt_cap = cnt;
  }
  if (!t.desc) {
    CF_TRY(dalloc(&t.desc, (size_t)kMaxProblems));
    CF_TRY(dalloc(&t.e_prob, (size_t)(kMaxEnergyCtas + kMaxProblems)));
    CF_TRY(dalloc(&t.node_prob, (size_t)w.max_nodes));
  }
  if ((long long)bin_prob.size() > t.bin_cap) {
    dfree(t.bin_prob);
    t.bin_cap = 0;
    h->h_bin_prob.clear();  // the new buffer holds nothing yet
    CF_TRY(dalloc(&t.bin_prob, (size_t)B + kMaxProblems));
    t.bin_cap = (long long)B + kMaxProblems;
  }
  std::vector<int> node_prob;
  node_prob.reserve((size_t)Nt);
  for (int p = 0; p < P; p++) node_prob.insert(node_prob.end(), in[p].N, p);
  CF_TRY(upload_if_changed(t.desc, h->h_desc, in, s));
  CF_TRY(upload_if_changed(t.bin_prob, h->h_bin_prob, bin_prob, s));
  CF_TRY(upload_if_changed(t.e_prob, h->h_e_prob, e_prob, s));
  CF_TRY(upload_if_changed(t.node_prob, h->h_node_prob, node_prob, s));
  t.P = P;
  t.n_bin = (int)bin_prob.size();
  t.n_e = (int)e_prob.size();
  t.M = (int)Mt;
  t.N = (int)Nt;
  t.max_N = maxN;
  t.max_chunk = 0;
  for (int p = 0; p < P; p++) t.max_chunk = std::max(t.max_chunk, in[p].chunk);
  return CF_OK;
}

// Builds the pattern and every topology-derived array from host nodes (the
// problems' nodes concatenated, neighbour ids global; problem p owns rows
// [prob_off[p], prob_off[p+1])).
cf_status build_pattern_host(cf_gn* h, const std::vector<cf_deform_node>& nodes, const std::vector<int>& prob_off) {
  const int N = (int)nodes.size();
  const int P = (int)prob_off.size() - 1;
  // kernels/solver_kernels.cu:498-541: diagonal + directed edges both ways
  std::vector<std::vector<int>> rows(N);
  for (int i = 0; i < N; i++) rows[i].push_back(i);
  for (int i = 0; i < N; i++) {
    int nn = std::min(nodes[i].num_neighbors, CF_K_GRAPH);
    for (int k = 0; k < nn; k++) {
      int nb = nodes[i].neighbors[k];
      if (nb < 0 || nb >= N) continue;
      rows[i].push_back(nb);
      rows[nb].push_back(i);
    }
  }
  std::vector<int> row_ptr(N + 1), col_idx;
  for (int i = 0; i < N; i++) {
    row_ptr[i] = (int)col_idx.size();
    auto& c = rows[i];
    std::sort(c.begin(), c.end());
    c.erase(std::unique(c.begin(), c.end()), c.end());
    col_idx.insert(col_idx.end(), c.begin(), c.end());
  }
  row_ptr[N] = (int)col_idx.size();
  const int nnzb = row_ptr[N];
  auto find = [&](int r, int c) -> int {
    auto b = col_idx.begin() + row_ptr[r], e = col_idx.begin() + row_ptr[r + 1];
    auto it = std::lower_bound(b, e, c);
    return (it != e && *it == c) ? (int)(it - col_idx.begin()) : -1;
  };
  std::vector<int> diag_pos(N), trans_pos(nnzb), upper_pos, upper_row, upper_of_pos(nnzb, -1);
  for (int i = 0; i < N; i++) {
    diag_pos[i] = find(i, i);
    for (int q = row_ptr[i]; q < row_ptr[i + 1]; q++) trans_pos[q] = find(col_idx[q], i);
    for (int q = diag_pos[i]; q < row_ptr[i + 1]; q++) {
      upper_of_pos[q] = (int)upper_pos.size();
      upper_pos.push_back(q);
      upper_row.push_back(i);
    }
  }
  const int n_upper = (int)upper_pos.size();
  // ARAP edges in the reference's visiting order (solver_kernels.cu:225-233)
  std::vector<int> eijk;
  for (int i = 0; i < N; i++) {
    int nn = std::min(nodes[i].num_neighbors, CF_K_GRAPH);
    for (int k = 0; k < nn; k++) {
      int j = nodes[i].neighbors[k];
      if (j < 0 || j >= N || j <= i) continue;
      eijk.push_back(i); eijk.push_back(j); eijk.push_back(k);
    }
  }
  const int n_edges = (int)eijk.size() / 3;
  std::vector<int> arow_ptr(N + 1, 0), ablk_ptr(n_upper + 1, 0);
  for (int e = 0; e < n_edges; e++) {
    arow_ptr[eijk[3 * e] + 1]++;
    arow_ptr[eijk[3 * e + 1] + 1]++;
    int u = upper_of_pos[find(eijk[3 * e], eijk[3 * e + 1])];
    ablk_ptr[u + 1]++;
  }
  for (int i = 0; i < N; i++) arow_ptr[i + 1] += arow_ptr[i];
  for (int u = 0; u < n_upper; u++) ablk_ptr[u + 1] += ablk_ptr[u];
  std::vector<int> arow_inc(std::max(1, arow_ptr[N])), ablk_edge(std::max(1, ablk_ptr[n_upper]));
  {
    std::vector<int> fr(arow_ptr.begin(), arow_ptr.end() - 1), fb(ablk_ptr.begin(), ablk_ptr.end() - 1);
    for (int e = 0; e < n_edges; e++) {
      int i = eijk[3 * e], j = eijk[3 * e + 1];
      arow_inc[fr[i]++] = (e << 1) | 0;
      arow_inc[fr[j]++] = (e << 1) | 1;
      ablk_edge[fb[upper_of_pos[find(i, j)]]++] = e;
    }
  }
  // PCG partition: each problem gets a group of CTAs (in proportion to its
  // blocks, at least one), each CTA contiguous rows of its problem with
  // balanced block counts; per CTA the distinct halo columns and, per block,
  // its operand slot ([own | halo])
  const bool pipe = h->pcg_pipelined != 0;
  int G = h->pcg_ctas_override > 0 ? h->pcg_ctas_override : std::min(h->sms, std::max(1, N / 8));
  G = std::max(P, std::min({G, N, kMaxPcgCtas}));
  if (P > kMaxPcgCtas) return CF_ERR_CAPACITY;
  std::vector<int> rb2, g_vidx(std::max(1, nnzb)), g_halo_ptr, g_halo_col, cta_off2, cta_prob2;
  int smem = 0;
  bool a_smem = true;
  // G CTAs over the problems (one each, the rest by largest share of
  // blocks), each problem's rows split into contiguous ranges of balanced
  // block counts
  auto split_rows = [&](int G_, std::vector<int>& rb, std::vector<int>& cta_off, std::vector<int>& cta_prob) {
    std::vector<int> gp(P, 1);
    {
      std::vector<std::pair<double, int>> rem;
      int left = G_ - P;
      for (int q = 0; q < P; q++) {
        const double share = (double)(row_ptr[prob_off[q + 1]] - row_ptr[prob_off[q]]) / std::max(1, nnzb) * G_;
        int extra = std::min(std::max(0, (int)share - 1), prob_off[q + 1] - prob_off[q] - 1);
        extra = std::max(0, std::min(extra, left));
        gp[q] += extra;
        left -= extra;
        rem.push_back({share - gp[q], q});
      }
      std::sort(rem.begin(), rem.end(), [](const std::pair<double, int>& x, const std::pair<double, int>& y) {
        return x.first != y.first ? x.first > y.first : x.second < y.second;
      });
      for (size_t k = 0; k < rem.size() && left > 0; k++) {
        const int q = rem[k].second;
        if (gp[q] < prob_off[q + 1] - prob_off[q]) {
          gp[q]++;
          left--;
        }
      }
    }
    rb.assign(1, 0);
    cta_off.assign(1, 0);
    cta_prob.clear();
    for (int q = 0; q < P; q++) {
      const int q0 = prob_off[q], q1 = prob_off[q + 1];
      const long long target = ((long long)(row_ptr[q1] - row_ptr[q0]) + gp[q] - 1) / gp[q];
      int start = q0;
      for (int c = 0; c < gp[q] && start < q1; c++) {
        const int rem = gp[q] - c;
        int end = start + 1;
        if (rem == 1) {
          end = q1;
        } else {
          while (end < q1 - (rem - 1) && row_ptr[end] - row_ptr[start] < target) end++;
        }
        rb.push_back(end);
        cta_prob.push_back(q);
        start = end;
      }
      if (q1 == q0) {  // a problem without nodes still owns one (empty) CTA
        rb.push_back(q0);
        cta_prob.push_back(q);
      }
      rb.back() = q1;
      cta_off.push_back((int)cta_prob.size());
    }
  };
  // the shared-memory kernel keeps per row at least the FP64 inverse, the
  // operand and the state vectors (~410 B) and 4 B per block: skip it when
  // that cannot fit in the GPU's shared memory
  const bool grid_fits = (double)N * 410.0 + 4.0 * nnzb < 0.9 * (double)h->sms * 200.0 * 1024.0;
  std::set<int> tried{G};
  for (int attempt = 0; attempt < 64 && h->pcg_mode != 3 && grid_fits; attempt++) {
    std::vector<int> rb, cta_off, cta_prob;
    split_rows(G, rb, cta_off, cta_prob);
    const int Gc = (int)rb.size() - 1;
    g_halo_ptr.assign(1, 0);
    g_halo_col.clear();
    int need_a = 0, need_noa = 0;
    for (int c = 0; c < Gc; c++) {
      const int r0 = rb[c], r1 = rb[c + 1];
      std::vector<int> halo;
      for (int q = row_ptr[r0]; q < row_ptr[r1]; q++)
        if (col_idx[q] < r0 || col_idx[q] >= r1) halo.push_back(col_idx[q]);
      std::sort(halo.begin(), halo.end());
      halo.erase(std::unique(halo.begin(), halo.end()), halo.end());
      for (int q = row_ptr[r0]; q < row_ptr[r1]; q++) {
        int j = col_idx[q];
        g_vidx[q] = (j >= r0 && j < r1) ? j - r0
                                         : (r1 - r0) + (int)(std::lower_bound(halo.begin(), halo.end(), j) - halo.begin());
      }
      g_halo_col.insert(g_halo_col.end(), halo.begin(), halo.end());
      g_halo_ptr.push_back((int)g_halo_col.size());
      const int nb = row_ptr[r1] - row_ptr[r0], nr = r1 - r0, nh = (int)halo.size();
      need_a = std::max(need_a, pcg_grid_smem_bytes(nb, nr, nh, true, pipe));
      need_noa = std::max(need_noa, pcg_grid_smem_bytes(nb, nr, nh, false, pipe));
    }
    const int limit = 200 * 1024;
    a_smem = need_a <= limit;
    smem = a_smem ? need_a : need_noa;
    if (smem > limit) {
      if (G >= std::min(N, kMaxPcgCtas)) break;
      G = std::min(std::min(N, kMaxPcgCtas), G * 2);
      if (!tried.insert(G).second) break;
      continue;
    }
    int cap = pcg_max_active_ctas(smem, a_smem, pipe);
    if (cap < P) break;
    if (Gc > cap) {
      G = cap;
      if (!tried.insert(G).second) break;
      continue;
    }
    rb2 = rb;
    cta_off2 = cta_off;
    cta_prob2 = cta_prob;
    break;
  }
  // systems too large for shared memory (or mode 3): the streaming PCG
  std::vector<int> tile_ptr, tile_row, tile_cols;
  const bool stream = rb2.empty();
  if (stream) {
    const int TB = h->stream_tile == 128 ? 128 : 256;
    const int cap = pcg_stream_max_active_ctas(TB);
    if (cap < P) return CF_ERR_CAPACITY;
    int Gs = h->pcg_ctas_override > 0 ? h->pcg_ctas_override : cap;
    Gs = std::max(P, std::min({Gs, cap, N, kMaxPcgCtas}));
    split_rows(Gs, rb2, cta_off2, cta_prob2);
    tile_ptr.assign(1, 0);
    for (size_t c = 0; c + 1 < rb2.size(); c++) {
      const int r0 = rb2[c], r1 = rb2[c + 1];
      tile_row.push_back(r0);
      for (int i = r0; i < r1; i++)
        if (row_ptr[i + 1] - row_ptr[tile_row.back()] > TB) tile_row.push_back(i);
      if (r1 > r0) tile_row.push_back(r1);  // end of the last tile
      tile_ptr.push_back((int)tile_row.size());
    }
    // each tile's column indices, padded to TB with -1 (a stage's second copy)
    tile_cols.assign(tile_row.size() * (size_t)TB, -1);
    for (size_t c = 0; c + 1 < tile_ptr.size(); c++)
      for (int t = tile_ptr[c]; t + 1 < tile_ptr[c + 1]; t++) {
        const int b0 = row_ptr[tile_row[t]], b1 = row_ptr[tile_row[t + 1]];
        for (int q = b0; q < b1 && q - b0 < TB; q++) tile_cols[(size_t)t * TB + (q - b0)] = col_idx[q];
      }
    g_halo_ptr.assign(rb2.size(), 0);
    g_halo_col.clear();
    smem = pcg_stream_smem_bytes(TB);
    a_smem = false;
  }
  G = (int)rb2.size() - 1;
  std::vector<int> edge_off(P + 1, 0);
  for (int q = 0, e = 0; q <= P; q++) {
    while (q < P && e < n_edges && eijk[3 * e] < prob_off[q]) e++;
    edge_off[q] = (q < P) ? e : n_edges;
  }

  std::vector<int> ustart(N + 1, 0);
  for (int i = 0; i < N; i++) ustart[i + 1] = ustart[i] + (row_ptr[i + 1] - diag_pos[i]);
  // single-cluster PCG plan: rows split over C CTAs in contiguous ranges of
  // balanced block counts.  Per block the operand slot of its column (own row,
  // or the CTA's halo); per halo row its owner and its row there.
  int clu_C = 0, clu_smem = 0, clu_blk = 0, clu_rows = 0, clu_nhalo = 0;
  std::vector<int> clu_rb, clu_vidx(std::max(1, nnzb)), clu_hptr, clu_halo;
  if (h->pcg_mode != 1 && h->pcg_mode != 3 && !stream && P == 1) {
    const int cands[2] = {16, 8};
    for (int ci = 0; ci < 2 && !clu_C; ci++) {
      const int C = cands[ci];
      if (N < C) continue;
      if (h->pcg_mode == 0 && N > kClusterAutoRows * C) continue;
      std::vector<int> rb(1, 0);
      const long long target = ((long long)nnzb + C - 1) / C;
      int start = 0;
      for (int c = 0; c < C; c++) {
        const int rem = C - c;
        int end = start + 1;
        if (rem == 1) {
          end = N;
        } else {
          while (end < N - (rem - 1) && row_ptr[end] - row_ptr[start] < target) end++;
        }
        rb.push_back(end);
        start = end;
      }
      std::vector<int> owner(N), hptr(1, 0), halo;
      for (int c = 0; c < C; c++)
        for (int r = rb[c]; r < rb[c + 1]; r++) owner[r] = c;
      int nb = 0, nr = 0, nh = 0;
      for (int c = 0; c < C; c++) {
        const int r0 = rb[c], r1 = rb[c + 1];
        std::vector<int> cols;  // the CTA's halo
        for (int q = row_ptr[r0]; q < row_ptr[r1]; q++)
          if (col_idx[q] < r0 || col_idx[q] >= r1) cols.push_back(col_idx[q]);
        std::sort(cols.begin(), cols.end());
        cols.erase(std::unique(cols.begin(), cols.end()), cols.end());
        for (int q = row_ptr[r0]; q < row_ptr[r1]; q++) {
          const int j = col_idx[q];
          clu_vidx[q] = (j >= r0 && j < r1) ? j - r0
                                            : (r1 - r0) + (int)(std::lower_bound(cols.begin(), cols.end(), j) - cols.begin());
        }
        for (int j : cols) halo.push_back((owner[j] << 24) | (j - rb[owner[j]]));
        hptr.push_back((int)halo.size());
        nb = std::max(nb, row_ptr[r1] - row_ptr[r0]);
        nr = std::max(nr, r1 - r0);
        nh = std::max(nh, (int)cols.size());
      }
      if (nr > pcg_cluster_max_rows() || nr + nh > 0xffff) continue;
      const int sm = pcg_cluster_smem_bytes(nb, nr, nh, C);
      if (sm > 227 * 1024 - 1024) continue;
      if (pcg_cluster_max_active(C, nr, sm) < 1) continue;
      clu_C = C;
      clu_smem = sm;
      clu_blk = nb;
      clu_rows = nr;
      clu_nhalo = nh;
      clu_rb = rb;
      clu_hptr = hptr;
      clu_halo = halo;
    }
  }
  free_pattern(h->p);
  Pattern& p = h->p;
  p.P = P;
  p.N = N;
  p.nnzb = nnzb;
  p.n_upper = n_upper;
  p.n_edges = n_edges;
  p.pcg_ctas = G;
  p.pcg_smem = smem;
  p.pcg_a_in_smem = a_smem ? 1 : 0;
  p.pcg_pipelined = pipe ? 1 : 0;
  p.pcg_stream = stream ? 1 : 0;
  p.st_tile_blocks = h->stream_tile == 128 ? 128 : 256;
  auto up = [](int** d, const std::vector<int>& v) -> cudaError_t {
    cudaError_t e = dalloc(d, v.size());
    if (e != cudaSuccess) return e;
    return v.empty() ? cudaSuccess : cudaMemcpy(*d, v.data(), v.size() * sizeof(int), cudaMemcpyHostToDevice);
  };
  CF_TRY(up(&p.row_ptr, row_ptr));
  CF_TRY(up(&p.col_idx, col_idx));
  CF_TRY(up(&p.diag_pos, diag_pos));
  {
    std::vector<int4> meta(n_upper);
    for (int u = 0; u < n_upper; u++) {
      const int q = upper_pos[u];
      meta[u] = make_int4(upper_row[u], q, col_idx[q], trans_pos[q]);
    }
    CF_TRY(dalloc(&p.upper_meta, (size_t)n_upper));
    CF_TRY(cudaMemcpy(p.upper_meta, meta.data(), meta.size() * sizeof(int4), cudaMemcpyHostToDevice));
  }
  CF_TRY(up(&p.arap_row_ptr, arow_ptr));
  CF_TRY(up(&p.arap_row_inc, arow_inc));
  CF_TRY(up(&p.arap_blk_ptr, ablk_ptr));
  CF_TRY(up(&p.arap_blk_edge, ablk_edge));
  CF_TRY(up(&p.edge_ijk, eijk));
  CF_TRY(dalloc(&p.edge_terms, (size_t)kEdgeTerms4 * std::max(1, n_edges)));
  CF_TRY(dalloc(&p.edge_energy, (size_t)std::max(1, n_edges)));
  CF_TRY(up(&p.pcg_row_begin, rb2));
  CF_TRY(up(&p.pcg_cta_off, cta_off2));
  CF_TRY(up(&p.pcg_prob, cta_prob2));
  CF_TRY(up(&p.prob_edge_off, edge_off));
  if (stream) {
    CF_TRY(up(&p.st_tile_ptr, tile_ptr));
    CF_TRY(up(&p.st_tile_row, tile_row));
    CF_TRY(up(&p.st_tile_cols, tile_cols));
    Work& w = h->w;
    if (!w.minv32) {
      CF_TRY(dalloc(&w.r, 6 * (size_t)w.max_nodes));
      CF_TRY(dalloc(&w.ap, 6 * (size_t)w.max_nodes));
      CF_TRY(dalloc(&w.zp, 24 * (size_t)w.max_nodes));
      CF_TRY(dalloc(&w.minv32, 36 * (size_t)w.max_nodes));
    }
  }
  CF_TRY(up(&p.g_vidx, g_vidx));
  CF_TRY(up(&p.g_halo_ptr, g_halo_ptr));
  CF_TRY(up(&p.g_halo_col, g_halo_col));
  p.use_cluster = clu_C ? 1 : 0;
  p.clu_C = clu_C;
  p.clu_smem = clu_smem;
  p.clu_blk_max = clu_blk;
  p.clu_rows_max = clu_rows;
  p.clu_halo_max = clu_nhalo;
  CF_TRY(up(&p.ustart, ustart));
  if (clu_C) {
    CF_TRY(up(&p.clu_row_begin, clu_rb));
    CF_TRY(up(&p.clu_vidx, clu_vidx));
    CF_TRY(up(&p.clu_halo_ptr, clu_hptr));
    CF_TRY(up(&p.clu_halo, clu_halo.empty() ? std::vector<int>(1, 0) : clu_halo));
  }
  CF_TRY(dalloc(&p.values, (size_t)nnzb * 36));
  CF_TRY(cudaMemset(p.values, 0, sizeof(float) * (size_t)std::max(1, nnzb) * 36));
  h->h_row_ptr = row_ptr;
  h->h_col_idx = col_idx;
  h->pattern_version++;
  h->pattern_valid = true;
  return CF_OK;
}

// The pattern of a single problem, rebuilt when N changes (the reference's
// cache key, kernels/solver_kernels.cu:545-549) or after invalidation.
cf_status ensure_pattern(cf_gn* h, const cf_deform_node* d_nodes, int N, cudaStream_t s) {
  const std::vector<int> key{N};
  if (h->pattern_valid && h->pattern_key == key) return CF_OK;
  std::vector<cf_deform_node> hn(N);
  CF_TRY(cudaMemcpyAsync(hn.data(), d_nodes, sizeof(cf_deform_node) * (size_t)N, cudaMemcpyDeviceToHost, s));
  CF_TRY(cudaStreamSynchronize(s));
  cf_status st = build_pattern_host(h, hn, {0, N});
  if (st == CF_OK) h->pattern_key = key;
  return st;
}

// The block-diagonal pattern of a batch, rebuilt when the problem sizes
// change or after invalidation.
cf_status ensure_pattern_batch(cf_gn* h, const std::vector<ProbDesc>& pr, cudaStream_t s) {
  std::vector<int> key{-(int)pr.size()};
  for (auto& d : pr) key.push_back(d.N);
  if (h->pattern_valid && h->pattern_key == key) return CF_OK;
  std::vector<int> off(1, 0);
  for (auto& d : pr) off.push_back(off.back() + d.N);
  std::vector<cf_deform_node> hn(off.back());
  for (size_t q = 0; q < pr.size(); q++)
    CF_TRY(cudaMemcpyAsync(hn.data() + off[q], pr[q].nodes, sizeof(cf_deform_node) * (size_t)pr[q].N,
                           cudaMemcpyDeviceToHost, s));
  CF_TRY(cudaStreamSynchronize(s));
  for (size_t q = 0; q < pr.size(); q++)
    for (int i = off[q]; i < off[q + 1]; i++) {
      cf_deform_node& nd = hn[i];
      const int nn = std::min(std::max(nd.num_neighbors, 0), CF_K_GRAPH);
      for (int k = 0; k < CF_K_GRAPH; k++) {
        const int j = nd.neighbors[k];
        nd.neighbors[k] = (k < nn && j >= 0 && j < pr[q].N) ? j + off[q] : -1;
      }
    }
  cf_status st = build_pattern_host(h, hn, off);
  if (st == CF_OK) h->pattern_key = key;
  return st;
}

// Per-solve sort of the correspondences by their node sets (counting sort by
// the first node, then within each node's bucket) and the nodes' task lists;
// resets the error word and, when asked, the statistics, and sets up the nodes.
cf_status bin_correspondences(cf_gn* h, bool reset_stats, cudaStream_t s) {
  Work& w = h->w;
  const Table& t = h->tb;
  if (t.n_bin > 0) {
    { Timed tm(h, s, kProfPack, 1); CF_TRY(launch_key_count(w, t, s)); }
    { Timed tm(h, s, kProfBinScan, 2); CF_TRY(launch_bin_scan(w, t, reset_stats, s)); }
    { Timed tm(h, s, kProfScatter, 1); CF_TRY(launch_bin_scatter(w, t, s)); }
    { Timed tm(h, s, kProfSort, 1); CF_TRY(launch_bucket_sort(w, t, s)); }
    { Timed tm(h, s, kProfLists, 3); CF_TRY(launch_list_scan(w, t, s)); CF_TRY(launch_node_lists(w, t, h->p, s)); }
  } else {
    CF_TRY(cudaMemsetAsync(w.inc_start, 0, sizeof(int) * (size_t)(t.N + 1), s));
    CF_TRY(cudaMemsetAsync(w.cl_start, 0, sizeof(int) * (size_t)(t.N + 1), s));
    { Timed tm(h, s, kProfNodePlain, 1); CF_TRY(launch_node_setup(w, t, reset_stats, s)); }
  }
  return CF_OK;
}

cudaError_t launch_pcg_any(cf_gn* h, const SolveArgs& a, int slot, cudaStream_t s) {
  if (h->p.use_cluster) return launch_pcg_cluster(h->w, h->p, a, slot, s);
  if (h->p.pcg_stream) return launch_pcg_stream(h->w, h->p, a, slot, s);
  return launch_pcg(h->w, h->p, a, slot, s);
}

SolveArgs make_args(const cf_gn* h, const cf_deform_node* nodes, int N, int M) {
  SolveArgs a;
  memset(&a, 0, sizeof(a));
  a.nodes = nodes;
  a.N = N;
  a.M = M;
  a.lambda_smooth = h->params.lambda_smooth;
  a.lambda_damping = h->params.lambda_damping;
  a.pcg_iterations = std::max(0, h->params.pcg_iterations);
  a.pcg_tolerance = h->params.pcg_tolerance;
  a.arap_consistent = h->arap_consistent;
  a.spin_limit = h->spin_limit;
  a.bar_extra = h->bar_extra;
  a.timers = h->phase_timers ? h->w.timers : nullptr;
  a.tb = h->tb;
  return a;
}

ProbDesc make_desc(const cf_correspondence* corrs, const float* canon, const cf_deform_node* nodes,
                   cf_dual_quat* T, int M, int N, float max_rot, float max_trans, float scale) {
  ProbDesc d;
  memset(&d, 0, sizeof(d));
  d.corrs = corrs;
  d.canon = canon;
  d.nodes = nodes;
  d.T = T;
  d.M = M;
  d.N = N;
  d.max_rot = max_rot;
  d.max_trans = max_trans;
  d.update_scale = scale;
  return d;
}

}  // namespace

namespace {

// G GN iterations and the final energy over the current table.
cf_status run_gn(cf_gn* h, SolveArgs& a, cudaStream_t s) {
  Work& w = h->w;
  const int G = h->params.gn_iterations;
  for (int g = 0; g < G; g++) {
    { Timed t(h, s, kProfResidual, 1); CF_TRY(launch_residual(w, h->tb, h->p, a, a.transforms, true, s)); }
    { Timed t(h, s, kProfAssemble, 1); CF_TRY(launch_assemble(w, h->p, a, s)); }
    { Timed t(h, s, kProfPcg, 1); CF_TRY(launch_pcg_any(h, a, g, s)); }
  }
  { Timed t(h, s, kProfEnergy, a.tb.P > 1 ? 2 : 1); CF_TRY(launch_final_energy(w, h->p, a, G, s)); }
  h->last_gn = G;
  return CF_OK;
}

// Per-problem statistics (out[o] from table problem slot_of[o], -1: none)
// and the error word; synchronises.
cf_status read_stats(cf_gn* h, cf_solve_stats* stats, const std::vector<int>& slot_of, int n_out, cudaStream_t s) {
  Work& w = h->w;
  const int P = h->tb.P, G = h->params.gn_iterations;
  CF_TRY(cudaMemcpyAsync(h->h_stats, w.stats, sizeof(DevStats) * (size_t)P, cudaMemcpyDeviceToHost, s));
  int herr = 0;
  CF_TRY(cudaMemcpyAsync(&herr, w.err, sizeof(int), cudaMemcpyDeviceToHost, s));
  CF_TRY(cudaStreamSynchronize(s));
  for (int o = 0; o < n_out; o++) {
    cf_solve_stats* out = stats + o;
    memset(out, 0, sizeof(*out));
    const int q = slot_of[o];
    if (q < 0) continue;
    const DevStats& d = h->h_stats[q];
    out->energy_initial = d.energy[0];
    out->energy_final = d.energy[G];
    for (int g = 0; g <= G && g < CF_MAX_GN_ITERS; g++) out->energy_per_iter[g] = d.energy[g];
    for (int g = 0; g < G; g++) {
      out->pcg_iterations[g] = d.pcg_iters[g];
      out->pcg_residual[g] = d.pcg_res[g];
    }
    out->gn_iterations_run = G;
    out->num_blocks = h->p.nnzb;
    out->precond_fallbacks = d.fallbacks;
    out->error_flags = herr;
    out->energy_warm_start = d.gate[0];
    out->energy_predicted = d.gate[1];
    out->init_rejected = d.init_rejected;
  }
  if (herr & kErrTimeoutBit) return CF_ERR_TIMEOUT;
  if (herr & kErrNonFiniteBit) return CF_ERR_NON_FINITE;
  return CF_OK;
}

// The device work of a solve after the host-side preparation: statistics
// reset, (batched: gather), binning, G GN iterations, final energy,
// (batched: scatter).  kind 0: single problem, 1: batch.
cf_status enqueue_solve(cf_gn* h, int kind, SolveArgs& a, cudaStream_t s) {
  Work& w = h->w;
  if (kind == 1) {
    Timed t(h, s, kProfOther, 1);
    CF_TRY(launch_batch_gather(w, h->tb, s));
  }
  cf_status st = bin_correspondences(h, true, s);
  if (st != CF_OK) return st;
  if (kind == 2) {
    // learned start: features at the warm start, the network's increment,
    // kept only if it lowers the energy (the plain warm start otherwise)
    Mpnn& net = *h->learn_net;
      // the warm start's energy, and each task's residual statistics for the features
    { Timed t(h, s, kProfEnergy, 1); CF_TRY(launch_final_energy(w, h->p, a, -1, s, true)); }
    {
      Timed t(h, s, kProfLearned, 6);
      CF_TRY(launch_features(w, a.transforms, h->learn_hist, a.N, net.feat, s));
      CF_TRY(mpnn_graph_from_nodes(net, a.nodes, a.N, s));
      CF_TRY(mpnn_forward(net, net.feat, net.out, s));
    }
    { Timed t(h, s, kProfLearned, 1); CF_TRY(launch_apply_prediction(w, a.transforms, a.nodes, net.out, a.N, s)); }
    { Timed t(h, s, kProfEnergy, 1); CF_TRY(launch_final_energy(w, h->p, a, -2, s)); }
    { Timed t(h, s, kProfLearned, 1); CF_TRY(launch_gate_prediction(w, a.transforms, a.nodes, a.N, s)); }
  }
  st = run_gn(h, a, s);
  if (st != CF_OK) return st;
  if (kind == 1) {
    Timed t(h, s, kProfOther, 1);
    CF_TRY(launch_batch_scatter(w, h->tb, s));
  }
  return CF_OK;
}

// Runs enqueue_solve as a CUDA graph: captured once per distinct set of
// launch arguments (the problem table itself lives in device memory, so new
// caller buffers of the same sizes replay the same graph), replayed after.
// Falls back to direct launches when graphs are off, while profiling, on the
// legacy default stream, inside a caller's own capture, or if capture fails.
cf_status solve_graphed(cf_gn* h, int kind, SolveArgs& a, cudaStream_t s) {
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  h->graph_last = 0;
  if (!h->use_graph || h->profile || s == nullptr || cudaStreamIsCapturing(s, &cs) != cudaSuccess ||
      cs != cudaStreamCaptureStatusNone)
    return enqueue_solve(h, kind, a, s);
  std::vector<unsigned char> key(sizeof(int) * 2 + sizeof(unsigned) + sizeof(cf_gn_params) + sizeof(SolveArgs) +
                                 2 * sizeof(void*));
  unsigned char* k = key.data();
  const void* lp[2] = {kind == 2 ? (const void*)h->learn_net : nullptr, kind == 2 ? (const void*)h->learn_hist : nullptr};
  memcpy(k, lp, sizeof(lp)); k += sizeof(lp);
  memcpy(k, &kind, sizeof(int)); k += sizeof(int);
  memcpy(k, &h->tb.P, sizeof(int)); k += sizeof(int);
  memcpy(k, &h->pattern_version, sizeof(unsigned)); k += sizeof(unsigned);
  memcpy(k, &h->params, sizeof(cf_gn_params)); k += sizeof(cf_gn_params);
  memcpy(k, &a, sizeof(SolveArgs));
  if (key == h->graph_key) {
    if (h->graph_key_failed) return enqueue_solve(h, kind, a, s);
    h->launches += h->graph_launches;
    CF_TRY(cudaGraphLaunch(h->graph_exec, s));
    h->graph_last = 1;
    return CF_OK;
  }
  if (h->graph_exec) {
    cudaGraphExecDestroy(h->graph_exec);
    h->graph_exec = nullptr;
  }
  h->graph_key = key;
  h->graph_key_failed = false;
  const long long before = h->launches;
  cudaGraph_t g = nullptr;
  cf_status st = from_cuda(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
  if (st == CF_OK) {
    st = enqueue_solve(h, kind, a, s);
    const cudaError_t e = cudaStreamEndCapture(s, &g);
    if (st == CF_OK && e != cudaSuccess) st = from_cuda(e);
    if (st == CF_OK && cudaGraphInstantiate(&h->graph_exec, g, 0) != cudaSuccess) st = CF_ERR_CUDA;
  }
  if (g) cudaGraphDestroy(g);
  h->graph_launches = h->launches - before;
  h->launches = before;
  if (st != CF_OK) {  // not capturable here: remember, and launch directly
    cudaGetLastError();
    if (h->graph_exec) cudaGraphExecDestroy(h->graph_exec);
    h->graph_exec = nullptr;
    h->graph_key_failed = true;
    return enqueue_solve(h, kind, a, s);
  }
  h->launches += h->graph_launches;
  CF_TRY(cudaGraphLaunch(h->graph_exec, s));
  h->graph_last = 1;
  return CF_OK;
}

}  // namespace

extern "C" {

const char* cf_status_string(cf_status s) {
  switch (s) {
    case CF_OK: return "ok";
    case CF_ERR_INVALID_ARG: return "invalid argument";
    case CF_ERR_OOM: return "device out of memory";
    case CF_ERR_NON_FINITE: return "non-finite value in the solution or energy";
    case CF_ERR_TIMEOUT: return "in-kernel barrier timed out";
    case CF_ERR_CUDA: return "CUDA error";
    case CF_ERR_CAPACITY: return "size exceeds the handle's capacity";
    case CF_ERR_NOT_IMPLEMENTED: return "not implemented";
    case CF_ERR_NO_DEVICE: return "no CUDA device";
  }
  return "unknown status";
}

cf_status cf_gn_params_default(cf_gn_params* p) {
  if (!p) return CF_ERR_INVALID_ARG;
  p->gn_iterations = 3;
  p->pcg_iterations = 10;
  p->pcg_tolerance = 1e-4f;
  p->lambda_smooth = 1.0f;
  p->lambda_rot = 1.0f;
  p->lambda_damping = 1e-2f;
  p->debug = 0;
  return CF_OK;
}

cf_status cf_gn_create(const cf_gn_params* params, int max_nodes, int max_corrs, cf_gn** out) {
  if (!out) return CF_ERR_INVALID_ARG;
  *out = nullptr;
  if (!params || max_nodes <= 0 || max_corrs < 0 || max_corrs >= (1 << 26)) return CF_ERR_INVALID_ARG;
  if (params->gn_iterations < 0 || params->gn_iterations > CF_MAX_GN_ITERS || params->pcg_iterations < 0)
    return CF_ERR_INVALID_ARG;
  int dev = 0, count = 0;
  cudaError_t e = cudaGetDeviceCount(&count);
  if (e != cudaSuccess || count == 0) {
    snprintf(g_last_error, sizeof(g_last_error), "%s", cudaGetErrorString(e));
    return CF_ERR_NO_DEVICE;
  }
  CF_TRY(cudaGetDevice(&dev));
  cf_gn* h = new cf_gn();
  h->params = *params;
  h->max_nodes = max_nodes;
  h->max_corrs = max_corrs;
  h->device = dev;
  cudaDeviceGetAttribute(&h->sms, cudaDevAttrMultiProcessorCount, dev);
  e = alloc_work(h->w, max_nodes, max_corrs, 2 * h->sms);
  if (e == cudaSuccess) e = cudaMallocHost((void**)&h->h_stats, sizeof(DevStats) * (size_t)kMaxProblems);
  if (e != cudaSuccess) {
    free_work(h->w);
    delete h;
    return from_cuda(e);
  }
  *out = h;
  return CF_OK;
}

cf_status cf_gn_destroy(cf_gn* h) {
  if (!h) return CF_ERR_INVALID_ARG;
  cudaDeviceSynchronize();
  if (h->graph_exec) cudaGraphExecDestroy(h->graph_exec);
  free_pattern(h->p);
  free_work(h->w);
  free_table(h->tb);
  if (h->h_stats) cudaFreeHost(h->h_stats);
  for (auto& pe : h->prof_pool) {
    cudaEventDestroy(pe.a);
    cudaEventDestroy(pe.b);
  }
  delete h;
  return CF_OK;
}

cf_status cf_gn_set_params(cf_gn* h, const cf_gn_params* params) {
  if (!h || !params || params->gn_iterations < 0 || params->gn_iterations > CF_MAX_GN_ITERS ||
      params->pcg_iterations < 0)
    return CF_ERR_INVALID_ARG;
  h->params = *params;
  return CF_OK;
}

cf_status cf_gn_get_params(const cf_gn* h, cf_gn_params* params) {
  if (!h || !params) return CF_ERR_INVALID_ARG;
  *params = h->params;
  return CF_OK;
}

cf_status cf_gn_set_option(cf_gn* h, int option, int value) {
  if (!h) return CF_ERR_INVALID_ARG;
  switch (option) {
    case CF_OPT_ARAP_CONSISTENT:
      h->arap_consistent = value ? 1 : 0;
      return CF_OK;
    case CF_OPT_PCG_PIPELINED:
      h->pcg_pipelined = value ? 1 : 0;
      h->pattern_valid = false;
      return CF_OK;
    case CF_OPT_PCG_MODE:
      if (value < 0 || value > 3) return CF_ERR_INVALID_ARG;
      h->pcg_mode = value;
      h->pattern_valid = false;
      return CF_OK;
    case CF_OPT_GRAPH:
      h->use_graph = value ? 1 : 0;
      return CF_OK;
    case CF_OPT_SPIN_LIMIT:
      if (value < 0) return CF_ERR_INVALID_ARG;
      h->spin_limit = value ? (unsigned)value : (1u << 22);
      return CF_OK;
    case CF_OPT_TEST_BARRIER_EXTRA:
      if (value < 0) return CF_ERR_INVALID_ARG;
      h->bar_extra = (unsigned)value;
      return CF_OK;
    case CF_OPT_STREAM_TILE:
      if (value != 0 && value != 128 && value != 256) return CF_ERR_INVALID_ARG;
      h->stream_tile = value ? value : 256;
      h->pattern_valid = false;
      return CF_OK;
    case CF_OPT_PCG_CTAS:
      if (value < 0 || value > kMaxPcgCtas) return CF_ERR_INVALID_ARG;
      h->pcg_ctas_override = value;
      h->pattern_valid = false;
      return CF_OK;
  }
  return CF_ERR_INVALID_ARG;
}

cf_status cf_gn_get_option(const cf_gn* h, int option, int* value) {
  if (!h || !value) return CF_ERR_INVALID_ARG;
  switch (option) {
    case CF_OPT_ARAP_CONSISTENT: *value = h->arap_consistent; return CF_OK;
    case CF_OPT_PCG_CTAS: *value = h->pcg_ctas_override; return CF_OK;
    case CF_OPT_PCG_MODE: *value = h->pcg_mode; return CF_OK;
    case CF_OPT_PCG_PIPELINED: *value = h->pcg_pipelined; return CF_OK;
    case CF_OPT_GRAPH: *value = h->use_graph; return CF_OK;
    case CF_OPT_GRAPH_ACTIVE: *value = h->graph_last; return CF_OK;
    case CF_OPT_SPIN_LIMIT: *value = (int)h->spin_limit; return CF_OK;
    case CF_OPT_TEST_BARRIER_EXTRA: *value = (int)h->bar_extra; return CF_OK;
    case CF_OPT_STREAM_TILE: *value = h->stream_tile; return CF_OK;
    case CF_OPT_PCG_ACTIVE:
      *value = !h->pattern_valid ? 0 : h->p.use_cluster ? 2 : h->p.pcg_stream ? 3 : 1;
      return CF_OK;
  }
  return CF_ERR_INVALID_ARG;
}

cf_status cf_gn_invalidate_pattern(cf_gn* h) {
  if (!h) return CF_ERR_INVALID_ARG;
  h->pattern_valid = false;
  return CF_OK;
}

cf_status cf_gn_linearize_solve(cf_gn* h, const cf_correspondence* d_corrs, int num_corrs,
                                const cf_deform_node* d_nodes, const cf_dual_quat* d_transforms, int num_nodes,
                                float* d_delta_x, void* stream) {
  if (!h || num_corrs < 0 || num_nodes < 0) return CF_ERR_INVALID_ARG;
  if (num_nodes > h->max_nodes || num_corrs > h->max_corrs) return CF_ERR_CAPACITY;
  if (num_nodes == 0) return CF_OK;
  if (!d_nodes || !d_transforms || !d_delta_x || (num_corrs > 0 && !d_corrs)) return CF_ERR_INVALID_ARG;
  if ((reinterpret_cast<uintptr_t>(d_corrs) & 3u) || (reinterpret_cast<uintptr_t>(d_transforms) & 15u))
    return CF_ERR_INVALID_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  cf_status st = ensure_pattern(h, d_nodes, num_nodes, s);
  if (st != CF_OK) return st;
  st = prepare_table(h, {make_desc(d_corrs, nullptr, d_nodes, const_cast<cf_dual_quat*>(d_transforms), num_corrs,
                                   num_nodes, 0.f, 0.f, 1.f)},
                     true, s);
  if (st != CF_OK) return st;
  Work& w = h->w;
  st = bin_correspondences(h, true, s);
  if (st != CF_OK) return st;
  SolveArgs a = make_args(h, d_nodes, num_nodes, num_corrs);
  a.delta_x = d_delta_x;
  { Timed t(h, s, kProfResidual, 1); CF_TRY(launch_residual(w, h->tb, h->p, a, d_transforms, false, s)); }
  { Timed t(h, s, kProfAssemble, 1); CF_TRY(launch_assemble(w, h->p, a, s)); }
  { Timed t(h, s, kProfPcg, 1); CF_TRY(launch_pcg_any(h, a, 0, s)); }
  h->last_gn = 1;
  return CF_OK;
}

cf_status cf_gn_solve(cf_gn* h, const cf_problem* prob, cf_dual_quat* d_transforms, cf_solve_stats* stats,
                      void* stream) {
  if (!h || !prob || prob->num_nodes < 0 || prob->num_corrs < 0) return CF_ERR_INVALID_ARG;
  const int N = prob->num_nodes, M = prob->num_corrs;
  if (N > h->max_nodes || M > h->max_corrs) return CF_ERR_CAPACITY;
  if (stats) memset(stats, 0, sizeof(*stats));
  if (N == 0) return CF_OK;
  if (!prob->nodes || !d_transforms || (M > 0 && (!prob->corrs || !prob->canon_points))) return CF_ERR_INVALID_ARG;
  if ((reinterpret_cast<uintptr_t>(prob->corrs) & 3u) || (reinterpret_cast<uintptr_t>(d_transforms) & 15u))
    return CF_ERR_INVALID_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  cf_status st = ensure_pattern(h, prob->nodes, N, s);
  if (st != CF_OK) return st;
  st = prepare_table(h, {make_desc(prob->corrs, prob->canon_points, prob->nodes, d_transforms, M, N, prob->max_rot,
                                   prob->max_trans, prob->update_scale)},
                     true, s);
  if (st != CF_OK) return st;
  SolveArgs a = make_args(h, prob->nodes, N, M);
  a.transforms = d_transforms;
  a.max_rot = prob->max_rot;
  a.max_trans = prob->max_trans;
  a.update_scale = prob->update_scale;
  st = solve_graphed(h, 0, a, s);
  if (st != CF_OK || !stats) return st;
  return read_stats(h, stats, {0}, 1, s);
}

cf_status cf_gn_solve_batched(cf_gn* h, const cf_problem* problems, int num_problems,
                              cf_dual_quat* const* d_transforms, cf_solve_stats* stats, void* stream) {
  if (!h || num_problems < 0 || (num_problems > 0 && (!problems || !d_transforms))) return CF_ERR_INVALID_ARG;
  if (num_problems > kMaxProblems) return CF_ERR_CAPACITY;
  std::vector<ProbDesc> pr;
  std::vector<int> slot_of(num_problems, -1);
  long long Nt = 0, Mt = 0;
  for (int q = 0; q < num_problems; q++) {
    const cf_problem& p = problems[q];
    if (p.num_nodes < 0 || p.num_corrs < 0) return CF_ERR_INVALID_ARG;
    if (p.num_nodes == 0) continue;  // nothing to solve; its statistics stay zero
    if (!p.nodes || !d_transforms[q] || (p.num_corrs > 0 && (!p.corrs || !p.canon_points))) return CF_ERR_INVALID_ARG;
    if ((reinterpret_cast<uintptr_t>(p.corrs) & 3u) || (reinterpret_cast<uintptr_t>(d_transforms[q]) & 15u))
      return CF_ERR_INVALID_ARG;
    slot_of[q] = (int)pr.size();
    pr.push_back(make_desc(p.corrs, p.canon_points, p.nodes, d_transforms[q], p.num_corrs, p.num_nodes, p.max_rot,
                           p.max_trans, p.update_scale));
    Nt += p.num_nodes;
    Mt += p.num_corrs;
  }
  if (Nt > h->max_nodes || Mt > h->max_corrs) return CF_ERR_CAPACITY;
  if (stats) memset(stats, 0, sizeof(*stats) * (size_t)num_problems);
  if (pr.empty()) return CF_OK;
  cudaStream_t s = (cudaStream_t)stream;
  cf_status st = ensure_pattern_batch(h, pr, s);
  if (st != CF_OK) return st;
  st = prepare_table(h, pr, false, s);
  if (st != CF_OK) return st;
  Work& w = h->w;
  if (!w.nodes_cat) {
    CF_TRY(dalloc(&w.nodes_cat, (size_t)w.max_nodes));
    CF_TRY(dalloc(&w.T_cat, (size_t)w.max_nodes));
  }
  SolveArgs a = make_args(h, w.nodes_cat, (int)Nt, (int)Mt);
  a.transforms = w.T_cat;
  st = solve_graphed(h, 1, a, s);
  if (st != CF_OK || !stats) return st;
  return read_stats(h, stats, slot_of, num_problems, s);
}

// ---- autotuner ------------------------------------------------------------

namespace {

struct TuneChoice {
  int pcg_mode, pcg_ctas, stream_tile;
  double ms_best, ms_default;
};

std::mutex g_tune_mu;
std::map<std::string, TuneChoice> g_tune_cache;
bool g_tune_loaded = false;

const char* tune_file() { return getenv("CF_AUTOTUNE_CACHE"); }

void tune_load_locked() {
  if (g_tune_loaded) return;
  g_tune_loaded = true;
  const char* path = tune_file();
  if (!path) return;
  FILE* f = fopen(path, "r");
  if (!f) return;
  char key[512];
  TuneChoice c;
  while (fscanf(f, "%511s %d %d %d %lf %lf", key, &c.pcg_mode, &c.pcg_ctas, &c.stream_tile, &c.ms_best,
                &c.ms_default) == 6)
    g_tune_cache[key] = c;
  fclose(f);
}

void tune_store_locked(const std::string& key, const TuneChoice& c) {
  g_tune_cache[key] = c;
  const char* path = tune_file();
  if (!path) return;
  FILE* f = fopen(path, "a");
  if (!f) return;
  fprintf(f, "%s %d %d %d %.6f %.6f\n", key.c_str(), c.pcg_mode, c.pcg_ctas, c.stream_tile, c.ms_best,
          c.ms_default);
  fclose(f);
}

// the shape of a tuning problem: device, sizes and the solver settings the
// PCG's speed depends on
std::string tune_key(const cf_gn* h, const cf_problem* pr, int num) {
  long long N = 0, M = 0;
  for (int q = 0; q < num; q++) {
    N += pr[q].num_nodes;
    M += pr[q].num_corrs;
  }
  char buf[256];
  snprintf(buf, sizeof(buf), "sm%d/P%d/N%lld/M%lld/G%d/I%d/pipe%d", h->sms, num, N, M, h->params.gn_iterations,
           h->params.pcg_iterations, h->pcg_pipelined);
  return buf;
}

}  // namespace

cf_status cf_gn_autotune(cf_gn* h, const cf_problem* problems, int num_problems, cf_dual_quat* const* d_transforms,
                         cf_tune_result* out, void* stream) {
  if (!h || !problems || !d_transforms || num_problems < 1) return CF_ERR_INVALID_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  const std::string key = tune_key(h, problems, num_problems);
  {
    std::lock_guard<std::mutex> lock(g_tune_mu);
    tune_load_locked();
    auto it = g_tune_cache.find(key);
    if (it != g_tune_cache.end()) {
      const TuneChoice& c = it->second;
      h->pcg_mode = c.pcg_mode;
      h->pcg_ctas_override = c.pcg_ctas;
      h->stream_tile = c.stream_tile;
      h->pattern_valid = false;
      if (out) *out = cf_tune_result{c.pcg_mode, c.pcg_ctas, c.stream_tile, 0, c.ms_best, c.ms_default, 1};
      return CF_OK;
    }
  }
  // scratch copies of the transforms: the candidates never touch the caller's
  std::vector<cf_dual_quat*> scratch(num_problems, nullptr);
  cf_status st = CF_OK;
  for (int q = 0; q < num_problems && st == CF_OK; q++) {
    const size_t n = (size_t)std::max(problems[q].num_nodes, 1);
    if (cudaMalloc(&scratch[q], sizeof(cf_dual_quat) * n) != cudaSuccess) st = CF_ERR_OOM;
  }
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  if (st == CF_OK && (cudaEventCreate(&e0) != cudaSuccess || cudaEventCreate(&e1) != cudaSuccess)) st = CF_ERR_CUDA;
  const int mode0 = h->pcg_mode, ctas0 = h->pcg_ctas_override, tile0 = h->stream_tile;
  struct Cand {
    int mode, ctas, tile;
  };
  std::vector<Cand> cands = {{mode0, ctas0, tile0}};  // the configuration in effect first: the baseline
  for (int ctas : {0, h->sms, 2 * h->sms}) cands.push_back({1, ctas, 256});
  if (num_problems == 1) cands.push_back({2, 0, 256});
  for (int tile : {256, 128})
    for (int ctas : {0, h->sms}) cands.push_back({3, ctas, tile});
  double best = 1e30, baseline = 0.0;
  Cand pick = cands[0];
  int timed = 0;
  std::set<std::vector<int>> seen;  // effective configurations already timed
  for (const Cand& c : cands) {
    if (st != CF_OK) break;
    h->pcg_mode = c.mode;
    h->pcg_ctas_override = c.ctas;
    h->stream_tile = c.tile;
    h->pattern_valid = false;
    auto run = [&]() -> cf_status {
      for (int q = 0; q < num_problems; q++)
        if (problems[q].num_nodes > 0)
          CF_TRY(cudaMemcpyAsync(scratch[q], d_transforms[q], sizeof(cf_dual_quat) * problems[q].num_nodes,
                                 cudaMemcpyDeviceToDevice, s));
      return num_problems == 1 ? cf_gn_solve(h, problems, scratch[0], nullptr, s)
                               : cf_gn_solve_batched(h, problems, num_problems, scratch.data(), nullptr, s);
    };
    cf_status r = run();  // builds the pattern, captures the graph
    if (r == CF_ERR_CAPACITY) continue;  // not feasible at this size
    if (r != CF_OK) {
      st = r;
      break;
    }
    const std::vector<int> eff{h->p.pcg_stream, h->p.pcg_ctas, h->p.use_cluster, h->p.st_tile_blocks};
    if (!seen.insert(eff).second && timed > 0) continue;
    std::vector<float> ms;
    for (int k = 0; k < 3 && st == CF_OK; k++) {
      cudaEventRecord(e0, s);
      st = run();
      cudaEventRecord(e1, s);
      if (cudaEventSynchronize(e1) != cudaSuccess) st = CF_ERR_CUDA;
      float t = 0.f;
      cudaEventElapsedTime(&t, e0, e1);
      ms.push_back(t);
    }
    if (st != CF_OK) break;
    std::sort(ms.begin(), ms.end());
    const double med = ms[ms.size() / 2];
    if (timed == 0) baseline = med;
    timed++;
    if (med < best) {
      best = med;
      pick = c;
    }
  }
  if (e0) cudaEventDestroy(e0);
  if (e1) cudaEventDestroy(e1);
  cudaStreamSynchronize(s);
  for (auto p : scratch)
    if (p) cudaFree(p);
  h->pcg_mode = st == CF_OK ? pick.mode : mode0;
  h->pcg_ctas_override = st == CF_OK ? pick.ctas : ctas0;
  h->stream_tile = st == CF_OK ? pick.tile : tile0;
  h->pattern_valid = false;
  if (st != CF_OK) return st;
  const TuneChoice choice{pick.mode, pick.ctas, pick.tile, best, baseline};
  {
    std::lock_guard<std::mutex> lock(g_tune_mu);
    tune_store_locked(key, choice);
  }
  if (out) *out = cf_tune_result{pick.mode, pick.ctas, pick.tile, timed, best, baseline, 0};
  return CF_OK;
}

// ---- learned initial increment ------------------------------------------

struct cf_mpnn {
  Mpnn m;
};

cf_status cf_mpnn_create(int max_nodes, cf_mpnn** out) {
  if (!out || max_nodes <= 0) return CF_ERR_INVALID_ARG;
  *out = nullptr;
  int count = 0;
  if (cudaGetDeviceCount(&count) != cudaSuccess || count == 0) return CF_ERR_NO_DEVICE;
  cf_mpnn* n = new cf_mpnn();
  cudaError_t e = mpnn_alloc(n->m, max_nodes);
  if (e == cudaSuccess) e = cudaMemset(n->m.w, 0, sizeof(float) * CF_MPNN_PARAMS);
  if (e == cudaSuccess) e = mpnn_refresh_bf16(n->m, nullptr);
  if (e != cudaSuccess) {
    mpnn_free(n->m);
    delete n;
    return from_cuda(e);
  }
  *out = n;
  return CF_OK;
}

cf_status cf_mpnn_destroy(cf_mpnn* net) {
  if (!net) return CF_ERR_INVALID_ARG;
  cudaDeviceSynchronize();
  mpnn_free(net->m);
  delete net;
  return CF_OK;
}

cf_status cf_mpnn_set_weights(cf_mpnn* net, const float* h_params, int n) {
  if (!net || !h_params || n != CF_MPNN_PARAMS) return CF_ERR_INVALID_ARG;
  Mpnn& m = net->m;
  CF_TRY(cudaMemcpy(m.w, h_params, sizeof(float) * n, cudaMemcpyHostToDevice));
  CF_TRY(cudaMemset(m.m, 0, sizeof(float) * n));
  CF_TRY(cudaMemset(m.v, 0, sizeof(float) * n));
  m.step = 0;
  CF_TRY(mpnn_refresh_bf16(m, nullptr));
  CF_TRY(cudaDeviceSynchronize());
  return CF_OK;
}

cf_status cf_mpnn_get_weights(cf_mpnn* net, float* h_params, int n) {
  if (!net || !h_params || n != CF_MPNN_PARAMS) return CF_ERR_INVALID_ARG;
  CF_TRY(cudaMemcpy(h_params, net->m.w, sizeof(float) * n, cudaMemcpyDeviceToHost));
  return CF_OK;
}

cf_status cf_mpnn_set_graph(cf_mpnn* net, const int* d_nbr, int num_nodes, void* stream) {
  if (!net || num_nodes < 0 || (num_nodes > 0 && !d_nbr)) return CF_ERR_INVALID_ARG;
  Mpnn& m = net->m;
  if (num_nodes > m.max_nodes) return CF_ERR_CAPACITY;
  cudaStream_t s = (cudaStream_t)stream;
  const int N = num_nodes;
  std::vector<int> nbr((size_t)N * CF_K_GRAPH);
  if (N) CF_TRY(cudaMemcpyAsync(nbr.data(), d_nbr, sizeof(int) * nbr.size(), cudaMemcpyDeviceToHost, s));
  CF_TRY(cudaStreamSynchronize(s));
  std::vector<float> inv_deg(std::max(1, N), 0.f);
  std::vector<int> rev_ptr(N + 1, 0), rev_idx;
  for (int i = 0; i < N; i++) {
    int deg = 0;
    for (int k = 0; k < CF_K_GRAPH; k++) {
      int& j = nbr[(size_t)i * CF_K_GRAPH + k];
      if (j < 0 || j >= N) j = -1;
      if (j >= 0) {
        deg++;
        rev_ptr[j + 1]++;
      }
    }
    inv_deg[i] = deg ? 1.f / (float)deg : 0.f;
  }
  for (int j = 0; j < N; j++) rev_ptr[j + 1] += rev_ptr[j];
  rev_idx.assign(std::max(1, rev_ptr[N]), 0);
  {
    std::vector<int> fill(rev_ptr.begin(), rev_ptr.end() - 1);
    for (int i = 0; i < N; i++)
      for (int k = 0; k < CF_K_GRAPH; k++) {
        const int j = nbr[(size_t)i * CF_K_GRAPH + k];
        if (j >= 0) rev_idx[fill[j]++] = i;
      }
  }
  if (N) {
    CF_TRY(cudaMemcpy(m.nbr, nbr.data(), sizeof(int) * nbr.size(), cudaMemcpyHostToDevice));
    CF_TRY(cudaMemcpy(m.inv_deg, inv_deg.data(), sizeof(float) * N, cudaMemcpyHostToDevice));
    CF_TRY(cudaMemcpy(m.rev_ptr, rev_ptr.data(), sizeof(int) * (N + 1), cudaMemcpyHostToDevice));
    CF_TRY(cudaMemcpy(m.rev_idx, rev_idx.data(), sizeof(int) * rev_idx.size(), cudaMemcpyHostToDevice));
  }
  m.N = N;
  return CF_OK;
}

cf_status cf_mpnn_forward(cf_mpnn* net, const float* d_features, float* d_out, void* stream) {
  if (!net || !d_features || !d_out) return CF_ERR_INVALID_ARG;
  CF_TRY(mpnn_forward(net->m, d_features, d_out, (cudaStream_t)stream));
  return CF_OK;
}

cf_status cf_mpnn_gradients(cf_mpnn* net, const float* d_features, const float* d_targets, float* h_grad,
                            double* h_loss, void* stream) {
  if (!net || !d_features || !d_targets) return CF_ERR_INVALID_ARG;
  Mpnn& m = net->m;
  cudaStream_t s = (cudaStream_t)stream;
  CF_TRY(mpnn_gradients(m, d_features, d_targets, s));
  if (h_grad) CF_TRY(cudaMemcpyAsync(h_grad, m.g, sizeof(float) * CF_MPNN_PARAMS, cudaMemcpyDeviceToHost, s));
  if (h_loss) CF_TRY(cudaMemcpyAsync(h_loss, m.loss, sizeof(double), cudaMemcpyDeviceToHost, s));
  CF_TRY(cudaStreamSynchronize(s));
  return CF_OK;
}

cf_status cf_mpnn_train_step(cf_mpnn* net, const float* d_features, const float* d_targets, float lr,
                             double* h_loss, void* stream) {
  if (!net || !d_features || !d_targets || !(lr >= 0.f)) return CF_ERR_INVALID_ARG;
  Mpnn& m = net->m;
  cudaStream_t s = (cudaStream_t)stream;
  CF_TRY(mpnn_gradients(m, d_features, d_targets, s));
  CF_TRY(mpnn_adam(m, lr, s));
  if (h_loss) {
    CF_TRY(cudaMemcpyAsync(h_loss, m.loss, sizeof(double), cudaMemcpyDeviceToHost, s));
    CF_TRY(cudaStreamSynchronize(s));
  }
  return CF_OK;
}

cf_status cf_dq_increments(const cf_dual_quat* d_to, const cf_dual_quat* d_from, int n, float* d_out, void* stream) {
  if (n < 0 || (n > 0 && (!d_to || !d_from || !d_out))) return CF_ERR_INVALID_ARG;
  if ((reinterpret_cast<uintptr_t>(d_to) | reinterpret_cast<uintptr_t>(d_from)) & 15u) return CF_ERR_INVALID_ARG;
  CF_TRY(launch_increments(d_to, d_from, n, d_out, (cudaStream_t)stream));
  return CF_OK;
}

namespace {
cf_status check_problem(cf_gn* h, const cf_problem* prob, const void* d_T) {
  if (!h || !prob || prob->num_nodes < 0 || prob->num_corrs < 0) return CF_ERR_INVALID_ARG;
  if (prob->num_nodes > h->max_nodes || prob->num_corrs > h->max_corrs) return CF_ERR_CAPACITY;
  if (prob->num_nodes == 0) return CF_OK;
  if (!prob->nodes || !d_T || (prob->num_corrs > 0 && (!prob->corrs || !prob->canon_points))) return CF_ERR_INVALID_ARG;
  if ((reinterpret_cast<uintptr_t>(prob->corrs) & 3u) || (reinterpret_cast<uintptr_t>(d_T) & 15u))
    return CF_ERR_INVALID_ARG;
  return CF_OK;
}
}  // namespace

cf_status cf_gn_features(cf_gn* h, const cf_problem* prob, const cf_dual_quat* d_transforms,
                         const cf_dual_quat* d_history, float* d_features, void* stream) {
  cf_status st = check_problem(h, prob, d_transforms);
  if (st != CF_OK || prob->num_nodes == 0) return st;
  if (!d_history || !d_features || (reinterpret_cast<uintptr_t>(d_history) & 15u)) return CF_ERR_INVALID_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  const int N = prob->num_nodes, M = prob->num_corrs;
  if ((st = ensure_pattern(h, prob->nodes, N, s)) != CF_OK) return st;
  if ((st = prepare_table(h, {make_desc(prob->corrs, prob->canon_points, prob->nodes,
                                        const_cast<cf_dual_quat*>(d_transforms), M, N, 0.f, 0.f, 1.f)},
                          true, s)) != CF_OK)
    return st;
  Work& w = h->w;
  if ((st = bin_correspondences(h, false, s)) != CF_OK) return st;
  SolveArgs a = make_args(h, prob->nodes, N, M);
  a.transforms = const_cast<cf_dual_quat*>(d_transforms);  // (read only here)
  CF_TRY(launch_final_energy(w, h->p, a, kNoSlot, s, true));
  CF_TRY(launch_features(w, d_transforms, d_history, N, d_features, s));
  return CF_OK;
}

cf_status cf_gn_solve_learned(cf_gn* h, cf_mpnn* net, const cf_problem* prob, cf_dual_quat* d_transforms,
                              const cf_dual_quat* d_history, cf_solve_stats* stats, void* stream) {
  if (!net) return CF_ERR_INVALID_ARG;
  if (stats) memset(stats, 0, sizeof(*stats));
  cf_status st = check_problem(h, prob, d_transforms);
  if (st != CF_OK || prob->num_nodes == 0) return st;
  if (!d_history || (reinterpret_cast<uintptr_t>(d_history) & 15u)) return CF_ERR_INVALID_ARG;
  const int N = prob->num_nodes, M = prob->num_corrs;
  if (N > net->m.max_nodes) return CF_ERR_CAPACITY;
  cudaStream_t s = (cudaStream_t)stream;
  if ((st = ensure_pattern(h, prob->nodes, N, s)) != CF_OK) return st;
  if ((st = prepare_table(h, {make_desc(prob->corrs, prob->canon_points, prob->nodes, d_transforms, M, N,
                                        prob->max_rot, prob->max_trans, prob->update_scale)},
                          true, s)) != CF_OK)
    return st;
  Work& w = h->w;
  if (!w.T_save) CF_TRY(dalloc(&w.T_save, (size_t)w.max_nodes));
  SolveArgs a = make_args(h, prob->nodes, N, M);
  a.transforms = d_transforms;
  a.max_rot = prob->max_rot;
  a.max_trans = prob->max_trans;
  a.update_scale = prob->update_scale;
  h->learn_net = &net->m;
  h->learn_hist = d_history;
  net->m.N = N;
  st = solve_graphed(h, 2, a, s);
  if (st != CF_OK || !stats) return st;
  return read_stats(h, stats, {0}, 1, s);
}

cf_status cf_gn_last_stats(cf_gn* h, cf_solve_stats* stats, int num, void* stream) {
  if (!h || !stats || num < 1) return CF_ERR_INVALID_ARG;
  std::vector<int> slots(num, -1);
  for (int q = 0; q < num && q < h->tb.P; q++) slots[q] = q;
  return read_stats(h, stats, slots, num, (cudaStream_t)stream);
}

cf_status cf_gn_profile_enable(cf_gn* h, int on) {
  if (!h) return CF_ERR_INVALID_ARG;
  if (h->prof_used) prof_collect(h);
  h->profile = on != 0;
  for (int i = 0; i < CF_PROF_SLOTS; i++) {
    h->prof_ms[i] = 0.0;
    h->prof_n[i] = 0;
  }
  return CF_OK;
}

cf_status cf_gn_profile_read(cf_gn* h, double* ms, int* launches, int n_slots) {
  if (!h || n_slots < 0) return CF_ERR_INVALID_ARG;
  prof_collect(h);
  for (int i = 0; i < n_slots && i < CF_PROF_SLOTS; i++) {
    if (ms) ms[i] = h->prof_ms[i];
    if (launches) launches[i] = h->prof_n[i];
  }
  return CF_OK;
}

const char* cf_gn_profile_name(int slot) {
  return (slot >= 0 && slot < CF_PROF_SLOTS) ? kProfNames[slot] : "";
}

cf_status cf_gn_launch_count(const cf_gn* h, long long* launches) {
  if (!h || !launches) return CF_ERR_INVALID_ARG;
  *launches = h->launches;
  return CF_OK;
}

// Debug: clock64 phase cycles of CTA 0 of the grid-wide PCG, accumulated
// over every launch since the call with reset != 0 (which also enables them).
extern "C" CF_API cf_status cf_gn_debug_pcg_timers(cf_gn* h, int reset, long long* out, int n) {
  if (!h) return CF_ERR_INVALID_ARG;
  if (reset) {
    h->phase_timers = 1;
    CF_TRY(cudaMemset(h->w.timers, 0, sizeof(long long) * kTimerSlots));
    return CF_OK;
  }
  CF_TRY(cudaDeviceSynchronize());
  if (out && n > 0)
    CF_TRY(cudaMemcpy(out, h->w.timers, sizeof(long long) * std::min(n, kTimerSlots), cudaMemcpyDeviceToHost));
  return CF_OK;
}

cf_status cf_gn_check(cf_gn* h, void* stream) {
  if (!h) return CF_ERR_INVALID_ARG;
  int herr = 0;
  CF_TRY(cudaMemcpyAsync(&herr, h->w.err, sizeof(int), cudaMemcpyDeviceToHost, (cudaStream_t)stream));
  CF_TRY(cudaStreamSynchronize((cudaStream_t)stream));
  if (herr & kErrTimeoutBit) return CF_ERR_TIMEOUT;
  if (herr & kErrNonFiniteBit) return CF_ERR_NON_FINITE;
  return CF_OK;
}

cf_status cf_gn_get_system(cf_gn* h, int* num_rows, int* num_blocks, int* h_row_ptr, int* h_col_idx,
                           float* h_values, float* h_rhs, void* stream) {
  if (!h) return CF_ERR_INVALID_ARG;
  const int N = h->pattern_valid ? h->p.N : 0;
  const int nnzb = h->pattern_valid ? h->p.nnzb : 0;
  if (num_rows) *num_rows = N;
  if (num_blocks) *num_blocks = nnzb;
  if (N == 0) return CF_OK;
  cudaStream_t s = (cudaStream_t)stream;
  if (h_row_ptr) memcpy(h_row_ptr, h->h_row_ptr.data(), sizeof(int) * (N + 1));
  if (h_col_idx) memcpy(h_col_idx, h->h_col_idx.data(), sizeof(int) * nnzb);
  if (h_values)
    CF_TRY(cudaMemcpyAsync(h_values, h->p.values, sizeof(float) * 36 * (size_t)nnzb, cudaMemcpyDeviceToHost, s));
  if (h_rhs) CF_TRY(cudaMemcpyAsync(h_rhs, h->w.rhs, sizeof(float) * 6 * (size_t)N, cudaMemcpyDeviceToHost, s));
  CF_TRY(cudaStreamSynchronize(s));
  return CF_OK;
}

cf_status cf_energy_noalloc(const cf_problem* problem, const cf_dual_quat* d_transforms, float lambda_smooth,
                            double* d_energy, void* stream) {
  if (!problem || !d_energy || problem->num_nodes < 0 || problem->num_corrs < 0) return CF_ERR_INVALID_ARG;
  if (problem->num_nodes > CF_NOALLOC_MAX_NODES) return CF_ERR_CAPACITY;
  if (problem->num_nodes > 0 && (!problem->nodes || !d_transforms)) return CF_ERR_INVALID_ARG;
  if (problem->num_corrs > 0 && (!problem->corrs || !problem->canon_points)) return CF_ERR_INVALID_ARG;
  if (reinterpret_cast<uintptr_t>(d_transforms) & 15u) return CF_ERR_INVALID_ARG;
  CF_TRY(launch_energy_noalloc(problem, d_transforms, lambda_smooth, d_energy, (cudaStream_t)stream));
  return CF_OK;
}

cf_status cf_warp_apply_twist(cf_dual_quat* d_transforms, const float* d_delta_x, int num_nodes, float max_rot,
                              float max_trans, float update_scale, void* stream) {
  if (num_nodes < 0) return CF_ERR_INVALID_ARG;
  if (num_nodes == 0) return CF_OK;
  if (!d_transforms || !d_delta_x || (reinterpret_cast<uintptr_t>(d_transforms) & 15u)) return CF_ERR_INVALID_ARG;
  CF_TRY(launch_apply_twist(d_transforms, d_delta_x, num_nodes, max_rot, max_trans, update_scale,
                            (cudaStream_t)stream));
  return CF_OK;
}

cf_status cf_warp_skin_points(const float* d_points, const int* d_node_ids, const float* d_node_ws, int num_points,
                              const cf_deform_node* d_nodes, const cf_dual_quat* d_transforms, int num_nodes,
                              float* d_out, void* stream) {
  if (num_points < 0 || num_nodes < 0) return CF_ERR_INVALID_ARG;
  if (num_points == 0) return CF_OK;
  if (!d_points || !d_node_ids || !d_node_ws || !d_out || (num_nodes > 0 && (!d_nodes || !d_transforms)))
    return CF_ERR_INVALID_ARG;
  CF_TRY(launch_skin_points(d_points, d_node_ids, d_node_ws, num_points, d_nodes, d_transforms, num_nodes, d_out,
                            (cudaStream_t)stream));
  return CF_OK;
}

struct cf_corr_search {
  int max_w = 0, max_h = 0;
  cf::CorrScratch sc = {};
  int chunks = 0;  // row chunks per tile; 0 = chosen per frame
  long long launches = 0;
  // cf_line_search: its best trial's outputs and the chain of best RMSEs
  // (allocated by the first line search, grown with the frame)
  unsigned char* keep = nullptr;
  size_t keep_bytes = 0;
};

namespace {
void corr_free(cf_corr_search* h) {
  cudaFree(h->keep);
  cudaFree(h->sc.A);
  cudaFree(h->sc.B);
  cudaFree(h->sc.part_a);
  cudaFree(h->sc.part_g);
  cudaFree(h->sc.rows);
  cudaFree(h->sc.todo);
  cudaFree(h->sc.box);
  cudaFree(h->sc.pix_v);
  cudaFree(h->sc.pix_n);
  cudaFree(h->sc.pix_row);
  cudaFree(h->sc.flag);
}
}  // namespace

cf_status cf_corr_search_create(int max_width, int max_height, cf_corr_search** out) {
  if (!out) return CF_ERR_INVALID_ARG;
  *out = nullptr;
  if (max_width <= 0 || max_height <= 0) return CF_ERR_INVALID_ARG;
  // per-pixel node lists are indexed with 32-bit pixel offsets times 4
  if ((long long)max_width * max_height > (1LL << 29)) return CF_ERR_CAPACITY;
  cf_corr_search* h = new cf_corr_search();
  h->max_w = max_width;
  h->max_h = max_height;
  const size_t P = (size_t)max_width * max_height;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&h->sc.sms, cudaDevAttrMultiProcessorCount, dev);
  if (e == cudaSuccess) e = dalloc(&h->sc.A, P);
  if (e == cudaSuccess) e = dalloc(&h->sc.B, P);
  h->sc.chunk_cap = corr_chunk_cap(P);
  if (e == cudaSuccess) e = dalloc(&h->sc.part_a, P * h->sc.chunk_cap);
  if (e == cudaSuccess) e = dalloc(&h->sc.part_g, P * h->sc.chunk_cap);
  if (e == cudaSuccess) e = dalloc(&h->sc.rows, corr_box_cap(P));
  if (e == cudaSuccess) e = dalloc(&h->sc.todo, 1 + corr_box_cap(P) * kCorrMaxChunks);
  if (e == cudaSuccess) e = cudaMalloc(&h->sc.box, corr_box_cap(P) * corr_box_bytes());
  if (e == cudaSuccess) e = dalloc(&h->sc.pix_v, P);
  if (e == cudaSuccess) e = dalloc(&h->sc.pix_n, P);
  if (e == cudaSuccess) e = dalloc(&h->sc.pix_row, P);
  if (e == cudaSuccess) e = dalloc(&h->sc.flag, 1);
  if (e != cudaSuccess) {
    corr_free(h);
    delete h;
    return from_cuda(e);
  }
  *out = h;
  return CF_OK;
}

cf_status cf_corr_search_destroy(cf_corr_search* h) {
  if (!h) return CF_OK;
  corr_free(h);
  delete h;
  return CF_OK;
}

cf_status cf_corr_search_set_chunks(cf_corr_search* h, int chunks) {
  if (!h || chunks < 0 || chunks > kCorrMaxChunks) return CF_ERR_INVALID_ARG;
  h->chunks = chunks;
  return CF_OK;
}

cf_status cf_find_correspondences(cf_corr_search* h, const cf_corr_frame* frame, const cf_camera* cam,
                                  const cf_mat4* T_cam_world, const cf_mat4* T_world_cam, const cf_corr_params* params,
                                  cf_correspondence* d_corrs, int* d_num_valid, int* d_stats, void* stream) {
  if (!h || !frame || !cam || !T_cam_world || !T_world_cam || !params || !d_num_valid) return CF_ERR_INVALID_ARG;
  if (cam->width < 0 || cam->height < 0) return CF_ERR_INVALID_ARG;
  if (cam->width > h->max_w || cam->height > h->max_h) return CF_ERR_CAPACITY;
  if ((long long)cam->width * cam->height > 0) {
    if (!frame->d_live_vertices || !frame->d_live_normals || !frame->d_depth || !frame->d_depth_normals || !d_corrs)
      return CF_ERR_INVALID_ARG;
    if (frame->d_pixel_knn) {
      if (!frame->d_pixel_knn_w) return CF_ERR_INVALID_ARG;
    } else {
      if (!frame->d_hit_voxel_idx || frame->num_voxels < 0) return CF_ERR_INVALID_ARG;
      if (frame->num_voxels > 0 && (!frame->d_voxel_knn || !frame->d_voxel_knn_w)) return CF_ERR_INVALID_ARG;
      if ((frame->d_pixel_knn_out == nullptr) != (frame->d_pixel_knn_w_out == nullptr)) return CF_ERR_INVALID_ARG;
    }
  }
  CF_TRY(launch_corr_search(frame, cam, T_cam_world, T_world_cam, params, h->sc, h->chunks, d_corrs, d_num_valid,
                            d_stats, (cudaStream_t)stream, &h->launches));
  return CF_OK;
}

cf_status cf_compute_pixel_knn(const int* d_hit_voxel_idx, int width, int height, const int* d_voxel_knn,
                               const float* d_voxel_knn_w, long long num_voxels, int* d_pixel_knn,
                               float* d_pixel_knn_w, void* stream) {
  if (width < 0 || height < 0 || num_voxels < 0) return CF_ERR_INVALID_ARG;
  if ((long long)width * height > (1LL << 29)) return CF_ERR_CAPACITY;
  const int P = width * height;
  if (P == 0) return CF_OK;
  if (!d_hit_voxel_idx || !d_pixel_knn || !d_pixel_knn_w) return CF_ERR_INVALID_ARG;
  if (num_voxels > 0 && (!d_voxel_knn || !d_voxel_knn_w)) return CF_ERR_INVALID_ARG;
  CF_TRY(launch_pixel_knn(d_hit_voxel_idx, P, d_voxel_knn, d_voxel_knn_w, num_voxels, d_pixel_knn, d_pixel_knn_w,
                          (cudaStream_t)stream));
  return CF_OK;
}

cf_status cf_corr_search_launch_count(const cf_corr_search* h, long long* launches) {
  if (!h || !launches) return CF_ERR_INVALID_ARG;
  *launches = h->launches;
  return CF_OK;
}

cf_status cf_skin_mesh_vertices(const float* d_canonical, float* d_warped, int num_vertices, const cf_voxel_grid* grid,
                                const cf_deform_node* d_nodes, const cf_dual_quat* d_transforms, int num_nodes,
                                const int* d_voxel_knn, const float* d_voxel_knn_w, void* stream) {
  if (num_vertices < 0 || num_nodes < 0 || !grid) return CF_ERR_INVALID_ARG;
  if (num_vertices == 0) return CF_OK;
  if (!d_canonical || !d_warped) return CF_ERR_INVALID_ARG;
  if (!(grid->voxel_size > 0.f) || grid->dims[0] < 0 || grid->dims[1] < 0 || grid->dims[2] < 0)
    return CF_ERR_INVALID_ARG;
  if ((long long)grid->dims[0] * grid->dims[1] * grid->dims[2] > (1LL << 31) / CF_K_NEIGHBORS) return CF_ERR_CAPACITY;
  CF_TRY(launch_mesh_skin(d_canonical, d_warped, num_vertices, grid, d_nodes, d_transforms, num_nodes, d_voxel_knn,
                          d_voxel_knn_w, (cudaStream_t)stream));
  return CF_OK;
}

struct cf_raster {
  int max_w = 0, max_h = 0;
  unsigned long long* ztri = nullptr;  // per pixel: depth bits << 32 | triangle, all ones = empty
  float4* cache = nullptr;             // per triangle: projection, area, normal, corners (112 B)
  int* big = nullptr;                  // (triangle, first row item) of the boxes over 128 pixels
  unsigned long long* big_ctr = nullptr;  // their number << 32 | row items (reset by the resolve)
  int cache_cap = 0;                   // triangles the cache and the list hold
  cf_dual_quat* plain = nullptr;       // per node: the plain DQ the skinning blends
  int plain_cap = 0;
  bool dirty = false;                  // a call failed after the buffer may have been written
  long long launches = 0;
  // the launch sequence of a call, captured once and replayed while the
  // call's arguments (and these buffers) are unchanged
  cudaGraphExec_t graph_exec = nullptr;
  std::vector<unsigned char> graph_key;
  bool graph_failed = false;
  long long graph_launches = 0;
};

cf_status cf_raster_create(int max_width, int max_height, cf_raster** out) {
  if (!out) return CF_ERR_INVALID_ARG;
  *out = nullptr;
  if (max_width <= 0 || max_height <= 0) return CF_ERR_INVALID_ARG;
  if ((long long)max_width * max_height > (1LL << 30)) return CF_ERR_CAPACITY;
  cf_raster* h = new cf_raster();
  h->max_w = max_width;
  h->max_h = max_height;
  const size_t P = (size_t)max_width * max_height;
  cudaError_t e = dalloc(&h->ztri, P);
  if (e == cudaSuccess) e = cudaMemset(h->ztri, 0xff, P * sizeof(unsigned long long));
  if (e == cudaSuccess) e = dalloc(&h->big_ctr, 1);
  if (e == cudaSuccess) e = cudaMemset(h->big_ctr, 0, sizeof(unsigned long long));
  if (e != cudaSuccess) {
    cudaFree(h->ztri);
    cudaFree(h->big_ctr);
    delete h;
    return from_cuda(e);
  }
  *out = h;
  return CF_OK;
}

cf_status cf_raster_destroy(cf_raster* h) {
  if (!h) return CF_OK;
  if (h->graph_exec) cudaGraphExecDestroy(h->graph_exec);
  cudaFree(h->ztri);
  cudaFree(h->cache);
  cudaFree(h->big);
  cudaFree(h->big_ctr);
  cudaFree(h->plain);
  delete h;
  return CF_OK;
}

namespace {

// The arguments of one prediction (skin = false: the rasterisation alone).
struct RasterCall {
  bool skin;
  const float* canon;
  float* warped;
  const int* tris;
  int V, NT;
  const cf_deform_node* nodes;
  const cf_dual_quat* T;
  int N;
  const int* vk;
  const float* vw;
  cf_camera cam;
  cf_mat4 Tcw;
  cf_voxel_grid grid;
  float *lv, *ln;
  int* hit;
};

// Checks the call and readies the handle's buffers (their growth allocates
// and synchronises; a failed earlier call's buffers are reset on the stream).
cf_status raster_prepare(cf_raster* h, const RasterCall& c, cudaStream_t s) {
  if (c.cam.width < 0 || c.cam.height < 0) return CF_ERR_INVALID_ARG;
  if (c.cam.width > h->max_w || c.cam.height > h->max_h) return CF_ERR_CAPACITY;
  if ((long long)c.cam.width * c.cam.height == 0) return CF_OK;
  if (!c.lv || !c.ln || !c.hit) return CF_ERR_INVALID_ARG;
  if (c.NT > 0 && (!c.canon || !c.warped || !c.tris)) return CF_ERR_INVALID_ARG;
  if (!(c.grid.voxel_size > 0.f) || c.grid.dims[0] < 0 || c.grid.dims[1] < 0 || c.grid.dims[2] < 0)
    return CF_ERR_INVALID_ARG;
  if (c.NT > h->cache_cap) {  // grows with the mesh (synchronous allocation)
    CF_TRY(cudaStreamSynchronize(s));
    cudaFree(h->cache);
    cudaFree(h->big);
    h->cache = nullptr;
    h->big = nullptr;
    h->cache_cap = 0;
    CF_TRY(dalloc(&h->cache, (size_t)c.NT * 7));
    CF_TRY(dalloc(&h->big, 2 * (size_t)c.NT));
    h->cache_cap = c.NT;
  }
  if (c.skin && c.N > h->plain_cap) {  // grows with the graph (synchronous allocation)
    CF_TRY(cudaStreamSynchronize(s));
    cudaFree(h->plain);
    h->plain = nullptr;
    h->plain_cap = 0;
    CF_TRY(dalloc(&h->plain, (size_t)c.N));
    h->plain_cap = c.N;
  }
  if (h->dirty) {
    CF_TRY(cudaMemsetAsync(h->ztri, 0xff, (size_t)h->max_w * h->max_h * sizeof(unsigned long long), s));
    CF_TRY(cudaMemsetAsync(h->big_ctr, 0, sizeof(unsigned long long), s));
    h->dirty = false;
  }
  return CF_OK;
}

// The call's skinning launches (when it skins).
cudaError_t raster_skin(cf_raster* h, const RasterCall& c, cudaStream_t s) {
  if (c.skin && c.V > 0) {
    // the nodes' plain DQs once, then the vertices (lists read 16 B at a
    // time when aligned); without nodes the vertices are copied
    const bool plain = c.N > 0 && c.nodes && c.T && c.vk && c.vw &&
                       ((reinterpret_cast<uintptr_t>(c.vk) | reinterpret_cast<uintptr_t>(c.vw)) & 15u) == 0;
    cudaError_t e;
    if (plain) {
      e = launch_tsdf_plain(c.nodes, c.T, h->plain, c.N, s);
      if (e == cudaSuccess) e = launch_mesh_skin_plain(c.canon, c.warped, c.V, &c.grid, h->plain, c.N, c.vk, c.vw, s);
      h->launches += 2;
    } else {
      e = launch_mesh_skin(c.canon, c.warped, c.V, &c.grid, c.nodes, c.T, c.N, c.vk, c.vw, s);
      h->launches += 1;
    }
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

// The call's launches (skinning, rasterisation, big boxes, resolve).
cudaError_t raster_enqueue(cf_raster* h, const RasterCall& c, cudaStream_t s) {
  const cudaError_t e = raster_skin(h, c, s);
  if (e != cudaSuccess) return e;
  return launch_raster(c.canon, c.warped, c.tris, c.V, c.NT, &c.cam, &c.Tcw, &c.grid, h->ztri, h->cache, h->big,
                       h->big_ctr, c.lv, c.ln, c.hit, s, &h->launches);
}

// On a stream of the caller's (not the legacy stream, not capturing), the
// launches run as a CUDA graph captured on the first call and replayed while
// the arguments and the handle's buffers are unchanged (the line search
// predicts ten times with the same ones); otherwise they are launched
// directly.
cf_status raster_run(cf_raster* h, const RasterCall& c, cudaStream_t s) {
  cf_status st = raster_prepare(h, c, s);
  if (st != CF_OK || (long long)c.cam.width * c.cam.height == 0) return st;
  auto direct = [&]() -> cf_status {
    const cudaError_t e = raster_enqueue(h, c, s);
    if (e != cudaSuccess) {
      h->dirty = true;
      return from_cuda(e);
    }
    return CF_OK;
  };
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  if (s == nullptr || cudaStreamIsCapturing(s, &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone) {
    cudaGetLastError();
    return direct();
  }
  std::vector<unsigned char> key(sizeof(RasterCall) + 4 * sizeof(void*));
  const void* bufs[4] = {h->cache, h->big, h->ztri, h->plain};
  memcpy(key.data(), &c, sizeof(RasterCall));
  memcpy(key.data() + sizeof(RasterCall), bufs, sizeof(bufs));
  if (key == h->graph_key) {
    if (h->graph_failed) return direct();
    h->launches += h->graph_launches;
    CF_TRY(cudaGraphLaunch(h->graph_exec, s));
    return CF_OK;
  }
  if (h->graph_exec) {
    cudaGraphExecDestroy(h->graph_exec);
    h->graph_exec = nullptr;
  }
  h->graph_key = key;
  h->graph_failed = false;
  const long long before = h->launches;
  cudaGraph_t g = nullptr;
  cudaError_t e = cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal);
  if (e == cudaSuccess) {
    e = raster_enqueue(h, c, s);
    const cudaError_t e2 = cudaStreamEndCapture(s, &g);
    if (e == cudaSuccess) e = e2;
    if (e == cudaSuccess) e = cudaGraphInstantiate(&h->graph_exec, g, 0);
  }
  if (g) cudaGraphDestroy(g);
  h->graph_launches = h->launches - before;
  h->launches = before;
  if (e != cudaSuccess) {  // not capturable here: remember, and launch directly
    cudaGetLastError();
    if (h->graph_exec) cudaGraphExecDestroy(h->graph_exec);
    h->graph_exec = nullptr;
    h->graph_failed = true;
    return direct();
  }
  h->launches += h->graph_launches;
  CF_TRY(cudaGraphLaunch(h->graph_exec, s));
  return CF_OK;
}

}  // namespace

cf_status cf_rasterize_live_surface(cf_raster* h, const float* d_canonical, const float* d_warped,
                                    const int* d_triangles, int num_vertices, int num_triangles, const cf_camera* cam,
                                    const cf_mat4* T_cam_world, const cf_voxel_grid* grid, float* d_live_vertices,
                                    float* d_live_normals, int* d_hit_voxel_idx, void* stream) {
  if (!h || !cam || !T_cam_world || !grid || num_vertices < 0 || num_triangles < 0) return CF_ERR_INVALID_ARG;
  RasterCall c{};
  c.skin = false;
  c.canon = d_canonical;
  c.warped = const_cast<float*>(d_warped);
  c.tris = d_triangles;
  c.V = num_vertices;
  c.NT = num_triangles;
  c.cam = *cam;
  c.Tcw = *T_cam_world;
  c.grid = *grid;
  c.lv = d_live_vertices;
  c.ln = d_live_normals;
  c.hit = d_hit_voxel_idx;
  return raster_run(h, c, (cudaStream_t)stream);
}

cf_status cf_predict_live_surface(cf_raster* h, const float* d_canonical, float* d_warped, const int* d_triangles,
                                  int num_vertices, int num_triangles, const cf_deform_node* d_nodes,
                                  const cf_dual_quat* d_transforms, int num_nodes, const int* d_voxel_knn,
                                  const float* d_voxel_knn_w, const cf_camera* cam, const cf_mat4* T_cam_world,
                                  const cf_voxel_grid* grid, float* d_live_vertices, float* d_live_normals,
                                  int* d_hit_voxel_idx, void* stream) {
  if (!h || !cam || !T_cam_world || !grid || num_vertices < 0 || num_triangles < 0 || num_nodes < 0)
    return CF_ERR_INVALID_ARG;
  // the checks of cf_skin_mesh_vertices
  if (num_vertices > 0) {
    if (!d_canonical || !d_warped) return CF_ERR_INVALID_ARG;
    if (!(grid->voxel_size > 0.f) || grid->dims[0] < 0 || grid->dims[1] < 0 || grid->dims[2] < 0)
      return CF_ERR_INVALID_ARG;
    if ((long long)grid->dims[0] * grid->dims[1] * grid->dims[2] > (1LL << 31) / CF_K_NEIGHBORS)
      return CF_ERR_CAPACITY;
  }
  RasterCall c{};
  c.skin = true;
  c.canon = d_canonical;
  c.warped = d_warped;
  c.tris = d_triangles;
  c.V = num_vertices;
  c.NT = num_triangles;
  c.nodes = d_nodes;
  c.T = d_transforms;
  c.N = num_nodes;
  c.vk = d_voxel_knn;
  c.vw = d_voxel_knn_w;
  c.cam = *cam;
  c.Tcw = *T_cam_world;
  c.grid = *grid;
  c.lv = d_live_vertices;
  c.ln = d_live_normals;
  c.hit = d_hit_voxel_idx;
  const cudaStream_t s = (cudaStream_t)stream;
  // with an empty image the skinning alone runs (the rasterisation has nothing to draw)
  if ((long long)cam->width * cam->height == 0) {
    if (cam->width < 0 || cam->height < 0) return CF_ERR_INVALID_ARG;
    if (num_vertices > 0) {
      CF_TRY(launch_mesh_skin(d_canonical, d_warped, num_vertices, grid, d_nodes, d_transforms, num_nodes,
                              d_voxel_knn, d_voxel_knn_w, s));
      h->launches += 1;
    }
    return CF_OK;
  }
  return raster_run(h, c, s);
}

cf_status cf_raster_launch_count(const cf_raster* h, long long* launches) {
  if (!h || !launches) return CF_ERR_INVALID_ARG;
  *launches = h->launches;
  return CF_OK;
}

// ---- update validation and line search -------------------------------------

namespace {
// device scratch of cf_validate_update: sums (4 doubles), maxima (4 floats as
// bits), the finite flag; one set per process, calls serialised by g_ls_mu
__device__ double g_ls_sums[4];
__device__ unsigned g_ls_max[4];
__device__ int g_ls_finite;
std::mutex g_ls_mu;
}  // namespace

cf_status cf_validate_update(const float* d_delta_x, int num_nodes, const cf_line_search_params* params,
                             cf_update_stats* stats, void* stream) {
  if (!params || !stats || num_nodes < 0 || (num_nodes > 0 && !d_delta_x)) return CF_ERR_INVALID_ARG;
  std::lock_guard<std::mutex> lock(g_ls_mu);
  cudaStream_t s = (cudaStream_t)stream;
  void *sums = nullptr, *maxima = nullptr, *finite = nullptr;
  CF_TRY(cudaGetSymbolAddress(&sums, g_ls_sums));
  CF_TRY(cudaGetSymbolAddress(&maxima, g_ls_max));
  CF_TRY(cudaGetSymbolAddress(&finite, g_ls_finite));
  const int one = 1;
  CF_TRY(cudaMemsetAsync(sums, 0, 4 * sizeof(double), s));
  CF_TRY(cudaMemsetAsync(maxima, 0, 4 * sizeof(unsigned), s));
  CF_TRY(cudaMemcpyAsync(finite, &one, sizeof(int), cudaMemcpyHostToDevice, s));
  CF_TRY(launch_update_stats(d_delta_x, num_nodes, params->update_scale, params->max_update_rot,
                             params->max_update_trans, (double*)sums, (unsigned*)maxima, (int*)finite, s));
  double hs[4];
  unsigned hm[4];
  int hf = 1;
  CF_TRY(cudaMemcpyAsync(hs, sums, sizeof(hs), cudaMemcpyDeviceToHost, s));
  CF_TRY(cudaMemcpyAsync(hm, maxima, sizeof(hm), cudaMemcpyDeviceToHost, s));
  CF_TRY(cudaMemcpyAsync(&hf, finite, sizeof(int), cudaMemcpyDeviceToHost, s));
  CF_TRY(cudaStreamSynchronize(s));
  cf_update_stats& st = *stats;
  st.rot_sum = hs[0];
  st.trans_sum = hs[1];
  st.eff_rot_sum = hs[2];
  st.eff_trans_sum = hs[3];
  float mx[4];
  memcpy(mx, hm, sizeof(mx));
  st.rot_max = mx[0];
  st.trans_max = mx[1];
  st.eff_rot_max = mx[2];
  st.eff_trans_max = mx[3];
  st.finite = hf;
  st.num_nodes = num_nodes;
  st.pad_ = 0;
  // the acceptance of fusion_app.h:460-489
  const float n1 = (float)(num_nodes > 1 ? num_nodes : 1);
  const float eff_rot_mean = (float)st.eff_rot_sum / n1, eff_trans_mean = (float)st.eff_trans_sum / n1;
  const float ur = params->update_scale;
  const float reject_rot = params->max_update_rot > 0.f ? 5.0f * params->max_update_rot : INFINITY;
  const float reject_trans = params->max_update_trans > 0.f ? 5.0f * params->max_update_trans : INFINITY;
  const bool bad_spike = (ur * st.rot_max > reject_rot) || (ur * st.trans_max > reject_trans);
  const bool mean_ok = (params->max_dx_mean <= 0.f) ||
                       (eff_rot_mean <= params->max_dx_mean && eff_trans_mean <= params->max_dx_mean);
  st.iter_ok = hf && std::isfinite(eff_rot_mean) && std::isfinite(eff_trans_mean) && std::isfinite(st.eff_rot_max) &&
               std::isfinite(st.eff_trans_max) && st.eff_rot_max < reject_rot && st.eff_trans_max < reject_trans &&
               mean_ok && !bad_spike;
  return CF_OK;
}

cf_status cf_scale_delta(const float* d_delta_x, int num_nodes, float max_rot, float max_trans, float scale,
                         float* d_out, void* stream) {
  if (num_nodes < 0) return CF_ERR_INVALID_ARG;
  if (num_nodes == 0) return CF_OK;
  if (!d_delta_x || !d_out) return CF_ERR_INVALID_ARG;
  CF_TRY(launch_scale_delta(d_delta_x, num_nodes, max_rot, max_trans, scale, d_out, (cudaStream_t)stream));
  return CF_OK;
}

cf_status cf_correspondence_rmse(const cf_correspondence* d_corrs, int num_corrs, double* d_partials, double* d_out,
                                 void* stream) {
  if (num_corrs < 0 || !d_partials || !d_out || (num_corrs > 0 && !d_corrs)) return CF_ERR_INVALID_ARG;
  CF_TRY(launch_corr_rmse(d_corrs, num_corrs, d_partials, d_out, (cudaStream_t)stream));
  return CF_OK;
}

cf_status cf_line_search(cf_raster* raster, cf_corr_search* search, const float* d_mesh_canonical,
                         float* d_mesh_warped, const int* d_mesh_triangles, int num_vertices, int num_triangles,
                         const cf_voxel_grid* grid, const cf_deform_node* d_nodes, cf_dual_quat* d_transforms,
                         int num_nodes, const int* d_voxel_knn, const float* d_voxel_knn_w, const float* d_delta_x,
                         const cf_line_search_params* params, cf_corr_frame* frame, const cf_camera* cam,
                         const cf_mat4* T_cam_world, const cf_mat4* T_world_cam, const cf_corr_params* corr_params,
                         cf_correspondence* d_corrs, int* d_num_valid, double base_rmse, int base_valid,
                         cf_dual_quat* d_scratch_transforms, float* d_scratch_delta, double* d_scratch_rmse,
                         float* best_scale, double* best_rmse, double* trial_rmse, int* trial_valid, void* stream) {
  if (!raster || !search || !params || !frame || !cam || !T_cam_world || !T_world_cam || !corr_params ||
      !best_scale || !best_rmse || num_nodes < 0)
    return CF_ERR_INVALID_ARG;
  *best_scale = 0.f;
  *best_rmse = base_rmse;
  for (int t = 0; t < CF_LINE_SEARCH_TRIALS; ++t) {
    if (trial_rmse) trial_rmse[t] = NAN;
    if (trial_valid) trial_valid[t] = -1;
  }
  // fusion_app.h:496-497: no line search without a step or a finite base
  if (!(params->update_scale > 0.f) || !std::isfinite(base_rmse)) return CF_OK;
  if (!d_transforms || !d_delta_x || !d_scratch_transforms || !d_scratch_delta || !d_scratch_rmse || !d_corrs ||
      !d_num_valid || frame->d_pixel_knn || !frame->d_hit_voxel_idx || !frame->d_live_vertices ||
      !frame->d_live_normals)
    return CF_ERR_INVALID_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  const float u = params->update_scale;
  const float scales[CF_LINE_SEARCH_TRIALS] = {u,          0.5f * u,    0.25f * u,  0.125f * u, 0.0625f * u,
                                               -0.0625f * u, -0.125f * u, -0.25f * u, -0.5f * u,  -u};
  const size_t tbytes = (size_t)num_nodes * sizeof(cf_dual_quat);
  const int P = cam->width * cam->height;
  float* lv = const_cast<float*>(frame->d_live_vertices);
  float* ln = const_cast<float*>(frame->d_live_normals);
  int* hit = const_cast<int*>(frame->d_hit_voxel_idx);
  double* partials = d_scratch_rmse;
  double* slots = d_scratch_rmse + 2 * CF_RMSE_BLOCKS;
  cf_status st = CF_OK;
  // the saved transforms with the increment at a scale
  auto transforms = [&](float scale) -> cf_status {
    if (num_nodes > 0 && (reinterpret_cast<uintptr_t>(d_transforms) & 15u)) return CF_ERR_INVALID_ARG;
    return from_cuda(launch_trial_transforms(d_scratch_transforms, d_delta_x, num_nodes, params->max_update_rot,
                                             params->max_update_trans, scale, d_scratch_delta, d_transforms, s));
  };
  // one trial, or the final application: transforms, predict, search
  auto apply = [&](float scale) -> cf_status {
    cf_status r = transforms(scale);
    if (r == CF_OK) r = cf_predict_live_surface(raster, d_mesh_canonical, d_mesh_warped, d_mesh_triangles,
                                                num_vertices, num_triangles, d_nodes, d_transforms, num_nodes,
                                                d_voxel_knn, d_voxel_knn_w, cam, T_cam_world, grid, lv, ln, hit,
                                                stream);
    if (r == CF_OK) r = cf_find_correspondences(search, frame, cam, T_cam_world, T_world_cam, corr_params, d_corrs,
                                                d_num_valid, nullptr, stream);
    return r;
  };
  // The best trial's outputs are kept on the search handle while the trials
  // run (ls_keep_kernel applies the acceptance rule after each RMSE), so the
  // accepted trial is not predicted and searched again: its records, maps and
  // valid count are copied back, its transforms recomputed and the mesh
  // re-skinned, which gives the bits of a repeated trial.
  const size_t Pz = (size_t)P;
  const bool pk_out = frame->d_pixel_knn_out && frame->d_pixel_knn_w_out;
  auto al = [](size_t v) { return (v + 255) & ~(size_t)255; };
  const size_t off_kept = al(sizeof(double) * (CF_LINE_SEARCH_TRIALS + 1));
  const size_t off_nv = off_kept + 256, off_corr = off_nv + 256;
  const size_t off_lv = al(off_corr + Pz * sizeof(cf_correspondence));
  const size_t off_ln = al(off_lv + Pz * 12), off_hit = al(off_ln + Pz * 12);
  const size_t off_pk = al(off_hit + Pz * 4), off_pw = al(off_pk + (pk_out ? Pz * 16 : 0));
  const size_t keep_need = off_pw + (pk_out ? Pz * 16 : 0);
  if (search->keep_bytes < keep_need) {  // grows with the frame (synchronous allocation)
    CF_TRY(cudaStreamSynchronize(s));
    cudaFree(search->keep);
    search->keep = nullptr;
    search->keep_bytes = 0;
    CF_TRY(dalloc(&search->keep, keep_need));
    search->keep_bytes = keep_need;
  }
  unsigned char* kb = search->keep;
  double* best_chain = reinterpret_cast<double*>(kb);
  int* kept = reinterpret_cast<int*>(kb + off_kept);
  CF_TRY(cudaMemsetAsync(kept, 0xff, sizeof(int), s));
  const int need = (int)(0.75f * (float)base_valid);
  LsKeepArgs ka{};
  ka.best0 = base_rmse;
  ka.kept = kept;
  ka.min_valid = params->min_valid_corrs;
  ka.need = need;
  struct KeepBuf {
    int* live;
    size_t off, words;
  };
  std::vector<KeepBuf> bufs = {{d_num_valid, off_nv, 1},
                               {reinterpret_cast<int*>(d_corrs), off_corr, Pz * (sizeof(cf_correspondence) / 4)},
                               {reinterpret_cast<int*>(lv), off_lv, Pz * 3},
                               {reinterpret_cast<int*>(ln), off_ln, Pz * 3},
                               {hit, off_hit, Pz}};
  if (pk_out) {
    bufs.push_back({frame->d_pixel_knn_out, off_pk, Pz * 4});
    bufs.push_back({reinterpret_cast<int*>(frame->d_pixel_knn_w_out), off_pw, Pz * 4});
  }
  ka.nbuf = (int)bufs.size();
  for (int i = 0; i < ka.nbuf; ++i) {
    ka.src[i] = bufs[i].live;
    ka.dst[i] = reinterpret_cast<int*>(kb + bufs[i].off);
    ka.words[i] = bufs[i].words;
  }
  CF_TRY(cudaMemcpyAsync(d_scratch_transforms, d_transforms, tbytes, cudaMemcpyDeviceToDevice, s));  // save
  for (int t = 0; t < CF_LINE_SEARCH_TRIALS && st == CF_OK; ++t) {
    st = apply(scales[t]);
    if (st == CF_OK) st = from_cuda(launch_corr_rmse(d_corrs, P, partials, nullptr, s));
    if (st == CF_OK) {
      ka.part = partials;
      ka.valid = d_num_valid;
      ka.slot = slots + 3 * t;
      ka.best_in = t > 0 ? best_chain + t : nullptr;
      ka.best_out = best_chain + t + 1;
      ka.trial = t;
      st = from_cuda(launch_ls_keep(ka, s));
    }
  }
  if (st != CF_OK) {
    cudaMemcpyAsync(d_transforms, d_scratch_transforms, tbytes, cudaMemcpyDeviceToDevice, s);
    return st;
  }
  double h[3 * CF_LINE_SEARCH_TRIALS];
  int h_kept = -1;
  CF_TRY(cudaMemcpyAsync(h, slots, sizeof(h), cudaMemcpyDeviceToHost, s));
  CF_TRY(cudaMemcpyAsync(&h_kept, kept, sizeof(int), cudaMemcpyDeviceToHost, s));
  CF_TRY(cudaStreamSynchronize(s));
  // the acceptance of each trial (fusion_app.h:575-582)
  int best_t = -1;
  for (int t = 0; t < CF_LINE_SEARCH_TRIALS; ++t) {
    const double sum = h[3 * t], wsum = h[3 * t + 1];
    const int valid = (int)h[3 * t + 2];
    const double rmse = wsum > 0.0 ? std::sqrt(sum / wsum) : INFINITY;
    if (trial_rmse) trial_rmse[t] = rmse;
    if (trial_valid) trial_valid[t] = valid;
    if (valid >= params->min_valid_corrs && valid >= need && std::isfinite(rmse) && rmse < *best_rmse) {
      *best_rmse = rmse;
      *best_scale = scales[t];
      best_t = t;
    }
  }
  if (*best_scale == 0.f) {  // fusion_app.h:586-592: restore and stop; the maps stay the last trial's
    CF_TRY(cudaMemcpyAsync(d_transforms, d_scratch_transforms, tbytes, cudaMemcpyDeviceToDevice, s));
  } else if (h_kept == best_t) {
    // the accepted trial's transforms (as apply computes them), its skinned
    // mesh (the prediction's skinning launches), its records and maps
    if ((st = transforms(*best_scale)) != CF_OK) return st;
    RasterCall c{};
    c.skin = true;
    c.canon = d_mesh_canonical;
    c.warped = d_mesh_warped;
    c.V = num_vertices;
    c.nodes = d_nodes;
    c.T = d_transforms;
    c.N = num_nodes;
    c.vk = d_voxel_knn;
    c.vw = d_voxel_knn_w;
    c.grid = *grid;
    CF_TRY(raster_skin(raster, c, s));
    for (const KeepBuf& kbuf : bufs)
      CF_TRY(cudaMemcpyAsync(kbuf.live, kb + kbuf.off, kbuf.words * 4, cudaMemcpyDeviceToDevice, s));
  } else {  // (the device's record disagrees with the host's choice: predict and search again)
    st = apply(*best_scale);
    if (st != CF_OK) return st;
  }
  CF_TRY(cudaStreamSynchronize(s));
  return CF_OK;
}

// ---- warped TSDF integration ----

namespace {

bool tsdf_voxels(const cf_tsdf_params* p, unsigned* V) {
  if (!p) return false;
  long long n = 1;
  for (int a = 0; a < 3; ++a) {
    if (p->dims[a] < 0) return false;
    n *= p->dims[a];
    if (n >= (1LL << 31)) return false;
  }
  *V = (unsigned)n;
  return true;
}

// src/tsdf_volume.cu:34-50: R^T and -(R^T t), each sum of products taken left
// to right with every product and sum rounded (the reference's host build).
void world_to_camera(const cf_mat4& pose, float* rows) {
  float m[3][4];
  for (int i = 0; i < 3; ++i)
    for (int j = 0; j < 3; ++j) m[i][j] = pose.m[j][i];
  for (int i = 0; i < 3; ++i) {
    volatile float a = m[i][0] * pose.m[0][3];
    volatile float b = m[i][1] * pose.m[1][3];
    volatile float c = m[i][2] * pose.m[2][3];
    volatile float ab = a + b;
    volatile float abc = ab + c;
    m[i][3] = -abc;
  }
  for (int i = 0; i < 3; ++i)
    for (int j = 0; j < 4; ++j) rows[4 * i + j] = m[i][j];
}

}  // namespace

cf_status cf_tsdf_reset(cf_tsdf_voxel* d_voxels, long long num_voxels, void* stream) {
  if (num_voxels < 0 || num_voxels >= (1LL << 31) || (num_voxels > 0 && !d_voxels)) return CF_ERR_INVALID_ARG;
  CF_TRY(launch_tsdf_init(d_voxels, (unsigned)num_voxels, (cudaStream_t)stream));
  return CF_OK;
}

cf_status cf_tsdf_world_to_camera(const cf_mat4* camera_pose, cf_mat4* T_cam_world) {
  if (!camera_pose || !T_cam_world) return CF_ERR_INVALID_ARG;
  float rows[12];
  world_to_camera(*camera_pose, rows);
  cf_mat4 out;
  for (int i = 0; i < 3; ++i)
    for (int j = 0; j < 4; ++j) out.m[i][j] = rows[4 * i + j];
  out.m[3][0] = out.m[3][1] = out.m[3][2] = 0.f;
  out.m[3][3] = 1.f;
  *T_cam_world = out;
  return CF_OK;
}

cf_status cf_tsdf_integrate(cf_tsdf_voxel* d_voxels, const cf_tsdf_params* params, const float* d_depth,
                            const cf_camera* cam, const cf_mat4* camera_pose, const cf_deform_node* d_nodes,
                            const cf_dual_quat* d_transforms, int num_nodes, const int* d_voxel_knn,
                            const float* d_voxel_knn_w, const int* d_voxel_opt_counts, int min_opt_count,
                            cf_dual_quat* d_scratch_plain, void* stream) {
  unsigned V = 0;
  if (!tsdf_voxels(params, &V) || !cam || !camera_pose || num_nodes < 0) return CF_ERR_INVALID_ARG;
  if (V == 0) return CF_OK;
  if (!d_voxels || !d_depth || cam->width < 0 || cam->height < 0) return CF_ERR_INVALID_ARG;
  if ((reinterpret_cast<uintptr_t>(d_voxels) | reinterpret_cast<uintptr_t>(d_depth)) & 3u) return CF_ERR_INVALID_ARG;
  // TSDFVolume::integrate: use_warp = (nodes != nullptr && num_nodes > 0)
  const bool warp = d_nodes != nullptr && num_nodes > 0;
  if (warp) {
    if (!d_transforms || !d_voxel_knn || !d_voxel_knn_w || !d_scratch_plain) return CF_ERR_INVALID_ARG;
    if ((reinterpret_cast<uintptr_t>(d_voxel_knn) | reinterpret_cast<uintptr_t>(d_voxel_knn_w) |
         reinterpret_cast<uintptr_t>(d_transforms) | reinterpret_cast<uintptr_t>(d_scratch_plain)) & 15u)
      return CF_ERR_INVALID_ARG;
    if (d_voxel_opt_counts && (reinterpret_cast<uintptr_t>(d_voxel_opt_counts) & 3u)) return CF_ERR_INVALID_ARG;
  }
  float rows[12];
  world_to_camera(*camera_pose, rows);
  cudaStream_t s = (cudaStream_t)stream;
  if (warp) CF_TRY(launch_tsdf_plain(d_nodes, d_transforms, d_scratch_plain, num_nodes, s));
  CF_TRY(launch_tsdf_integrate(reinterpret_cast<float*>(d_voxels), params, d_depth, cam, rows,
                               warp ? d_voxel_knn : nullptr, warp ? d_voxel_knn_w : nullptr,
                               warp ? d_scratch_plain : nullptr, warp ? num_nodes : 0,
                               warp ? d_voxel_opt_counts : nullptr, min_opt_count, s));
  return CF_OK;
}

cf_status cf_tsdf_warp_voxel_centres(float* d_points, const cf_tsdf_params* params, const cf_deform_node* d_nodes,
                                     const cf_dual_quat* d_transforms, int num_nodes, const int* d_voxel_knn,
                                     const float* d_voxel_knn_w, cf_dual_quat* d_scratch_plain, void* stream) {
  unsigned V = 0;
  if (!tsdf_voxels(params, &V) || num_nodes < 0) return CF_ERR_INVALID_ARG;
  if (V == 0) return CF_OK;
  if (!d_points) return CF_ERR_INVALID_ARG;
  const bool warp = d_nodes != nullptr && num_nodes > 0;
  if (warp && (!d_transforms || !d_voxel_knn || !d_voxel_knn_w || !d_scratch_plain ||
               ((reinterpret_cast<uintptr_t>(d_voxel_knn) | reinterpret_cast<uintptr_t>(d_voxel_knn_w) |
                 reinterpret_cast<uintptr_t>(d_transforms) | reinterpret_cast<uintptr_t>(d_scratch_plain)) & 15u)))
    return CF_ERR_INVALID_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  if (warp) CF_TRY(launch_tsdf_plain(d_nodes, d_transforms, d_scratch_plain, num_nodes, s));
  CF_TRY(launch_tsdf_centres(d_points, params, warp ? d_voxel_knn : nullptr, warp ? d_voxel_knn_w : nullptr,
                             warp ? d_scratch_plain : nullptr, warp ? num_nodes : 0, s));
  return CF_OK;
}

cf_status cf_compute_voxel_knn(const cf_tsdf_voxel* d_voxels, const cf_tsdf_params* params,
                               const cf_deform_node* d_nodes, int num_nodes, int* d_voxel_knn, float* d_voxel_knn_w,
                               void* stream) {
  unsigned V = 0;
  if (!tsdf_voxels(params, &V) || num_nodes < 0) return CF_ERR_INVALID_ARG;
  // src/warp_field.cu:962-963: no nodes, no launch and the outputs untouched
  if (V == 0 || num_nodes == 0) return CF_OK;
  if (num_nodes > voxel_knn_max_nodes()) return CF_ERR_CAPACITY;
  if (!d_voxels || !d_nodes || !d_voxel_knn || !d_voxel_knn_w) return CF_ERR_INVALID_ARG;
  if (reinterpret_cast<uintptr_t>(d_voxels) & 3u) return CF_ERR_INVALID_ARG;
  if ((reinterpret_cast<uintptr_t>(d_voxel_knn) | reinterpret_cast<uintptr_t>(d_voxel_knn_w) |
       reinterpret_cast<uintptr_t>(d_nodes)) & 15u)
    return CF_ERR_INVALID_ARG;
  CF_TRY(launch_voxel_knn(reinterpret_cast<const float*>(d_voxels), params, d_nodes, num_nodes, d_voxel_knn,
                          d_voxel_knn_w, 0, (cudaStream_t)stream));
  return CF_OK;
}

cf_status cf_mark_optimized_voxels(const cf_correspondence* d_corrs, const int* d_canonical_vidx, int num_pixels,
                                   const int dims[3], int frame_id, int* d_voxel_opt_counts, int* d_voxel_opt_frame,
                                   void* stream) {
  if (!dims || num_pixels < 0) return CF_ERR_INVALID_ARG;
  long long n = 1;
  for (int a = 0; a < 3; ++a) {
    if (dims[a] <= 0) return CF_ERR_INVALID_ARG;
    n *= dims[a];
    if (n >= (1LL << 31)) return CF_ERR_INVALID_ARG;
  }
  if (num_pixels == 0) return CF_OK;
  if (!d_corrs || !d_canonical_vidx || !d_voxel_opt_counts || !d_voxel_opt_frame) return CF_ERR_INVALID_ARG;
  CF_TRY(launch_mark_optimized(d_corrs, d_canonical_vidx, num_pixels, dims, frame_id, d_voxel_opt_counts,
                               d_voxel_opt_frame, (cudaStream_t)stream));
  return CF_OK;
}

cf_status cf_get_version(int* major, int* minor, int* patch) {
  if (major) *major = 0;
  if (minor) *minor = 1;
  if (patch) *patch = 0;
  return CF_OK;
}

cf_status cf_last_cuda_error(char* buf, size_t len) {
  if (!buf || len == 0) return CF_ERR_INVALID_ARG;
  snprintf(buf, len, "%s", g_last_error);
  return CF_OK;
}

}  // extern "C"
