// cf_internal.h — structures shared by the host API (cf_api.cu) and the
// kernel launchers (cf_kernels.cu).  Not part of the public ABI.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <utility>

#include "../../include/cudafusion_b200.h"

namespace cf {

constexpr int kThreads = 256;

constexpr unsigned kEarlyCtas = 32 * 148;

// A kernel that may be set up while the one before it in the stream still runs:
// its CTAs take what room there is and wait in after_previous() until all of
// that kernel, and so all before it, is done and visible.  A call is a row of
// short kernels; what a launch costs between two of them is hidden this way:
// some 0.8 us per kernel of a solve (24 of them, 320 -> 300 us at 256 nodes), 1.8 of
// a prediction's five (39 -> 30 us).
template <typename... Params, typename... Args>
inline cudaError_t launch_next(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t s,
                               Args&&... args) {
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = &attr;
  // (past that many CTAs the launch no longer matters, and a wait per CTA does)
  cfg.numAttrs = (unsigned long long)grid.x * grid.y * grid.z <= kEarlyCtas ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

#ifdef __CUDACC__
// Every kernel that launch_next launches calls it, in all its CTAs and before an
// early return, before its first write and before it reads what the launch before
// it writes.  Only then is the next kernel let in, so what lies two or more launches
// back is done when a kernel starts, and that alone may be read ahead of the call.
// What the launch before writes is not constant for the kernel's life, even though it
// is read after the call: no __ldg and no const __restrict__ for it.
__device__ __forceinline__ void after_previous() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
#endif
constexpr int kErrTimeoutBit = 1;   // bounded barrier gave up
constexpr int kErrNonFiniteBit = 2; // NaN/Inf in the solution or energy
constexpr int kStatsSlots = CF_MAX_GN_ITERS + 1;
// float4 per ARAP edge in Pattern::edge_terms: diagonal block + rhs of i (7),
// of j (7), off-diagonal block (9)
constexpr int kEdgeTerms4 = 23;

// Device-side statistics of one solve (copied to cf_solve_stats on request).
struct DevStats {
  double energy[kStatsSlots];          // energy at each linearisation point; [G] = final
  double pcg_res[CF_MAX_GN_ITERS];     // final ||r|| per GN iteration
  int pcg_iters[CF_MAX_GN_ITERS];
  int fallbacks;                        // Cholesky fallbacks of the last GN iteration
  int init_rejected;                    // learned solve: the predicted start was not kept
  double gate[2];                       // learned solve: energy at the warm start, at the prediction
};

// One problem of a solve as the kernels see it; a single solve is a batch of
// one.  Correspondences and nodes of all problems live in one concatenated
// index space (node ids inside the packed records are global).
struct ProbDesc {
  const cf_correspondence* corrs;  // the caller's rows, indexed locally
  const float* canon;              // canonical points (nullptr: linearise at src)
  const cf_deform_node* nodes;     // the caller's nodes (batched solves gather them)
  cf_dual_quat* T;                 // the caller's transforms (batched solves gather/scatter)
  long long cnt_off;               // first histogram word of this problem in Work::cnt
  int M, N;
  int corr_off, node_off;          // first correspondence / node in the concatenated space
  int bin_cta0, bin_ctas, chunk;   // sort CTAs of this problem, correspondences per CTA
  int e_cta0, e_ctas;              // residual / energy CTAs, one FP64 partial each
  float max_rot, max_trans, update_scale;
  int pad_[2];
};
static_assert(sizeof(ProbDesc) == 96, "ProbDesc has no padding (compared bytewise)");

// Per-call problem table (device copies of the host arrays).
struct Table {
  int P = 0;
  int n_bin = 0, n_e = 0;    // total sort / energy CTAs
  int M = 0, N = 0;          // concatenated sizes
  int max_N = 0;             // largest problem (shared-memory histograms)
  int max_chunk = 0;         // most correspondences of one sort CTA
  ProbDesc* desc = nullptr;  // [P]
  int* bin_prob = nullptr;   // [n_bin] problem of each sort CTA
  long long bin_cap = 0;     // capacity of bin_prob
  int* e_prob = nullptr;     // [n_e] problem of each energy CTA
  int* node_prob = nullptr;  // [N] problem of each node
};

// Block pattern and everything derived from the graph topology.  Built on
// the host (cold path, kernels/solver_kernels.cu:498-541) and uploaded.
struct Pattern {
  int P = 1;               // problems (block-diagonal union for batched solves)
  int* prob_edge_off = nullptr;  // [P+1] ARAP edges of each problem (edge_ijk order)
  int* pcg_cta_off = nullptr;    // [P+1] PCG CTA group of each problem
  int* pcg_prob = nullptr;       // [pcg_ctas] problem of each PCG CTA
  int N = 0;
  int nnzb = 0;
  int n_upper = 0;      // blocks with col >= row (incl. diagonal)
  int n_edges = 0;      // ARAP edges visited by the reference (lower endpoint owns)
  int* row_ptr = nullptr;   // [N+1]
  int* col_idx = nullptr;   // [nnzb]
  int* diag_pos = nullptr;  // [N]
  int4* upper_meta = nullptr; // [n_upper] row, position, column, position of the transpose
  int* arap_row_ptr = nullptr;  // [N+1]
  int* arap_row_inc = nullptr;  // (edge << 1) | role, role 0 = lower endpoint
  int* arap_blk_ptr = nullptr;  // [n_upper+1] over upper off-diagonal blocks
  int* arap_blk_edge = nullptr;
  int* edge_ijk = nullptr;      // [3*n_edges] i, j, k (slot in i's list)
  float4* edge_terms = nullptr; // [kEdgeTerms4*n_edges] per GN iteration: the edge's block contributions
  double* edge_energy = nullptr; // [n_edges] per GN iteration: el |r|^2
  // per-pattern work arrays
  float* values = nullptr;  // [nnzb*36]
  // single-cluster PCG (cf_pcg_cluster.cu)
  int use_cluster = 0;
  int clu_C = 0;
  int clu_smem = 0;
  int clu_blk_max = 0, clu_rows_max = 0, clu_halo_max = 0;
  int* clu_row_begin = nullptr;  // [clu_C+1]
  int* ustart = nullptr;         // [N+1] first upper index of each row
  int* clu_vidx = nullptr;       // [nnzb] operand slot of the block's column in its CTA: own row, or rows + halo slot
  int* clu_halo_ptr = nullptr;   // [clu_C+1] halo rows before each CTA's
  int* clu_halo = nullptr;       // per CTA, its remote columns: (owner << 24) | row local to the owner
  // grid PCG partition
  int pcg_ctas = 0;
  int* pcg_row_begin = nullptr;  // [pcg_ctas+1]
  int pcg_smem = 0;
  int pcg_a_in_smem = 0;
  int pcg_pipelined = 0;
  int* g_vidx = nullptr;      // [nnzb] operand slot of each block's column in its CTA ([own | halo])
  int* g_halo_ptr = nullptr;  // [pcg_ctas+1]
  int* g_halo_col = nullptr;  // distinct columns of other CTAs touched by each CTA
  // streaming PCG (cf_pcg_stream.cu): A streamed from HBM in tiles of whole rows
  int pcg_stream = 0;
  int st_tile_blocks = 256;    // blocks per tile (256 or 128)
  int* st_tile_ptr = nullptr;  // [pcg_ctas+1] into st_tile_row
  int* st_tile_row = nullptr;  // per CTA: its tiles' first rows, then its end row
  int* st_tile_cols = nullptr; // [entries of st_tile_row][tile blocks] each tile's column indices, -1 padded
};

// Per-handle work buffers sized by (max_nodes, max_corrs).
struct Work {
  int max_nodes = 0, max_corrs = 0;
  int bin_ctas_max = 0;
  // the correspondences in the order of their node sets (cf_cells.cu)
  uint2* key = nullptr;       // [max_corrs] per correspondence: its distinct nodes, ascending, 16-bit local ids
  int* order = nullptr;       // [max_corrs] the correspondences in order of their first node
  int* sorted = nullptr;      // [max_corrs] and in order of the whole set
  float4* sp_src = nullptr;   // [max_corrs] canonical point (solve) or src (linearise), effective weight
  float4* sp_dst = nullptr;   // target, which node of the set each slot names (3 bits per slot, 7: none)
  float4* sp_nrm = nullptr;   // normal; w: residual (tasks without a record)
  float4* sp_uw = nullptr;    // the skin weights of the set's nodes
  unsigned char* task = nullptr;  // [max_corrs] size of the task that starts at the position, else 0
  int4* cell_ids = nullptr;   // [max_corrs] at a task's first position: its nodes, ascending, -1 past the last
  float* rec = nullptr;       // [max_corrs / kRecMin + 2][kRecFloats] the tasks' sums
  float4* raw = nullptr;      // [max_corrs] skinned src, fw (0 = skipped) of tasks without a record
  float4* cstat = nullptr;    // [max_corrs] at a task's first position: sum |r|, max |r|, count (learned start)
  int* cl_total = nullptr;    // [max_nodes] tasks that contain the node
  int* cl_start = nullptr;    // [max_nodes+1]
  int* cl_cur = nullptr;      // [max_nodes]
  float4* npos = nullptr;     // [max_nodes] node positions
  int* clist = nullptr;       // [4*max_corrs] per node its tasks, in position order
  int* cnt = nullptr;         // per sort CTA, a histogram over its problem's nodes
  long long cnt_cap = 0;      // words allocated for cnt
  int* node_total = nullptr;  // [max_nodes]
  int* inc_start = nullptr;   // [max_nodes+1] first sorted position of each node's bucket
  uint4* cdesc = nullptr;     // [4*max_corrs] their descriptions for the gather
  float* rhs = nullptr;       // [6*max_nodes]
  cf_dual_quat* plain = nullptr;  // [max_nodes]
  float* x = nullptr;         // [6*max_nodes]
  float* z = nullptr;
  float* p0 = nullptr;
  float* p1 = nullptr;
  float* zp = nullptr;        // [2][max_nodes][12] z and p of the streaming PCG
  double* partials = nullptr;  // [2 bufs][3 slots][max pcg ctas]
  unsigned* barrier = nullptr;  // [max pcg ctas] one arrival counter per PCG CTA group (zeroed by the gather)
  unsigned long long* dots = nullptr;  // [max pcg ctas][3 lines] per group: exchanged sums (cf_pcg_grid.cu)
  int* err = nullptr;
  unsigned* done = nullptr;       // CTAs of an energy launch that have finished (0 between launches)
  double* e_data_part = nullptr;  // [kMaxEnergyCtas + kMaxProblems] one partial per energy CTA
  double* e_arap_part = nullptr;  // [max_nodes] per row
  DevStats* stats = nullptr;      // [kMaxProblems]
  // streaming PCG: residual, A p and the FP32 block inverses in global memory
  float* r = nullptr;       // [6*max_nodes]
  float* ap = nullptr;      // [6*max_nodes]
  float* minv32 = nullptr;  // [36*max_nodes]
  cf_dual_quat* T_save = nullptr;  // [max_nodes] learned solve: the warm start
  // batched solves: the problems' nodes and transforms, concatenated
  cf_deform_node* nodes_cat = nullptr;  // [max_nodes]
  cf_dual_quat* T_cat = nullptr;        // [max_nodes]
  long long* timers = nullptr;  // [kTimerSlots] phase cycles of the grid PCG (debug)
};

// CTAs of the data term.  A single solve's share it evenly in one wave (two per
// SM; 148 SMs).  A batch's problems differ, so up to eight waves once each warp
// still has 16 windows of 32 correspondences: a problem's CTAs are whole ones.
constexpr int kEnergyCtas = 296;
constexpr int kMaxEnergyCtas = 8 * kEnergyCtas;
constexpr int kEnergyMinPerCta = 8 * 32 * 16;
constexpr int kMaxPcgCtas = 1024;
constexpr int kSortChunk = 512;  // sorted positions of a bucket's chunk (cf_cells.cu)
// Tasks of at least kRecMin correspondences leave a record of sums; one that
// starts at position q owns record ceil(q / kRecMin), which no other does,
// so records are bounded by the correspondences.  In smaller ones (under 2 % of
// the correspondences of a frame) the gather reads each correspondence.
constexpr int kRecMin = 4;
constexpr int kRecFloats = 236;  // 10 pairs x 21 sums, 4 x 6 right-hand sides, padded to 16 B
constexpr int kSortCorrs = 4096;     // correspondences per sort CTA of a batched solve (at least)
constexpr int kMaxSortCtas = 1 << 16;
// Rows per CTA up to which mode 0 picks the single-cluster PCG.  Its exchanges
// are shorter than the grid's, its 16 SMs hold more rows each; per launch of 12-13
// iterations on B200: 256 nodes 52 us (grid 78), 512 nodes 52 (grid 70), 1024
// nodes 75 (grid 72), 2048 nodes 105 (grid 81).
constexpr int kClusterAutoRows = 48;
constexpr int kMaxProblems = 1024;       // problems per batched solve
constexpr int kMaxProblemNodes = 48000;  // nodes per problem (per-CTA histograms in shared memory)

struct SolveArgs {
  const cf_deform_node* nodes;
  int N;
  int M;
  float lambda_smooth;
  float lambda_damping;
  int pcg_iterations;
  float pcg_tolerance;
  int arap_consistent;
  // node update (solve) or plain delta_x output (linearise)
  cf_dual_quat* transforms;  // in/out
  float* delta_x;            // non-null: write dx here and do not update
  float max_rot, max_trans, update_scale;
  unsigned spin_limit;
  unsigned bar_extra;  // test hook: arrivals every group barrier waits for beyond its CTAs (0)
  long long* timers;  // non-null: CTA 0 of the grid PCG accumulates phase cycles here
  Table tb;           // the problems of this solve
};
constexpr int kTimerSlots = 16;

#ifdef __CUDACC__
// clock64 phase timer of one thread of the persistent PCG kernels (debug;
// a.timers == nullptr disables it)
struct PhaseClock {
  long long* out;
  long long last;
  long long acc[kTimerSlots];
  __device__ PhaseClock(long long* o) : out(o), last(0) {
#ifdef __CUDA_ARCH__
    last = clock64();
#endif
    for (int i = 0; i < kTimerSlots; i++) acc[i] = 0;
  }
  __device__ __forceinline__ void mark(int slot) {
#ifdef __CUDA_ARCH__
    if (!out) return;
    const long long t = clock64();
    acc[slot] += t - last;
    last = t;
#endif
  }
  __device__ void flush() {
    if (!out) return;
    for (int i = 0; i < kTimerSlots; i++) atomicAdd(reinterpret_cast<unsigned long long*>(out + i), (unsigned long long)acc[i]);
  }
};
#endif


// ---- launchers (cf_kernels.cu) ----
cudaError_t launch_key_count(const Work& w, const Table& tb, cudaStream_t s);
cudaError_t launch_bin_scan(const Work& w, const Table& tb, bool reset_stats, cudaStream_t s);
cudaError_t launch_bin_scatter(const Work& w, const Table& tb, cudaStream_t s);
cudaError_t launch_node_setup(const Work& w, const Table& tb, bool reset_stats, cudaStream_t s);
cudaError_t launch_list_scan(const Work& w, const Table& tb, cudaStream_t s);
// cf_cells.cu
cudaError_t launch_bucket_sort(const Work& w, const Table& tb, cudaStream_t s);
cudaError_t launch_node_lists(const Work& w, const Table& tb, const Pattern& p, cudaStream_t s);
cudaError_t launch_residual(const Work& w, const Table& tb, const Pattern& p, const SolveArgs& a,
                            const cf_dual_quat* T, bool skin, cudaStream_t s);
cudaError_t launch_batch_gather(const Work& w, const Table& tb, cudaStream_t s);
cudaError_t launch_batch_scatter(const Work& w, const Table& tb, cudaStream_t s);
cudaError_t launch_assemble(const Work& w, const Pattern& p, const SolveArgs& a, cudaStream_t s);
cudaError_t launch_pcg(const Work& w, const Pattern& p, const SolveArgs& a, int gn_slot, cudaStream_t s);
constexpr int kNoSlot = -1000;  // (launch_final_energy) the energy is not kept
cudaError_t launch_final_energy(const Work& w, const Pattern& p, const SolveArgs& a, int slot, cudaStream_t s,
                                bool stats = false);
cudaError_t launch_apply_twist(cf_dual_quat* T, const float* dx, int N, float max_rot, float max_trans,
                               float scale, cudaStream_t s);
// cf_corr.cu: projective correspondence search
constexpr int kCorrMaxChunks = 8;
struct CorrScratch {
  float4* A;       // per pixel: unprojected point (x, y, z) and normal x
  float2* B;       // per pixel: normal y, z
  float4* part_a;  // [chunk_cap][pixels]: each row chunk's three least values, and their error bound
  int2* part_g;    // [chunk_cap][pixels]: the runs of the first two
  int2* rows;      // per tile of pixels: the rows that it scans, by chunk
  int* todo;       // [1 + kCorrMaxChunks * tiles]: what is left to the exact scan
  void* box;       // [blocks]: what is known of each block of 16 x 16 pixels
  float4 *pix_v, *pix_n;  // per pixel: its camera-frame point, normal, projection ...
  int* pix_row;           // ... and state
  int chunk_cap;
  int* flag;       // set when a value could make a distance NaN
  int sms;
};
int corr_pick_chunks(int tiles, int sms, int radius, int W, int H, bool filter);
int corr_chunk_cap(size_t P);
size_t corr_box_cap(size_t P);
size_t corr_box_bytes();
// cf_linesearch.cu: the GN step's acceptance
cudaError_t launch_update_stats(const float* dx, int N, float update_scale, float max_rot, float max_trans,
                                double* sums, unsigned* maxima, int* finite, cudaStream_t s);
cudaError_t launch_scale_delta(const float* dx, int N, float max_rot, float max_trans, float scale, float* out,
                               cudaStream_t s);
// The line search's record of its best trial (ls_keep_kernel).
struct LsKeepArgs {
  const double* part;  // the trial's block sums
  const int* valid;    // and valid count
  double* slot;        // where both go
  const double* best_in;  // nullptr: best0
  double best0;
  double* best_out;
  int* kept;
  int trial, min_valid, need, nbuf;
  const int* src[8];
  int* dst[8];
  size_t words[8];
};
cudaError_t launch_ls_keep(const LsKeepArgs& a, cudaStream_t s);
// out: nullptr leaves the block sums alone
cudaError_t launch_corr_rmse(const cf_correspondence* corrs, int M, double* partials, double* out, cudaStream_t s);
cudaError_t launch_trial_transforms(const cf_dual_quat* saved, const float* dx, int N, float max_rot, float max_trans,
                                    float scale, float* delta, cf_dual_quat* T, cudaStream_t s);
cudaError_t launch_tsdf_plain(const cf_deform_node* nodes, const cf_dual_quat* T, cf_dual_quat* plain, int N,
                              cudaStream_t s);
cudaError_t launch_tsdf_integrate(float* vox, const cf_tsdf_params* p, const float* depth, const cf_camera* cam,
                                  const float* cw, const int* knn, const float* knn_w, const cf_dual_quat* plain,
                                  int N, const int* counts, int min_opt, cudaStream_t s);
cudaError_t launch_tsdf_centres(float* out, const cf_tsdf_params* p, const int* knn, const float* knn_w,
                                const cf_dual_quat* plain, int N, cudaStream_t s);
cudaError_t launch_mark_optimized(const cf_correspondence* corrs, const int* vidx, int P, const int dims[3],
                                  int frame, int* counts, int* frames, cudaStream_t s);
cudaError_t launch_tsdf_init(cf_tsdf_voxel* vox, unsigned V, cudaStream_t s);
// cf_voxelknn.cu: the voxel kNN field (variant 0: default pruning, 1: tile
// pruning only, 2: tile and warp pruning)
int voxel_knn_max_nodes();
cudaError_t launch_voxel_knn(const float* vox, const cf_tsdf_params* p, const cf_deform_node* nodes, int N,
                             int* ids, float* ws, int variant, cudaStream_t s);
// cf_raster.cu: live-surface prediction
cudaError_t launch_mesh_skin(const float* canon, float* warped, int V, const cf_voxel_grid* grid,
                             const cf_deform_node* nodes, const cf_dual_quat* T, int N, const int* vk, const float* vw,
                             cudaStream_t s);
cudaError_t launch_mesh_skin_plain(const float* canon, float* warped, int V, const cf_voxel_grid* grid,
                                   const cf_dual_quat* plain, int N, const int* vk, const float* vw, cudaStream_t s);
cudaError_t launch_raster(const float* canon, const float* warped, const int* tris, int V, int NT,
                          const cf_camera* cam, const cf_mat4* Tcw, const cf_voxel_grid* grid,
                          unsigned long long* ztri, float4* cache, int* big, unsigned long long* big_ctr, float* lv,
                          float* ln, int* hit, cudaStream_t s, long long* launches);
cudaError_t launch_corr_search(const cf_corr_frame* f, const cf_camera* cam, const cf_mat4* Tcw, const cf_mat4* Twc,
                               const cf_corr_params* p, const CorrScratch& sc, int chunks, cf_correspondence* out,
                               int* num_valid, int* stats, cudaStream_t s, long long* launches);
cudaError_t launch_pixel_knn(const int* hit, int P, const int* vk, const float* vw, long long num_voxels, int* pk,
                             float* pw, cudaStream_t s);
cudaError_t launch_skin_points(const float* pts, const int* ids, const float* ws, int M,
                               const cf_deform_node* nodes, const cf_dual_quat* T, int N, float* out,
                               cudaStream_t s);
cudaError_t launch_energy_noalloc(const cf_problem* pr, const cf_dual_quat* T, float lambda, double* d_energy,
                                  cudaStream_t s);
int pcg_grid_smem_bytes(int nblk, int nrows, int nhalo, bool a_in_smem, bool pipelined);
int pcg_max_active_ctas(int smem, bool a_in_smem, bool pipelined);

int pcg_cluster_max_rows();
int pcg_cluster_smem_bytes(int blk_max, int rows_max, int nhalo_max, int C);
int pcg_cluster_max_active(int C, int rows_max, int smem);
cudaError_t launch_pcg_cluster(const Work& w, const Pattern& p, const SolveArgs& a, int gn_slot, cudaStream_t s);

// The learned initial increment (cf_mpnn.cu): parameters, graph, activations.
struct Mpnn {
  int max_nodes = 0, N = 0;
  long long step = 0;
  float *w = nullptr, *m = nullptr, *v = nullptr, *g = nullptr;  // FP32 master, Adam moments, gradient
  void* wb = nullptr;                                            // BF16 parameters
  int* nbr = nullptr;       // [N][8] neighbour lists, -1 = none
  float* inv_deg = nullptr;  // [N]
  int *rev_ptr = nullptr, *rev_idx = nullptr;  // reverse graph (training)
  float *feat = nullptr, *tgt = nullptr, *out = nullptr;
  void *h1 = nullptr, *h2 = nullptr, *h3 = nullptr;  // BF16 activations [N][64]
  float *dh = nullptr, *dcat2 = nullptr, *dcat = nullptr, *part = nullptr;
  double *loss_part = nullptr, *loss = nullptr;
};
int mpnn_param_count();
cudaError_t mpnn_alloc(Mpnn& m, int max_nodes);
void mpnn_free(Mpnn& m);
cudaError_t mpnn_refresh_bf16(const Mpnn& m, cudaStream_t s);
cudaError_t mpnn_graph_from_nodes(Mpnn& m, const cf_deform_node* nodes, int N, cudaStream_t s);
cudaError_t mpnn_forward(const Mpnn& m, const float* feat, float* out, cudaStream_t s);
cudaError_t mpnn_gradients(Mpnn& m, const float* feat, const float* tgt, cudaStream_t s);
cudaError_t mpnn_adam(Mpnn& m, float lr, cudaStream_t s);
cudaError_t launch_increments(const cf_dual_quat* to, const cf_dual_quat* from, int n, float* out, cudaStream_t s);
cudaError_t launch_features(const Work& w, const cf_dual_quat* T, const cf_dual_quat* hist, int N, float* feat,
                            cudaStream_t s);
cudaError_t launch_apply_prediction(const Work& w, cf_dual_quat* T, const cf_deform_node* nodes, const float* pred,
                                    int N, cudaStream_t s);
cudaError_t launch_gate_prediction(const Work& w, cf_dual_quat* T, const cf_deform_node* nodes, int N,
                                   cudaStream_t s);

int pcg_stream_smem_bytes(int tile_blocks);
int pcg_stream_max_active_ctas(int tile_blocks);
cudaError_t launch_pcg_stream(const Work& w, const Pattern& p, const SolveArgs& a, int gn_slot, cudaStream_t s);

}  // namespace cf
