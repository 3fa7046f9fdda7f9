// cf_pcg_cluster.cu — block-Jacobi PCG of one problem inside ONE thread-block
// cluster (sm_100a).
//
// Each CTA of a 16- or 8-CTA cluster owns a contiguous range of block rows
// (balanced by block count); their full rows of A stay in its shared memory.
// A warp holds whole rows (1, 2 or 5 of them, 4, 2 or 1 lanes per row
// element), so a row's residual and its product with the FP64 block inverse
// (a row of the inverse per element, in registers) stay within the warp.  The
// operand of other CTAs' rows (the CTA's halo) is kept as p = z + beta p_old
// from the owners' z, read through cluster-mapped shared memory, so p itself is
// never waited for.
//
// Two exchanges per iteration and no cluster barrier: p.Ap, and r.r with r.z.
// One warp adds the CTA's products and sends the sum to every CTA as an
// asynchronous remote store that completes a transaction on the receiver's
// mbarrier; a CTA goes on when its own barrier has counted a message from each
// CTA, and its first warp adds those in the same order as everywhere.  One message per CTA: with 1,
// 8 and 24 messages per CTA such an exchange takes 350, 1080 and 1420 cycles, a
// remote store followed by a cluster barrier 1090.  The second exchange also
// says that the owners' z is there.  A slot, and z, are written again only after
// the writer has heard, in the exchange between, from every CTA that reads them.
//
// Schedule and guards follow kernels/solver_kernels.cu:616-687 (PCG from
// x = 0, |p.Ap| < 1e-12 stops before the update, ||r|| < tol after it); FP64
// block inverses and dot products, FP32 matrix and vectors.  The waits are
// bounded (polls, and time): past the limit a CTA records kErrTimeout and leaves the
// iterations, the others follow when they see that, and none exits while a message
// may still be under way to it.
//
// Measured (B200, event time of a launch less its fixed 10-20 us): 2.8 us per
// iteration at 256 nodes, 3.1 at 512, 4.6 at 1024, 6.4 at 2048; with upper blocks
// only, transposed products pushed to their owners and three cluster barriers
// per iteration it was 4.05 at 256 and 8.6 at 2048 nodes.
//
// What bounds it: the chain of latencies of an iteration (row sums, an FP64 warp
// sum, a remote store, the sum of the messages, a divide, twice, and a remote
// load), and past about 60 rows per CTA the shared-memory reads of A.
#include <cooperative_groups.h>

#include "cf_device.cuh"
#include "cf_internal.h"

namespace cg = cooperative_groups;

namespace cf {

namespace {

__host__ __device__ inline int al16(int x) { return (x + 15) & ~15; }

constexpr int kInvGroupBytes = (72 + 36) * 8;  // inv6_group scratch and result, per 8 lanes

struct CluLayout {
  int a, vidx, urow, p, z, halo, tn, dot, msg, bar, ctl, total;
};

__host__ __device__ inline CluLayout clu_layout(int nblk, int rows, int nhalo, int threads, int C) {
  CluLayout L;
  int o = 0;
  // the rows of A; their space first holds the diagonal blocks and the scratch
  // of the inverses, one 8-lane group per row at a time
  int a = nblk * 36 * 4;
  const int scr = al16(rows * 36 * 4) + threads / 8 * kInvGroupBytes;
  a = a > scr ? a : scr;
  L.a = o; o += al16(a);
  L.vidx = o; o += al16(nblk * 2);
  L.urow = o; o += al16((rows + 1) * 4);
  L.p = o; o += al16((rows + nhalo) * 6 * 4);
  L.z = o; o += al16(rows * 6 * 4);
  L.halo = o; o += al16(nhalo * 4);
  L.tn = o; o += al16(rows * 48);
  L.dot = o; o += rows * 6 * 16;     // per element r.r and r.z, or p.Ap
  L.msg = o; o += C * (8 + 16 + 8);  // [C] p.Ap, [C] (r.r, r.z), [C] energy shares
  L.bar = o; o += 16;
  L.ctl = o; o += 16;                // the step of the CTA's threads: alpha or beta, stop
  L.total = o;
  return L;
}

struct CluArgs {
  Work w;
  Pattern pt;
  SolveArgs a;
  int slot;
};

// ---- cluster shared memory and its barriers (addresses in the shared window) ----
__device__ __forceinline__ unsigned smem_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ unsigned remote(unsigned addr, int rank) {
  unsigned r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void send_f64(unsigned addr, double v, unsigned bar) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(addr),
               "l"(__double_as_longlong(v)), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void send_f64x2(unsigned addr, double u, double v, unsigned bar) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.b64 [%0], {%1, %2}, [%3];" ::"r"(addr),
               "l"(__double_as_longlong(u)), "l"(__double_as_longlong(v)), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void bar_init(unsigned bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void bar_arrive_expect(unsigned bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.release.cta.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool bar_try(unsigned bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}

constexpr long long kClWaitCycles = 1ll << 32;  // a wait gives up after about two seconds, or spin_limit polls
constexpr long long kClDrainCycles = 1ll << 17;  // far longer than a message takes

// A row's residual, x, z and its row of the inverse live with the first of its
// kSpl lanes per element.
template <int kSpl>
__global__ void __launch_bounds__(kSpl == 1 ? 1024 : 768, 1) pcg_cluster_kernel(CluArgs P) {
  extern __shared__ __align__(16) unsigned char smem[];
  constexpr int kRowLanes = 6 * kSpl, kRowsPerWarp = 32 / kRowLanes;
  cg::cluster_group cluster = cg::this_cluster();
  const Work& w = P.w;
  const Pattern& pt = P.pt;
  const SolveArgs& a = P.a;
  const int C = (int)cluster.num_blocks();
  const int crank = (int)cluster.block_rank();
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, nthreads = blockDim.x;
  const ProbDesc& pd = a.tb.desc[0];  // the cluster path serves single solves
  DevStats* st = w.stats;
  const int r0 = pt.clu_row_begin[crank], r1 = pt.clu_row_begin[crank + 1];
  const int nrows = r1 - r0;
  const int b0 = pt.row_ptr[r0], nblk = pt.row_ptr[r1] - b0;
  const int h0 = pt.clu_halo_ptr[crank], nhalo = pt.clu_halo_ptr[crank + 1] - h0;
  const CluLayout L = clu_layout(pt.clu_blk_max, pt.clu_rows_max, pt.clu_halo_max, nthreads, C);
  float* sA = reinterpret_cast<float*>(smem + L.a);
  unsigned short* sVidx = reinterpret_cast<unsigned short*>(smem + L.vidx);
  int* sRow = reinterpret_cast<int*>(smem + L.urow);
  float* sP = reinterpret_cast<float*>(smem + L.p);  // own rows, then the halo
  float* sZ = reinterpret_cast<float*>(smem + L.z);
  int* sHalo = reinterpret_cast<int*>(smem + L.halo);
  float4* sTn = reinterpret_cast<float4*>(smem + L.tn);
  double* sDot = reinterpret_cast<double*>(smem + L.dot);
  double* msgA = reinterpret_cast<double*>(smem + L.msg);
  double* msgB = msgA + C;  // (r.r, r.z) pairs
  double* sEnergy = msgB + 2 * C;
  float* sStep = reinterpret_cast<float*>(smem + L.ctl);
  volatile int* sStop = reinterpret_cast<volatile int*>(smem + L.ctl + 4);
  const unsigned barA = smem_addr(smem + L.bar), barB = barA + 8;
  const int n6 = nrows * 6, h6 = nhalo * 6;
  int* err = w.err;
  if (tid == 0) {
    bar_init(barA, 1 + min(a.bar_extra, 1024u));
    bar_init(barB, 1 + min(a.bar_extra, 1024u));
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  // Distributed shared memory may be touched only once every CTA of the
  // cluster runs (and its barriers are there): arrive now, wait before the
  // first remote store.
  asm volatile("barrier.cluster.arrive.aligned;" ::: "memory");

  // ---- prologue ----
  // the plan, while the assembly may still run; then the diagonal blocks, by
  // cp.async, and everything small
  for (int k = tid; k < nblk; k += nthreads) sVidx[k] = (unsigned short)__ldg(pt.clu_vidx + b0 + k);
  for (int k = tid; k < nhalo; k += nthreads) sHalo[k] = __ldg(pt.clu_halo + h0 + k);
  for (int i = tid; i <= nrows; i += nthreads) sRow[i] = __ldg(pt.row_ptr + r0 + i) - b0;
  after_previous();
  const float* gA = pt.values + (size_t)b0 * 36;
  float* sD = sA;
  unsigned char* scr0 = smem + L.a + al16(nrows * 36 * 4);
  for (int e = tid; e < nrows * 9; e += nthreads) {
    const int i = e / 9, q = e - 9 * i;
    cp_async16(sD + 36 * i + 4 * q, pt.values + (size_t)__ldg(pt.diag_pos + r0 + i) * 36 + 4 * q);
  }
  if (!a.delta_x)  // the epilogue's operands (transform, node position)
    for (int i = tid; i < nrows; i += nthreads) {
      const float4* tq = reinterpret_cast<const float4*>(a.transforms + r0 + i);
      cp_async16(sTn + 3 * i, tq);
      cp_async16(sTn + 3 * i + 1, tq + 1);
      const float* np = reinterpret_cast<const float*>(a.nodes + r0 + i);
      float* sp = reinterpret_cast<float*>(sTn + 3 * i + 2);
      cp_async4(sp, np);
      cp_async4(sp + 1, np + 1);
      cp_async4(sp + 2, np + 2);
    }
  cp_async_commit();
  // this lane's row, its element and its share of the element's blocks
  const int rl = lane / kRowLanes, c = (lane - rl * kRowLanes) / kSpl, ks = lane % kSpl;
  const int row = wid * kRowsPerWarp + rl;
  const bool act = rl < kRowsPerWarp && row < nrows, own = act && ks == 0;
  const int t = act ? row * 6 + c : 0;
  float r = own ? __ldcg(w.rhs + r0 * 6 + t) : 0.f, x = 0.f;
  // this CTA's share of the energy at the linearisation point (the data
  // partials, then the ARAP node partials)
  double pen = 0.0;
  {
    const int n1 = pd.e_ctas, n = pd.e_ctas + pd.N, chunk = (n + C - 1) / C;
    const int k1 = min(n, (crank + 1) * chunk);
    for (int k = crank * chunk + tid; k < k1; k += nthreads)
      pen += k < n1 ? __ldcg(w.e_data_part + pd.e_cta0 + k) : __ldcg(w.e_arap_part + pd.node_off + (k - n1));
  }
  cp_async_wait<0>();
  __syncthreads();
  // block-Jacobi inverses in FP64, one 8-lane group per row; an element's
  // first lane keeps its row of the inverse
  double minv[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
  {
    double* scr = reinterpret_cast<double*>(scr0 + (tid >> 3) * kInvGroupBytes);
    const int groups = nthreads / 8;
    int nfb = 0;
    for (int i0 = 0; i0 < nrows; i0 += groups) {
      const int i = i0 + (tid >> 3);
      nfb += inv6_group(sD + (i < nrows ? i : 0) * 36, scr, scr + 72, i < nrows) && (tid & 7) == 0;
      __syncthreads();
      if (own && row >= i0 && row < i0 + groups) {
        const double* m = reinterpret_cast<const double*>(scr0 + (row - i0) * kInvGroupBytes) + 72 + 6 * c;
#pragma unroll
        for (int q = 0; q < 6; q++) minv[q] = m[q];
      }
      __syncthreads();
    }
    if (nfb) atomicAdd(&st->fallbacks, nfb);
  }
  // the rows of A, over the scratch
  for (int e = tid; e < nblk * 9; e += nthreads) cp_async16(sA + 4 * e, gA + 4 * e);
  cp_async_commit();

  bool dead = false;
  auto wait = [&](unsigned bar, unsigned parity) {
    if (dead || bar_try(bar, parity)) return;
    const long long t0 = clock64();
    for (unsigned tries = 1; !bar_try(bar, parity); tries++) {
      if (tries & 63) continue;
      if (tries > a.spin_limit || clock64() - t0 > kClWaitCycles) atomicOr(err, kErrTimeout);
      if (*(volatile int*)err & kErrTimeout) {
        dead = true;
        return;
      }
    }
  };
  // z = M^-1 r (FP64, rounded once): the row's residual from its first lanes
  auto precond = [&]() -> float {
    double zz = 0.0;
#pragma unroll
    for (int q = 0; q < 6; q++) zz += minv[q] * (double)__shfl_sync(0xffffffffu, r, min(rl * kRowLanes + q * kSpl, 31));
    return (float)zz;
  };
  // r.r and r.z of the CTA, with z in place, to every CTA
  float z = 0.f;
  auto send_b = [&]() {
    z = precond();
    if (own) {
      sZ[t] = z;
      *reinterpret_cast<double2*>(sDot + 2 * t) = make_double2((double)r * r, (double)r * z);
    }
    __syncthreads();
    if (wid == 0) {
      double rr = 0.0, rz = 0.0;
      for (int k = lane; k < n6; k += 32) {
        const double2 v = *reinterpret_cast<const double2*>(sDot + 2 * k);
        rr += v.x;
        rz += v.y;
      }
      rr = warp_sum_d(rr);
      rz = warp_sum_d(rz);
      if (lane < C) send_f64x2(remote(smem_addr(msgB + 2 * crank), lane), rr, rz, remote(barB, lane));
      if (lane == 0) bar_arrive_expect(barB, (unsigned)C * 16u);
    }
  };
  // the cluster's sums of the messages, the same bits in every CTA (warp 0)
  auto sum_a = [&]() -> double {
    const int k = lane & 15;
    double v = k < C ? msgA[k] : 0.0;
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
  };
  auto sum_b = [&](double& rr, double& rz) {
    const int k = lane & 15;
    const double2 m = k < C ? *reinterpret_cast<const double2*>(msgB + 2 * k) : make_double2(0.0, 0.0);
    rr = m.x;
    rz = m.y;
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) {
      rr += __shfl_xor_sync(0xffffffffu, rr, o);
      rz += __shfl_xor_sync(0xffffffffu, rz, o);
    }
  };
  {
    pen = warp_sum_d(pen);
    if (lane == 0) sDot[wid] = pen;  // (the element products come after the next CTA barrier)
    __syncthreads();
    const double e = wid == 0 ? warp_sum_d(lane < (nthreads >> 5) ? sDot[lane] : 0.0) : 0.0;
    __syncthreads();
    asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
    if (tid == 0) cluster.map_shared_rank(sEnergy, 0)[crank] = e;  // (read after the last barrier)
  }
  send_b();
  cp_async_wait<0>();  // A (the loop's first CTA barrier follows)

  const double tol = (double)a.pcg_tolerance, tol2 = tol * tol * (1.0 + 1e-14);
  double rz = 0.0, rr_last = 0.0;  // (warp 0)
  int used = 0;
  float p = 0.f;
  for (int it = 0;; it++) {
    // Warp 0 waits for the exchange and takes the step for everyone; the
    // others sleep at the CTA barrier (polling from every warp slows the
    // shared-memory pipe that the sums run through).
    if (wid == 0) {
      wait(barB, it & 1);
      double srr, srz;
      sum_b(srr, srz);
      rr_last = srr;
      used = it;
      float beta = 0.f;
      // (the root only where it can be below the tolerance) solver_kernels.cu:669
      bool stop = it >= a.pcg_iterations || dead;  // (lane 0's; after the other exchange this one ends the loop)
      if (it > 0) {
        stop |= !(srr >= tol2) && sqrt(srr) < tol;
        beta = (float)(srz / rz);
      }
      rz = srz;
      if (lane == 0) {
        *sStep = beta;
        *sStop = stop;
      }
    }
    __syncthreads();
    if (*sStop) break;
    const float betaf = *sStep;
    // ---- p = z + beta p_old: own rows, and the halo from the owners' z ----
    p = it == 0 ? z : __fmaf_rn(betaf, p, z);
    if (own) sP[t] = p;
    for (int e = tid; e < h6; e += nthreads) {
      const int h = sHalo[e / 6];
      const float zr = cluster.map_shared_rank(sZ, h >> 24)[(h & 0xffffff) * 6 + e % 6];
      sP[n6 + e] = it == 0 ? zr : __fmaf_rn(betaf, sP[n6 + e], zr);
    }
    __syncthreads();
    // ---- Ap (solver_kernels.cu:406-432): an element's lanes take its blocks
    //      in turn; combined by an xor butterfly ----
    float y = 0.f;
    if (act) {
      const int e1 = sRow[row + 1];
#pragma unroll 2
      for (int bl = sRow[row] + ks; bl < e1; bl += kSpl) {
        const float2* Ab = reinterpret_cast<const float2*>(sA + bl * 36 + c * 6);
        const float2* pv = reinterpret_cast<const float2*>(sP + sVidx[bl] * 6);
        const float2 a0 = Ab[0], a1 = Ab[1], a2 = Ab[2], p0 = pv[0], p1 = pv[1], p2 = pv[2];
        y = __fmaf_rn(a0.x, p0.x, y);
        y = __fmaf_rn(a0.y, p0.y, y);
        y = __fmaf_rn(a1.x, p1.x, y);
        y = __fmaf_rn(a1.y, p1.y, y);
        y = __fmaf_rn(a2.x, p2.x, y);
        y = __fmaf_rn(a2.y, p2.y, y);
      }
    }
#pragma unroll
    for (int o = kSpl >> 1; o > 0; o >>= 1) y += __shfl_xor_sync(0xffffffffu, y, o);
    if (own) sDot[t] = (double)p * y;
    __syncthreads();
    if (wid == 0) {
      double v = 0.0;
      for (int k = lane; k < n6; k += 32) v += sDot[k];
      v = warp_sum_d(v);
      if (lane < C) send_f64(remote(smem_addr(msgA + crank), lane), v, remote(barA, lane));
      if (lane == 0) bar_arrive_expect(barA, (unsigned)C * 8u);
      wait(barA, it & 1);
      const double pAp = sum_a();
      if (lane == 0) {
        *sStep = (float)(rz / pAp);
        *sStop = fabs(pAp) < 1e-12;  // solver_kernels.cu:647-653
      }
    }
    __syncthreads();
    if (*sStop) break;
    const float af = *sStep;
    x = __fmaf_rn(af, p, x);
    r = own ? __fmaf_rn(-af, y, r) : 0.f;
    send_b();
  }
  cluster.sync();  // no CTA leaves while another may still send to it or read it

  // ---- epilogue ----
  if (own && !isfinite(x)) atomicOr(err, kErrNonFinite);
  if (a.delta_x) {
    if (own) a.delta_x[r0 * 6 + t] = x;
  } else {
    if (own) sP[t] = x;
    __syncthreads();
    for (int i = tid; i < nrows; i += nthreads) {
      const int node = r0 + i;
      DQ T0;
      T0.r = sTn[3 * i];
      T0.d = sTn[3 * i + 1];
      const float4 xp = sTn[3 * i + 2];
      DQ Tn = twist_update(T0, sP + i * 6, pd.max_rot, pd.max_trans, pd.update_scale);
      store_dq(a.transforms + node, Tn);
      store_dq(w.plain + node, dq_centered(Tn, f3(xp.x, xp.y, xp.z)));
    }
  }
  if (crank == 0 && tid == 0) {
    double e = 0.0;
    for (int k = 0; k < C; k++) e += sEnergy[k];
    st->energy[P.slot] = e;
    if (!isfinite(e)) atomicOr(err, kErrNonFinite);
    st->pcg_iters[P.slot] = used;
    st->pcg_res[P.slot] = sqrt(rr_last);
  }
  if (dead)  // messages that were not waited for (who never gave up has received all of its own)
    for (const long long t0 = clock64(); clock64() - t0 < kClDrainCycles;) {
    }
}

// Lanes per row element: four while that takes at most 24 warps per CTA, else
// two, else one (up to 32 warps).  More lanes shorten the row sums, more warps
// lengthen the CTA barriers.
int pick_spl(int rows_max) { return rows_max <= 24 ? 4 : rows_max <= 48 ? 2 : 1; }
int pick_threads(int rows_max) {
  const int per = 32 / (6 * pick_spl(rows_max));
  return 32 * ((rows_max + per - 1) / per);
}

using Kernel = void (*)(CluArgs);
Kernel kernel_of(int rows_max) {
  const int spl = pick_spl(rows_max);
  return spl == 4 ? pcg_cluster_kernel<4> : spl == 2 ? pcg_cluster_kernel<2> : pcg_cluster_kernel<1>;
}

cudaError_t config_kernel(int C, int rows_max, int smem) {
  // the device's opt-in maximum, not this plan's size: another handle's plan
  // (with more shared memory) launches the same kernel
  int dev = 0, optin = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  if (smem > optin) return cudaErrorInvalidValue;
  cudaError_t e = cudaFuncSetAttribute(kernel_of(rows_max), cudaFuncAttributeMaxDynamicSharedMemorySize, optin);
  if (e != cudaSuccess) return e;
  if (C > 8) e = cudaFuncSetAttribute(kernel_of(rows_max), cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  return e;
}

// (attr: two; the second lets it start as launch_next does)
cudaLaunchConfig_t launch_config(int C, int threads, int smem, cudaLaunchAttribute* attr, cudaStream_t s) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(C);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = C;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  return cfg;
}

}  // namespace

// Rows per CTA that the kernel can hold: five per warp.
int pcg_cluster_max_rows() { return 160; }

int pcg_cluster_smem_bytes(int blk_max, int rows_max, int nhalo_max, int C) {
  return clu_layout(blk_max, rows_max, nhalo_max, pick_threads(rows_max), C).total;
}

int pcg_cluster_max_active(int C, int rows_max, int smem) {
  const int threads = pick_threads(rows_max);
  if (config_kernel(C, rows_max, smem) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  cudaLaunchAttribute attr[2];
  const cudaLaunchConfig_t cfg = launch_config(C, threads, smem, attr, nullptr);
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, kernel_of(rows_max), &cfg) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return n;
}

cudaError_t launch_pcg_cluster(const Work& w, const Pattern& p, const SolveArgs& a, int gn_slot, cudaStream_t s) {
  if (a.N <= 0) return cudaSuccess;
  CluArgs P;
  P.w = w;
  P.pt = p;
  P.a = a;
  P.slot = gn_slot;
  const int threads = pick_threads(p.clu_rows_max);
  cudaLaunchAttribute attr[2];
  const cudaLaunchConfig_t cfg = launch_config(p.clu_C, threads, p.clu_smem, attr, s);
  return cudaLaunchKernelEx(&cfg, kernel_of(p.clu_rows_max), P);
}

}  // namespace cf
