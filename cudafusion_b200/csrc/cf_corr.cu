// cf_corr.cu — projective correspondence search (point-to-plane ICP pairs).
//
// Restates DynamicFusionPipeline::find_correspondences
// (include/fusion_app.h:1791-1845): compute_pixel_knn_kernel
// (kernels/tsdf_kernels.cu:573-604) then find_correspondences_kernel
// (kernels/tsdf_kernels.cu:386-563).  Per live pixel: reject a missing live
// vertex or normal, project the vertex into the depth camera, reject a
// projection behind the camera or off the image and a normal seen edge-on,
// then scan the (2r+1)^2 depth pixels around the projection in row-major
// order.  A candidate is skipped without depth, farther than the Euclidean cap
// max(3 d, d + 0.03), without a normal, with |n_live . n_dst| below the angle
// threshold, or with a point-to-plane distance above d or not below the best
// so far; otherwise it becomes the best.  The pair stores the live vertex, the
// best candidate and its normal mapped back to the world, the squared mean of
// the three confidences and the pixel's node ids/weights.
//
// Arithmetic.  Every three-term product sum is accumulated left to right by
// fused multiply-adds, fmaf(a.z, b.z, fmaf(a.y, b.y, a.x * b.x)); every other
// operation is a single IEEE-rounded add, multiply, divide or square root.  The
// CPU oracle performs the same operations, so the two agree bit for bit.  (The
// reference is built with --use_fast_math, whose divide and square root are
// approximations; its results agree with these to rounding.)
//
// Launches per frame:
//  corr_prep_kernel    per depth pixel one 24-byte candidate record: the
//                      unprojected point and the normal.  The two skip cases
//                      are folded into z (0: no depth; -1: no normal) with x, y
//                      and the normal's x so large that the record's
//                      point-to-plane distance is +inf.  Per block of 16 x 16
//                      pixels the box of its real points and its longest normal.
//                      The reference recomputes the unprojection, two
//                      divisions, for every (pixel, candidate) pair.
//                      The live pixels' camera-frame points, projections and
//                      rejections are made here as well.
//  corr_search_kernel  (wide windows) finds, for each pixel and chunk of image
//                      rows, the runs of kGroup candidates that can hold the
//                      winner (below).
//  corr_exact_kernel   all candidates in the reference's arithmetic: every chunk
//                      where windows are narrower or an angle threshold is
//                      given, else those that the search leaves to it.
//  corr_merge_kernel   evaluates the runs with the reference's arithmetic,
//                      takes the least distance (of equal ones the first
//                      candidate in row-major order: the strict-less rule of
//                      one sequential scan, as no distance can be NaN: every
//                      value entering the search is finite and at most 1e18 in
//                      magnitude, so no product sum overflows), and writes the
//                      record.  A pixel or frame holding any other value is
//                      rescanned sequentially with the reference's rule as it
//                      stands (a NaN distance is accepted).  Small windows it
//                      scans itself, without a scan before.
//
// The search.  A CTA takes 32 x 16 pixels, a warp 8 x 8 of them, a lane two.
// The warp scans the union of its pixels' windows.  With o the centre of the
// CTA's points, w = v - o, and per candidate c = n . (p - o), made once per CTA as
// the records are staged, n . (v - p) is n . w - c: a contraction, done on the
// tensor cores eight candidates by 16 pixels at a time, with n, w and c as sums
// of two or three halfs (16 products per value).  It differs from the
// reference's rounded distance by at most
//   eps = u N (25 max |w| + 20 max |p - o|)       (u = 2^-24, N the longest normal):
// 4 u (both terms) for the reference's roundings, u and 4 u for those of w and
// c in FP32, 8 u for what two halfs leave of n and w, and 11 u for the tensor
// core's sum.  That sum cuts its 16 products, exact by themselves, to a common unit
// two bits below FP32's last place of the largest one's exponent, then the total
// to FP32 (1 + 15 x 2^-25 is short of 2^-23 x 3/4, 1 + 15 x 2^-26 is 1, wherever the 1
// stands and in either sign): less than u / 2 for each of 14 smaller products and 2 u of
// the total, 9 u in all; over 2.5 x 10^7 random sums no more was found.  eps is
// some 3e-7 m.  Per run of up to kGroup
// candidates of a row a lane takes the least |n . w - c| and keeps of these the
// least L1, the second L2 (with their runs) and the third L3, each less eps.  The
// winner's distance is at most U = min(L1 + 2 eps), so it is in a run of L <= U:
// usually one, and if a chunk's L3 <= U the merge scans the chunk's rows for that
// pixel, the CTA's warps taking such pixels from a list.
//
// Surfaces of equal distances (a plane, a cylinder along its axis) put the third
// run of most pixels in reach, and such a scan per pixel costs twelve times the
// search.  So a CTA counts these pixels, first after a few rows of its middle, and
// past kCsTies threads with them leaves the chunk to the exact scan.  It also does
// where the boxes do not prove every candidate within the Euclidean cap, or the
// values' ranges leave no room in halfs.
//
// What bounds the search: the legacy tensor path (8.2 clocks per step and SM
// quarter) and instruction issue (two lane-minima per step and 16 pixels, the
// masks of the windows' edges); the exact scan: instruction issue (6.5 per pixel
// and candidate) and shared memory's data path.  Measured on B200, us per call, in
// brackets a thread per two pixels with the reference's arithmetic throughout:
//                        noisy       plane       plane, third runs scanned per pixel
//   640 x 480 r 50       566 (1771)  1126 (1104)   4272
//             r 36       384 (1027)   694  (645)   2498
//             r 28       423  (692)   403  (441)   1688
//             r 20       269  (430)   258  (286)   1123
//             r 50 angle 1434 (2594) 1404 (1645)   5453
//   320 x 240 r 20       100  (152)    97  (103)    508
//   160 x 120 r 20        62   (72)    60   (57)    512
#include <cfloat>
#include <climits>
#include <cmath>

#include <cuda_fp16.h>

#include "cf_device.cuh"
#include "cf_internal.h"

namespace cf {

namespace {

constexpr int kCsTx = 32;  // pixels of a CTA
constexpr int kCsTy = 16;
constexpr int kCsThreads = 256;
constexpr int kCsSmem = 72 * 1024;  // one band of records; 3 CTAs per SM with the 1 KB reserve each
constexpr int kCsCtasPerSm = 3;
constexpr int kExSmem = 104 * 1024;  // the exact scan's; 2 CTAs per SM, whose 128 registers a lane's four pixels need
constexpr int kExCtasPerSm = 2;
constexpr int kCsTieRows = 4;  // rows after which ties are looked for first
// Threads of a CTA (two pixels each; of those that have any, as many in
// proportion) with ties beyond which its chunk is scanned exactly.  640 x 480,
// radius 50: a noise-free wavy surface 700 us with 64, 633 with 112 (one chunk alone
// takes the exact scan 77); a tilted plane in FP32 depth 1202 and 1263, radius 36 a
// plane 699 and 739.
constexpr int kCsTies = 64;
constexpr int kCsBlock = 16;  // side of the blocks whose boxes are known
constexpr int kGroup = 128;   // candidates of a run at most
constexpr int kSlab = 768;    // columns staged at a time at most
constexpr int kPad = 8;       // and the columns past them that a step may read
constexpr float kFarS = 3e5f;  // (scaled) distance of what is not there, above every real one
// Largest radius whose windows the merge scans itself, a lane per pixel: 640 x
// 480 takes 79 us at radius 5 that way and 127 at 8, 103 and 125 with the exact scan
// before it.  With an angle threshold the exact scan has more to do per candidate,
// the merge waits for its loads as before: at 8 136 and 147, past the cap 136 and 170.
constexpr int kCsDirect = 7, kCsDirectAngle = 8;
// Pixels times candidates past which the search goes before the exact scan: its
// fixed costs, and those of a surface that it leaves to the exact scan, weigh on
// narrower windows.  640 x 480 at radius 20 (5.2e8): 227 us with the search, 269
// without, on a plane 357 and 258; at 28 (1e9) 312 and 423, 522 and 402; at 36
// (1.6e9) 384 and 590, 694 and 571.
constexpr double kCsFilter = 1.2e9;
constexpr float kCsNone = 1e30f;  // distance of what is not there
constexpr float kU = 5.9604645e-8f;  // 2^-24
constexpr float kCsBig = 1e18f;  // squares and three-term sums of such values stay finite in FP32
constexpr float kCsFar = 1e30f;  // x, y and normal x of a skip record: its distance overflows to +inf

struct CorrConsts {
  float fx, fy, cx, cy;
  int W, H, P, radius, chunks;
  float cw[12];  // T_cam_world, rows 0..2
  float wc[12];  // T_world_cam, rows 0..2
  float dist_thr, angle_thr, view_thr;
  float cap, s_max, normal_eps, view_eps;
};

struct KnnSrc {
  const int* pixel_knn;
  const float* pixel_knn_w;
  const int* hit;
  const int* voxel_knn;
  const float* voxel_knn_w;
  long long num_voxels;
  int* pixel_knn_out;
  float* pixel_knn_w_out;
};

__device__ __forceinline__ float cs_dot(float ax, float ay, float az, float bx, float by, float bz) {
  return fmaf(az, bz, fmaf(ay, by, __fmul_rn(ax, bx)));
}

// Mat4::transform_point / transform_normal (include/types.h:37-57) on rows
// r[0..11] = M[0][0..3], M[1][0..3], M[2][0..3].
__device__ __forceinline__ float3 cs_point(const float* r, float x, float y, float z) {
  return make_float3(__fadd_rn(cs_dot(r[0], r[1], r[2], x, y, z), r[3]),
                     __fadd_rn(cs_dot(r[4], r[5], r[6], x, y, z), r[7]),
                     __fadd_rn(cs_dot(r[8], r[9], r[10], x, y, z), r[11]));
}
__device__ __forceinline__ float3 cs_normal(const float* r, float x, float y, float z) {
  return make_float3(cs_dot(r[0], r[1], r[2], x, y, z), cs_dot(r[4], r[5], r[6], x, y, z),
                     cs_dot(r[8], r[9], r[10], x, y, z));
}
// normalize3, include/se3_math.cuh:28-33.
__device__ __forceinline__ float3 cs_normalize(float3 v) {
  const float n = __fsqrt_rn(cs_dot(v.x, v.y, v.z, v.x, v.y, v.z));
  return n > 1e-9f ? make_float3(__fdiv_rn(v.x, n), __fdiv_rn(v.y, n), __fdiv_rn(v.z, n)) : v;
}
__device__ __forceinline__ float cs_norm(float x, float y, float z) { return __fsqrt_rn(cs_dot(x, y, z, x, y, z)); }
__device__ __forceinline__ bool cs_small(float v) { return fabsf(v) <= kCsBig; }  // false for NaN and inf

// The per-pixel part of find_correspondences_kernel before the window scan.
struct CsPixel {
  int code;      // debug counter when the pixel stops here, else -1
  bool search;   // the window is scanned
  bool special;  // the scan must run sequentially with the reference's NaN behaviour
  int pu, pv;
  float3 vl, vc, nc;
  float view_cos;
};

__device__ __forceinline__ CsPixel cs_pixel(const CorrConsts& k, const float* lv,
                                            const float* ln, int px) {
  CsPixel p;
  p.code = -1;
  p.search = false;
  p.special = false;
  p.pu = p.pv = 0;
  p.vl = make_float3(lv[3 * px], lv[3 * px + 1], lv[3 * px + 2]);
  p.vc = p.nc = make_float3(0.f, 0.f, 0.f);
  p.view_cos = 0.f;
  const float3 nl = make_float3(ln[3 * px], ln[3 * px + 1], ln[3 * px + 2]);
  if (cs_norm(p.vl.x, p.vl.y, p.vl.z) < 1e-6f || cs_norm(nl.x, nl.y, nl.z) < 1e-6f) {
    p.code = 0;
    return p;
  }
  p.vc = cs_point(k.cw, p.vl.x, p.vl.y, p.vl.z);
  if (p.vc.z <= 0.f) {
    p.code = 1;
    return p;
  }
  // CameraIntrinsics::project, include/types.h:152-155
  p.pu = __float2int_rn(__fadd_rn(__fdiv_rn(__fmul_rn(k.fx, p.vc.x), p.vc.z), k.cx));
  p.pv = __float2int_rn(__fadd_rn(__fdiv_rn(__fmul_rn(k.fy, p.vc.y), p.vc.z), k.cy));
  if (p.pu < 0 || p.pu >= k.W || p.pv < 0 || p.pv >= k.H) {
    p.code = 1;
    return p;
  }
  p.nc = cs_normal(k.cw, nl.x, nl.y, nl.z);
  const float3 vd = cs_normalize(make_float3(-p.vc.x, -p.vc.y, -p.vc.z));
  p.view_cos = fabsf(cs_dot(p.nc.x, p.nc.y, p.nc.z, vd.x, vd.y, vd.z));
  if (p.view_cos < k.view_thr) {
    p.code = 4;
    return p;
  }
  p.search = true;
  p.special = !(cs_small(p.vc.x) && cs_small(p.vc.y) && cs_small(p.vc.z) && cs_small(p.nc.x) && cs_small(p.nc.y) &&
                cs_small(p.nc.z));
  return p;
}

// A pixel's record: its camera-frame point and projection's column, its normal
// and view cosine, and its projection's row, with bit 30 for a special one, or
// -1 - the counter at which it stopped.
struct CsPix {
  float4* __restrict__ v;
  float4* __restrict__ n;
  int* __restrict__ row;
};
constexpr int kCsSpecial = 1 << 30;
__device__ __forceinline__ CsPixel cs_load_pixel(const CsPix& x, int px) {
  const int row = x.row[px];
  const float4 v = x.v[px], n = x.n[px];
  CsPixel p;
  p.search = row >= 0;
  p.code = row >= 0 ? -1 : -1 - row;
  p.special = row >= 0 && (row & kCsSpecial) != 0;
  p.pu = __float_as_int(v.w);
  p.pv = row & (kCsSpecial - 1);
  p.vl = make_float3(0.f, 0.f, 0.f);  // (the merge reads it when it is needed)
  p.vc = make_float3(v.x, v.y, v.z);
  p.nc = make_float3(n.x, n.y, n.z);
  p.view_cos = n.w;
  return p;
}

__device__ __forceinline__ float cs_warp_max(float v) {
  float d;
  asm("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(d) : "f"(v));
  return d;
}

// What is known of a block of 16 x 16 pixels.  Maxima throughout: of the
// depth's real points -x, -y, -z, |n|^2, x, y, z (-inf: none; |n|^2: 0), and of
// the live pixels that are scanned -pu, pu, -pv, pv (kCsOff: none) and their
// points' -x, -y, -z, x, y, z.
struct CsBox {
  float d[8];  // (d[7] unused)
  int p[4];
  float v[6];
  float pad[2];
};
static_assert(sizeof(CsBox) == 80, "whole 16-byte words");
constexpr int kCsOff = -(1 << 30);

// One thread per pixel: the depth's candidate record, the live pixel's record,
// and the block's box.
__global__ void __launch_bounds__(kCsBlock* kCsBlock)
    corr_prep_kernel(const CorrConsts k, const float* depth, const float* dn,
                     const float* lv, const float* ln, float4* __restrict__ A,
                     float2* __restrict__ B, const CsPix pix, CsBox* __restrict__ box, int* __restrict__ flag,
                     int* __restrict__ todo, int* __restrict__ num_valid, int* __restrict__ stats) {
  after_previous();
  __shared__ float s_f[kCsBlock * kCsBlock / 32][13];
  __shared__ int s_i[kCsBlock * kCsBlock / 32][4];
  const int tid = threadIdx.x;
  const int x = blockIdx.x * kCsBlock + (tid & (kCsBlock - 1)), y = blockIdx.y * kCsBlock + tid / kCsBlock;
  if (blockIdx.x == 0 && blockIdx.y == 0) {  // (counted by the merge, and by the search)
    if (tid == 0) *num_valid = *todo = 0;
    if (stats && tid < 6) stats[tid] = 0;
  }
  const float none = -INFINITY;
  float f[13] = {none, none, none, 0.f, none, none, none, none, none, none, none, none, none};
  int q[4] = {kCsOff, kCsOff, kCsOff, kCsOff};
  if (x < k.W && y < k.H) {
    const int i = y * k.W + x;
    const float d = depth[i];
    float4 a = make_float4(kCsFar, kCsFar, 0.f, kCsFar);
    float2 b = make_float2(0.f, 0.f);
    if (!(d <= 0.f)) {
      const float nx = dn[3 * i], ny = dn[3 * i + 1], nz = dn[3 * i + 2];
      if (cs_norm(nx, ny, nz) < 1e-6f) {
        a.z = -1.f;
      } else {
        // CameraIntrinsics::unproject, include/types.h:157-161
        a.x = __fdiv_rn(__fmul_rn(d, __fsub_rn((float)x, k.cx)), k.fx);
        a.y = __fdiv_rn(__fmul_rn(d, __fsub_rn((float)y, k.cy)), k.fy);
        a.z = d;
        a.w = nx;
        b = make_float2(ny, nz);
        if (!(cs_small(a.x) && cs_small(a.y) && cs_small(d) && cs_small(nx) && cs_small(ny) && cs_small(nz)))
          atomicOr(flag, 1);
        f[0] = -a.x; f[1] = -a.y; f[2] = -a.z;
        f[3] = nx * nx + ny * ny + nz * nz;
        f[4] = a.x; f[5] = a.y; f[6] = a.z;
      }
    }
    A[i] = a;
    B[i] = b;
    const CsPixel p = cs_pixel(k, lv, ln, i);
    pix.row[i] = p.search ? p.pv | (p.special ? kCsSpecial : 0) : -1 - p.code;
    pix.v[i] = make_float4(p.vc.x, p.vc.y, p.vc.z, __int_as_float(p.pu));
    pix.n[i] = make_float4(p.nc.x, p.nc.y, p.nc.z, p.view_cos);
    if (p.search && !p.special) {
      q[0] = -p.pu; q[1] = p.pu; q[2] = -p.pv; q[3] = p.pv;
      f[7] = -p.vc.x; f[8] = -p.vc.y; f[9] = -p.vc.z;
      f[10] = p.vc.x; f[11] = p.vc.y; f[12] = p.vc.z;
    }
  }
#pragma unroll
  for (int c = 0; c < 13; ++c) f[c] = cs_warp_max(f[c]);
#pragma unroll
  for (int c = 0; c < 4; ++c) q[c] = __reduce_max_sync(0xffffffffu, q[c]);
  if ((tid & 31) == 0) {
#pragma unroll
    for (int c = 0; c < 13; ++c) s_f[tid >> 5][c] = f[c];
#pragma unroll
    for (int c = 0; c < 4; ++c) s_i[tid >> 5][c] = q[c];
  }
  __syncthreads();
  CsBox* o = box + (size_t)blockIdx.y * gridDim.x + blockIdx.x;
  if (tid < 13) {
    float m = s_f[0][tid];
#pragma unroll
    for (int w = 1; w < kCsBlock * kCsBlock / 32; ++w) m = fmaxf(m, s_f[w][tid]);
    (tid < 7 ? o->d[tid] : o->v[tid - 7]) = m;
  } else if (tid < 17) {
    int m = s_i[0][tid - 13];
#pragma unroll
    for (int w = 1; w < kCsBlock * kCsBlock / 32; ++w) m = max(m, s_i[w][tid - 13]);
    o->p[tid - 13] = m;
  }
}

// A candidate's point-to-plane distance, +inf where the reference would skip
// it (finite values only).  A skip record's far-away point and huge normal
// make its distance +inf by themselves.  kAngle: apply the angle threshold.
// kCap: apply the Euclidean cap (left out where every candidate is within it).
template <bool kAngle, bool kCap = true>
__device__ __forceinline__ float cs_pd(const float3& v, const float3& n, const float4& a, const float2& b,
                                       const CorrConsts& k) {
  const float ex = __fsub_rn(v.x, a.x), ey = __fsub_rn(v.y, a.y), ez = __fsub_rn(v.z, a.z);
  float pd = fabsf(cs_dot(a.w, b.x, b.y, ex, ey, ez));
  if (kCap) pd = cs_dot(ex, ey, ez, ex, ey, ez) <= k.s_max ? pd : INFINITY;
  if (kAngle) pd = fabsf(cs_dot(n.x, n.y, n.z, a.w, b.x, b.y)) < k.angle_thr ? INFINITY : pd;
  return pd;
}

// One of a lane's two pixels.
struct CsLane {
  int pv;  // its projection's row; off the image when it is not scanned
  float L1, L2, L3;
  int g1, g2;  // the runs of L1 and L2: their first pixel
};

__device__ __forceinline__ float cs_min_abs(float a, float b, float c) {
  float d;
  asm("min.abs.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}

// A run's least value into the pixel's three least.
__device__ __forceinline__ void cs_track(CsLane& q, float m, float eps, int g) {
  const float L = m - eps;
  const bool c1 = L < q.L1, c2 = L < q.L2;
  q.L3 = fminf(q.L3, fmaxf(q.L2, L));
  q.L2 = fminf(q.L2, fmaxf(q.L1, L));
  q.g2 = c1 ? q.g1 : c2 ? g : q.g2;
  q.L1 = fminf(q.L1, L);
  q.g1 = c1 ? g : q.g1;
}

// D = A B of one tensor-core step: 16 pixels by 8 candidates over 16 products.
__device__ __forceinline__ void cs_mma(float (&d)[4], const unsigned (&a)[4], unsigned b0, unsigned b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.f));
}
__device__ __forceinline__ unsigned cs_h2(float x, float y) {  // two halfs, x in the lower one
  const __half2 h = __floats2half2_rn(x, y);
  return reinterpret_cast<const unsigned&>(h);
}
// x as a sum of halfs: the nearest, and the nearest to what is left
__device__ __forceinline__ float cs_hi(float x) { return __half2float(__float2half_rn(x)); }

// The 16 products that make n . w - c: the high and low halfs of n and w
// against each other, and c in three halfs against 4.  A candidate's halfs in
// the order in which lanes read them: lane t of a quad those of the products
// 2t, 2t + 1, 2t + 8, 2t + 9.
//   0..2  w_hi n_hi    3..5  w_lo n_hi    6..8  w_hi n_lo    9..11  w_lo n_lo
//   12..14  4 c'       (c' = -c / 4)      15  0
__device__ __forceinline__ void cs_store_mma(float4* o, float nx, float ny, float nz, float mc) {
  const float hx = cs_hi(nx), hy = cs_hi(ny), hz = cs_hi(nz), lx = nx - hx, ly = ny - hy, lz = nz - hz;
  const float c1 = cs_hi(mc), c2 = cs_hi(mc - c1), c3 = mc - c1 - c2;
  o[0] = make_float4(__uint_as_float(cs_h2(hx, hy)), __uint_as_float(cs_h2(lz, lx)), __uint_as_float(cs_h2(hz, hx)),
                     __uint_as_float(cs_h2(ly, lz)));
  o[1] = make_float4(__uint_as_float(cs_h2(hy, hz)), __uint_as_float(cs_h2(c1, c2)), __uint_as_float(cs_h2(lx, ly)),
                     __uint_as_float(cs_h2(c3, 0.f)));
}
// Lane t's part of a pixel (scaled w): products 2t, 2t + 1 and 2t + 8, 2t + 9.
__device__ __forceinline__ void cs_pixel_mma(float wx, float wy, float wz, int t, unsigned& k0, unsigned& k1) {
  const float hx = cs_hi(wx), hy = cs_hi(wy), hz = cs_hi(wz), lx = wx - hx, ly = wy - hy, lz = wz - hz;
  k0 = t == 0 ? cs_h2(hx, hy) : t == 1 ? cs_h2(hz, lx) : t == 2 ? cs_h2(ly, lz) : cs_h2(hx, hy);
  k1 = t == 0 ? cs_h2(hz, lx) : t == 1 ? cs_h2(ly, lz) : t == 2 ? cs_h2(4.f, 4.f) : cs_h2(4.f, 0.f);
}

// Eight candidates against the warp's 64 pixels, four 16-pixel tiles: lane
// 4 g + t has the values of the pixels g and g + 8 of each tile at the
// candidates 2 t and 2 t + 1.  kLeft, kRight: some windows begin, end here
// (first: their first columns, not clipped: outside the image nothing is there).
template <bool kLeft, bool kRight>
__device__ __forceinline__ void cs_step_mma(const uint2 b, const unsigned (&af)[4][4], const int (&first)[8], int col,
                                            int far, float (&m)[8]) {
  float d[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i) cs_mma(d[i], af[i], b.x, b.y);
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const float x = d[i >> 1][2 * (i & 1)], y = d[i >> 1][2 * (i & 1) + 1];
    if (!kLeft && !kRight) {
      m[i] = cs_min_abs(m[i], x, y);
    } else {
      if ((!kLeft || first[i] <= col) && (!kRight || first[i] >= far)) m[i] = fminf(m[i], fabsf(x));
      if ((!kLeft || first[i] <= col + 1) && (!kRight || first[i] >= far + 1)) m[i] = fminf(m[i], fabsf(y));
    }
  }
}

// The band's candidates (32 bytes each, as cs_store_mma writes them) against
// the warp's pixels, a run of a row at a time: the steps on its left that some
// windows do not reach, those that all hold, and the rest.  At the end of a run
// the quad's lanes exchange their values so that lane t has its own pixels,
// those of tile t.
__device__ __forceinline__ void cs_scan_mma(const float4* sm, int wu, int xs, int yb, int ca, int cb, int ia, int ib,
                                            int ya, int yz, const unsigned (&af)[4][4], const int (&first)[8], CsLane& q0,
                                            CsLane& q1, float eps, const CorrConsts& k) {
  const unsigned r = (unsigned)k.radius;
  const int lane = threadIdx.x & 31, t = lane & 3, t2 = 2 * t;
  for (int yy = ya; yy <= yz; ++yy) {
    const uint2* row = reinterpret_cast<const uint2*>(sm + (size_t)(yy - yb) * 2 * wu) + lane - 4 * xs;
    const bool in0 = (unsigned)(yy - q0.pv) + r <= 2 * r, in1 = (unsigned)(yy - q1.pv) + r <= 2 * r;
    const int base = yy * k.W;
    for (int g = ca; g <= cb; g += kGroup) {
      float m[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) m[i] = kFarS;
      const int e = min(cb, g + kGroup - 1);
      int c = g;
#pragma unroll 1
      for (; c <= e && c < ia; c += 8) {
        if (c + 7 <= ib) cs_step_mma<true, false>(row[4 * c], af, first, c + t2, 0, m);
        else cs_step_mma<true, true>(row[4 * c], af, first, c + t2, c + t2 - 2 * (int)r, m);
      }
      const int n = (min(e, ib) - c + 1) >> 3;  // steps that all windows hold
      const uint2* at = row + 4 * c;
#pragma unroll 4
      for (int j = 0; j < n; ++j, at += 32) cs_step_mma<false, false>(*at, af, first, 0, 0, m);
      c += 8 * max(n, 0);
#pragma unroll 1
      for (; c <= e; c += 8) cs_step_mma<false, true>(row[4 * c], af, first, 0, c + t2 - 2 * (int)r, m);
      // lane t keeps tile t's two pixels
      float s[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float send = t & 2 ? m[i] : m[4 + i], keep = t & 2 ? m[4 + i] : m[i];
        s[i] = fminf(keep, __shfl_xor_sync(0xffffffffu, send, 2));
      }
      float v[2];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const float send = t & 1 ? s[i] : s[2 + i], keep = t & 1 ? s[2 + i] : s[i];
        v[i] = fminf(keep, __shfl_xor_sync(0xffffffffu, send, 1));
      }
      // a window that does not reach this row holds nothing of the run
      cs_track(q0, in0 ? v[0] : kFarS, eps, base + g);
      cs_track(q1, in1 ? v[1] : kFarS, eps, base + g);
    }
  }
}

// find_correspondences_kernel's loop as it stands (kernels/tsdf_kernels.cu:470-524),
// for pixels or frames whose values could make a distance NaN.
__device__ __forceinline__ int cs_rescan(const CorrConsts& k, const CsPixel& p, const float4* A,
                                         const float2* B, bool& saw_depth) {
  const int r = k.radius;
  const int x0 = max(0, p.pu - r), x1 = min(k.W - 1, p.pu + r);
  const int y0 = max(0, p.pv - r), y1 = min(k.H - 1, p.pv + r);
  float best = k.dist_thr;
  int bi = -1;
  for (int yy = y0; yy <= y1; ++yy)
    for (int xx = x0; xx <= x1; ++xx) {
      const float4 a = A[yy * k.W + xx];
      if (a.z == 0.f) continue;
      saw_depth = true;
      if (a.z < 0.f) continue;
      const float ex = __fsub_rn(p.vc.x, a.x), ey = __fsub_rn(p.vc.y, a.y), ez = __fsub_rn(p.vc.z, a.z);
      if (cs_dot(ex, ey, ez, ex, ey, ez) > k.s_max) continue;
      const float2 b = B[yy * k.W + xx];
      if (fabsf(cs_dot(p.nc.x, p.nc.y, p.nc.z, a.w, b.x, b.y)) < k.angle_thr) continue;
      const float pd = fabsf(cs_dot(a.w, b.x, b.y, ex, ey, ez));
      if (pd > k.dist_thr || pd >= best) continue;
      best = pd;
      bi = yy * k.W + xx;
    }
  return bi;
}

// Whether the pixel's window holds any depth (no_depth vs far, for the
// debug counters of a pixel without a pair).
__device__ __forceinline__ bool cs_any_depth(const CorrConsts& k, const CsPixel& p, const float4* A) {
  const int r = k.radius;
  const int x0 = max(0, p.pu - r), x1 = min(k.W - 1, p.pu + r);
  const int y0 = max(0, p.pv - r), y1 = min(k.H - 1, p.pv + r);
  for (int yy = y0; yy <= y1; ++yy)
    for (int xx = x0; xx <= x1; ++xx)
      if (A[yy * k.W + xx].z != 0.f) return true;
  return false;
}

// Writes pixel px's record from its winner bi (-1: none) and adds the
// pixel to the valid count and to its debug counter (code, -1: none), both
// reduced per warp first.  Called by every thread of the warp, whose lanes
// hold consecutive pixels (the in-image ones a prefix): each lane's 19-word
// record goes to the warp's staging area (kCsRecWords words per lane, in
// shared memory), and the warp writes its records' words out in order, 32
// consecutive words per store.
constexpr int kCsRecWords = (int)(sizeof(cf_correspondence) / 4);
static_assert(sizeof(cf_correspondence) == 4 * kCsRecWords, "a record is whole words");
__device__ __forceinline__ void cs_emit(const CorrConsts& k, const CsPixel& p, bool inimg, int px, int bi, int code,
                                        const float4* A, const float2* B,
                                        const KnnSrc& knn, cf_correspondence* __restrict__ out,
                                        int* __restrict__ num_valid, int* __restrict__ stats, int lane,
                                        float* __restrict__ stage) {
  const bool valid = bi >= 0;
  if (inimg) {
    int ids[CF_K_NEIGHBORS];
    float ws[CF_K_NEIGHBORS];
#pragma unroll
    for (int j = 0; j < CF_K_NEIGHBORS; ++j) {
      ids[j] = -1;
      ws[j] = 0.f;
    }
    if (knn.pixel_knn) {
      if (valid) {
#pragma unroll
        for (int j = 0; j < CF_K_NEIGHBORS; ++j) {
          ids[j] = knn.pixel_knn[(size_t)px * CF_K_NEIGHBORS + j];
          ws[j] = knn.pixel_knn_w[(size_t)px * CF_K_NEIGHBORS + j];
        }
      }
    } else if (knn.hit) {
      const int v = knn.hit[px];
      if (v >= 0 && (long long)v < knn.num_voxels) {
#pragma unroll
        for (int j = 0; j < CF_K_NEIGHBORS; ++j) {
          ids[j] = knn.voxel_knn[(size_t)v * CF_K_NEIGHBORS + j];
          ws[j] = knn.voxel_knn_w[(size_t)v * CF_K_NEIGHBORS + j];
        }
      }
      if (knn.pixel_knn_out) {
#pragma unroll
        for (int j = 0; j < CF_K_NEIGHBORS; ++j) {
          knn.pixel_knn_out[(size_t)px * CF_K_NEIGHBORS + j] = ids[j];
          knn.pixel_knn_w_out[(size_t)px * CF_K_NEIGHBORS + j] = ws[j];
        }
      }
    }
    float3 src = make_float3(0.f, 0.f, 0.f), dst = src, nrm = src;
    float weight = 0.f;
    if (valid) {
      const float4 a = A[bi];
      const float2 b = B[bi];
      const float ex = __fsub_rn(p.vc.x, a.x), ey = __fsub_rn(p.vc.y, a.y), ez = __fsub_rn(p.vc.z, a.z);
      const float euclid = __fsqrt_rn(cs_dot(ex, ey, ez, ex, ey, ez));
      const float cosv = fabsf(cs_dot(p.nc.x, p.nc.y, p.nc.z, a.w, b.x, b.y));
      src = p.vl;
      dst = cs_point(k.wc, a.x, a.y, a.z);
      nrm = cs_normalize(cs_normal(k.wc, a.w, b.x, b.y));
      // kernels/tsdf_kernels.cu:510-514
      const float phi_d = fmaxf(0.f, __fsub_rn(1.f, __fdiv_rn(euclid, k.cap)));
      const float phi_n = fmaxf(0.f, __fsub_rn(1.f, __fdiv_rn(__fsub_rn(1.f, cosv), k.normal_eps)));
      const float phi_v = fmaxf(0.f, __fsub_rn(1.f, __fdiv_rn(__fsub_rn(1.f, p.view_cos), k.view_eps)));
      const float c = __fdiv_rn(__fadd_rn(__fadd_rn(phi_d, phi_n), phi_v), 3.f);
      weight = __fmul_rn(c, c);
    } else {
#pragma unroll
      for (int j = 0; j < CF_K_NEIGHBORS; ++j) {
        ids[j] = -1;
        ws[j] = 0.f;
      }
    }
    float* o = stage + lane * kCsRecWords;
    o[0] = src.x; o[1] = src.y; o[2] = src.z;
    o[3] = dst.x; o[4] = dst.y; o[5] = dst.z;
    o[6] = nrm.x; o[7] = nrm.y; o[8] = nrm.z;
#pragma unroll
    for (int j = 0; j < CF_K_NEIGHBORS; ++j) {
      o[9 + j] = __int_as_float(ids[j]);
      o[13 + j] = ws[j];
    }
    o[17] = weight;
    o[18] = __int_as_float(valid ? 1 : 0);  // bool valid + 3 zero pad bytes
  }
  {
    const unsigned mi = __ballot_sync(0xffffffffu, inimg);
    const int px0 = __shfl_sync(0xffffffffu, px, 0);
    __syncwarp();
    if (mi & 1u) {
      float* dst = reinterpret_cast<float*>(out + px0);
      const int words = __popc(mi) * kCsRecWords;
      for (int w = lane; w < words; w += 32) dst[w] = stage[w];
    }
    __syncwarp();
  }
  const unsigned mv = __ballot_sync(0xffffffffu, valid);
  if (lane == 0 && mv) atomicAdd(num_valid, __popc(mv));
  if (stats) {
#pragma unroll
    for (int c = 0; c < 6; ++c) {
      const unsigned m = __ballot_sync(0xffffffffu, code == c);
      if (lane == 0 && m) atomicAdd(stats + c, __popc(m));
    }
  }
}

// What a chunk of rows leaves of a pixel: its three least values less eps
// (a: L1, L2, L3, eps) and the runs of the first two; from the exact scan the
// least distance and the first run that has it, with eps 0.
struct CsPart {
  float4* __restrict__ a;
  int2* __restrict__ g;
  int2* __restrict__ rows;  // per tile of pixels: its first row, and the rows of a chunk
  int* __restrict__ todo;   // the exact scan's share: how many, then each (chunk * tiles + tile) * 2 + near
};

// The exact scan and the merge start as the kernel before them ends (their
// CTAs beside a running search cost more than the launch).
__device__ __forceinline__ void cs_after_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// A CTA's tile of pixels and chunk of rows: the columns and rows that its windows cover.
struct CsTile {
  int xlo, xhi, ylo, yhi, per, c0, c1;
  float v[6];  // the live pixels' box: maxima of -x, -y, -z, x, y, z
};
// False (over the CTA): nothing is scanned here.
__device__ __forceinline__ bool cs_tile(const CorrConsts& k, const CsBox* box, const int* flag,
                                        int tx, int ty, int chunk, CsTile& t) {
  // the pixels' boxes: the tile is two blocks
  const int r = k.radius, bpr = (k.W + kCsBlock - 1) / kCsBlock;
  const CsBox* bt = box + (size_t)ty * bpr + 2 * tx;
  const bool two = 2 * tx + 1 < bpr;
  int bx[4];
#pragma unroll
  for (int c = 0; c < 4; ++c) bx[c] = max(bt[0].p[c], two ? bt[1].p[c] : kCsOff);
  if (*flag || bx[1] < -bx[0]) return false;  // a frame scanned sequentially, or no pixel
#pragma unroll
  for (int c = 0; c < 6; ++c) t.v[c] = fmaxf(bt[0].v[c], two ? bt[1].v[c] : -INFINITY);
  t.xlo = max(0, -bx[0] - r) & ~1;
  t.xhi = min(k.W - 1, bx[1] + r);
  t.ylo = max(0, -bx[2] - r);
  t.yhi = min(k.H - 1, bx[3] + r);
  t.per = (t.yhi - t.ylo + k.chunks) / k.chunks;  // ceil(rows / chunks)
  t.c0 = t.ylo + chunk * t.per;
  t.c1 = min(t.yhi, t.c0 + t.per - 1);
  return true;
}
// The box of the chunk's real candidates (CsBox::d) and what follows from it.
struct CsReach {
  float o[3];     // the centre of the live pixels' points
  float wr, ar;   // the largest |v - o| and |p - o|
  float nn;       // the longest normal
  bool any, cap;  // a real candidate; all of them within the Euclidean cap of all pixels
};
__device__ __forceinline__ CsReach cs_reach(const CorrConsts& k, const CsBox* box, const CsTile& t) {
  __shared__ float s_d[kCsThreads / 32][7];
  const int tid = threadIdx.x, bpr = (k.W + kCsBlock - 1) / kCsBlock;
  float v[7] = {-INFINITY, -INFINITY, -INFINITY, 0.f, -INFINITY, -INFINITY, -INFINITY};
  if (t.c0 <= t.c1) {
    const int b0 = t.xlo / kCsBlock, bw = t.xhi / kCsBlock - b0 + 1, r0 = t.c0 / kCsBlock,
              bh = t.c1 / kCsBlock - r0 + 1;
    for (int i = tid; i < bw * bh; i += kCsThreads) {
      const float4* b = reinterpret_cast<const float4*>(box[(size_t)(r0 + i / bw) * bpr + b0 + i % bw].d);
      const float4 lo = b[0], hi = b[1];
      v[0] = fmaxf(v[0], lo.x);
      v[1] = fmaxf(v[1], lo.y);
      v[2] = fmaxf(v[2], lo.z);
      v[3] = fmaxf(v[3], lo.w);
      v[4] = fmaxf(v[4], hi.x);
      v[5] = fmaxf(v[5], hi.y);
      v[6] = fmaxf(v[6], hi.z);
    }
  }
#pragma unroll
  for (int c = 0; c < 7; ++c) {
    v[c] = cs_warp_max(v[c]);
    if ((tid & 31) == 0) s_d[tid >> 5][c] = v[c];
  }
  __syncthreads();
#pragma unroll
  for (int c = 0; c < 7; ++c) {
    v[c] = s_d[0][c];
#pragma unroll
    for (int w = 1; w < kCsThreads / 32; ++w) v[c] = fmaxf(v[c], s_d[w][c]);
  }
  CsReach q;
  q.any = v[4] >= -v[0];
  float ww = 0.f, aa = 0.f, dd = 0.f;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    q.o[c] = 0.5f * (t.v[3 + c] - t.v[c]);
    const float hw = fmaxf(fabsf(t.v[3 + c] - q.o[c]), fabsf(-t.v[c] - q.o[c]));
    const float ha = fmaxf(fabsf(v[4 + c] - q.o[c]), fabsf(-v[c] - q.o[c]));
    const float d = fmaxf(fabsf(t.v[3 + c] + v[c]), fabsf(v[4 + c] + t.v[c]));
    ww += hw * hw;
    aa += ha * ha;
    dd += d * d;
  }
  q.nn = sqrtf(v[3]);
  q.wr = sqrtf(ww);
  q.ar = sqrtf(aa);
  // (a relative margin of 1e-4 over the few-ulp rounding of the squared distances)
  q.cap = dd * 1.0001f <= k.s_max;
  return q;
}

__global__ void __launch_bounds__(kCsThreads, kCsCtasPerSm)
    corr_search_kernel(const CorrConsts k, const float4* A, const float2* B, const CsPix pix,
                       const CsBox* box, const int* flag, const CsPart part) {
  extern __shared__ float4 cs_smem[];
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int x = blockIdx.x * kCsTx + (wid & 3) * 8 + (lane >> 2);
  const int y0 = blockIdx.y * kCsTy + (wid >> 2) * 8 + 2 * (lane & 3), y1 = y0 + 1;
  const int chunk = blockIdx.z, r = k.radius;
  const int px0 = y0 * k.W + x, px1 = px0 + k.W;
  const int tile = blockIdx.y * gridDim.x + blockIdx.x;
  CsTile t;
  if (!cs_tile(k, box, flag, blockIdx.x, blockIdx.y, chunk, t)) return;
  if (chunk == 0 && tid == 0) part.rows[tile] = make_int2(t.ylo, t.per);
  const CsReach q = cs_reach(k, box, t);
  auto leave_to_exact = [&]() {
    if (tid == 0)
      part.todo[1 + atomicAdd(part.todo, 1)] = 2 * (chunk * (int)(gridDim.x * gridDim.y) + tile) + (q.cap ? 1 : 0);
  };
  if (q.any && !(q.cap && q.nn >= 1e-6f && q.nn <= 1e6f && q.wr + q.ar >= 1e-6f && q.wr + q.ar <= 1e6f)) {
    leave_to_exact();
    return;
  }
  CsPixel p0, p1;
  p0.search = p1.search = p0.special = p1.special = false;
  p0.pu = p1.pu = p0.pv = p1.pv = 0;
  p0.vc = p1.vc = make_float3(0.f, 0.f, 0.f);
  if (x < k.W && y0 < k.H) p0 = cs_load_pixel(pix, px0);
  if (x < k.W && y1 < k.H) p1 = cs_load_pixel(pix, px1);
  const bool on0 = p0.search && !p0.special, on1 = p1.search && !p1.special;
  // the warp's windows: the union of their columns and rows, and the columns common to all
  constexpr int kFar = 1 << 30;
  const int wul = __reduce_min_sync(0xffffffffu, min(on0 ? p0.pu : kFar, on1 ? p1.pu : kFar));
  const int wuh = __reduce_max_sync(0xffffffffu, max(on0 ? p0.pu : -kFar, on1 ? p1.pu : -kFar));
  const int wvl = __reduce_min_sync(0xffffffffu, min(on0 ? p0.pv : kFar, on1 ? p1.pv : kFar));
  const int wvh = __reduce_max_sync(0xffffffffu, max(on0 ? p0.pv : -kFar, on1 ? p1.pv : -kFar));
  // w and n up to 256 each: c then up to 2^16, a quarter of it fits a half
  const float sw = q.any ? ldexpf(1.f, 7 - ilogbf(q.wr + q.ar)) : 1.f, sn = q.any ? ldexpf(1.f, 7 - ilogbf(q.nn)) : 1.f;
  const float eps = q.any ? kU * q.nn * (25.f * q.wr + 20.f * q.ar) * (sw * sn) : 0.f;
  CsLane q0, q1;
  q0.pv = on0 ? p0.pv : -kFar;
  q1.pv = on1 ? p1.pv : -kFar;
  q0.L1 = q0.L2 = q0.L3 = q1.L1 = q1.L2 = q1.L3 = kCsNone;
  q0.g1 = q0.g2 = q1.g1 = q1.g2 = -1;
  if (q.any && t.c0 <= t.c1) {
    const bool some = wuh >= wul;
    const int most = __syncthreads_count(on0 || on1) * kCsTies / kCsThreads;
    const int ua = max(0, wul - r), ub = min(k.W - 1, wuh + r);  // the warp's columns
    const int ia = max(0, wuh - r), ib = min(k.W - 1, wul + r);  // those of every window
    unsigned af[4][4];
    int first[8];
    {
      const float3 a0 = on0 ? make_float3((p0.vc.x - q.o[0]) * sw, (p0.vc.y - q.o[1]) * sw, (p0.vc.z - q.o[2]) * sw)
                            : make_float3(0.f, 0.f, 0.f);
      const float3 a1 = on1 ? make_float3((p1.vc.x - q.o[0]) * sw, (p1.vc.y - q.o[1]) * sw, (p1.vc.z - q.o[2]) * sw)
                            : make_float3(0.f, 0.f, 0.f);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int src = (lane & 28) | i;  // the lane that holds this lane's pixels of tile i
        cs_pixel_mma(__shfl_sync(0xffffffffu, a0.x, src), __shfl_sync(0xffffffffu, a0.y, src),
                     __shfl_sync(0xffffffffu, a0.z, src), lane & 3, af[i][0], af[i][2]);
        cs_pixel_mma(__shfl_sync(0xffffffffu, a1.x, src), __shfl_sync(0xffffffffu, a1.y, src),
                     __shfl_sync(0xffffffffu, a1.z, src), lane & 3, af[i][1], af[i][3]);
        first[2 * i] = __shfl_sync(0xffffffffu, on0 ? p0.pu - r : kFar, src);
        first[2 * i + 1] = __shfl_sync(0xffffffffu, on1 ? p1.pu - r : kFar, src);
      }
    }
    // (in shared memory: registers are what the scan is short of)
    __shared__ float s_k[6];
    if (tid == 0) {
      s_k[0] = q.o[0];
      s_k[1] = q.o[1];
      s_k[2] = q.o[2];
      s_k[3] = sn;
      s_k[4] = -0.25f * sw * sn;
      s_k[5] = fminf(k.dist_thr * (sw * sn), 0.5f * kFarS);  // (past that nothing is there)
    }
    __syncthreads();
    // a third run in reach: the merge would scan the chunk's rows for the pixel
    auto tied = [&]() {
      const float reach = 2.25f * eps, thr = s_k[5];
      const bool tie = q0.L3 <= fminf(q0.L1 + reach, thr) || q1.L3 <= fminf(q1.L1 + reach, thr);
      return __syncthreads_count(tie) > most;
    };
    for (int xs = t.xlo; xs <= t.xhi; xs += kSlab) {
      const int xe = min(t.xhi, xs + kSlab - 1);
      const int wu = xe - xs + 1 + kPad;
      const int band = kCsSmem / (wu * 32);
      // The bands from the middle one on, whose rows most windows hold, and its
      // first rows alone: ties show there.
      const int n = (t.c1 - t.c0 + band) / band;
      int at = n / 2, yb = t.c0 + at * band, step = min(band, kCsTieRows);
      for (int left = n; left > 0;) {
        const int end = min(t.c1, t.c0 + at * band + band - 1);
        const int rows = min(step, end - yb + 1);
        if (tied()) {
          leave_to_exact();
          return;
        }
        for (int j = tid; j < rows * wu; j += kCsThreads) {
          const int rr = j / wu, c = j - rr * wu;
          float nx = 0.f, ny = 0.f, nz = 0.f, mc = 0.25f * kFarS * 0.8f;
          if (xs + c <= xe) {
            const int g = (yb + rr) * k.W + xs + c;
            const float4 a = A[g];
            if (a.z > 0.f) {
              const float2 b = B[g];
              nx = a.w * s_k[3];
              ny = b.x * s_k[3];
              nz = b.y * s_k[3];
              mc = s_k[4] * cs_dot(a.w, b.x, b.y, a.x - s_k[0], a.y - s_k[1], a.z - s_k[2]);
            }
          }
          cs_store_mma(cs_smem + 2 * j, nx, ny, nz, mc);
        }
        __syncthreads();
        if (some) {
          const int ca = max(xs, ua), cb = min(xe, ub), ya = max(yb, wvl - r), yz = min(yb + rows - 1, wvh + r);
          if (ca <= cb) cs_scan_mma(cs_smem, wu, xs, yb, ca, cb, ia, ib, ya, yz, af, first, q0, q1, eps, k);
        }
        yb += step;
        step = band;
        if (yb > end) {
          --left;
          if (++at == n) at = 0;
          yb = t.c0 + at * band;
        }
      }
    }
    if (tied()) {
      leave_to_exact();
      return;
    }
  }
  // back to metres (powers of two); what is not there has no value
  const float un = 1.f / (sw * sn);
  auto leave = [&](CsLane& l, int px) {
    const size_t at = (size_t)chunk * k.P + px;
    part.a[at] = make_float4(l.L1 < 0.5f * kFarS ? l.L1 * un : kCsNone, l.L2 < 0.5f * kFarS ? l.L2 * un : kCsNone,
                             l.L3 < 0.5f * kFarS ? l.L3 * un : kCsNone, eps * un);
    part.g[at] = make_int2(l.L1 < 0.5f * kFarS ? l.g1 : -1, l.L2 < 0.5f * kFarS ? l.g2 : -1);
  };
  if (on0) leave(q0, px0);
  if (on1) leave(q1, px1);
}

// ----------------------------------------------------------------------------
// exact scan
// ----------------------------------------------------------------------------
constexpr int kExPx = 4;  // a lane's pixels, one below the other

// The rows [yb, yb + rows) of the columns [xs, xe], of which the lane takes every
// second row, against the lane's pixels.
template <bool kAngle, bool kCap>
__device__ __forceinline__ void cs_scan_exact(const float4* sA, const float2* sB, int wu, int xs, int xe, int yb, int rows,
                                              int half, int lo, int hi, int il, int ih, int pl, int ph,
                                              const float3 (&v)[kExPx], const float3 (&n)[kExPx],
                                              const int (&pu)[kExPx], const int (&pv)[kExPx], float (&L)[kExPx],
                                              int (&G)[kExPx], const CorrConsts& k) {
  const int r = k.radius, ca = max(lo, xs), cb = min(hi, xe), yz = min(yb + rows - 1, ph);
  int yy = max(yb, pl);
  yy += (yy ^ half) & 1;
  for (; yy <= yz; yy += 2) {
    const float4* ra = sA + (yy - yb) * wu - xs;
    const float2* rb = sB + (yy - yb) * wu - xs;
    for (int g = ca; g <= cb; g += kGroup) {
      const int e = min(cb, g + kGroup - 1);
      float m[kExPx];
#pragma unroll
      for (int i = 0; i < kExPx; ++i) m[i] = INFINITY;
      auto edge = [&](int c) {  // a column that some of the windows hold
        const float4 a = ra[c];
        const float2 b = rb[c];
#pragma unroll
        for (int i = 0; i < kExPx; ++i) {
          const float d = cs_pd<kAngle, kCap>(v[i], n[i], a, b, k);
          m[i] = (unsigned)(c - pu[i] + r) <= 2u * r ? fminf(m[i], d) : m[i];
        }
      };
      int c = g;
      for (; c < il && c <= e; ++c) edge(c);
      const int z = min(e, ih);
#pragma unroll 2
      for (; c < z; c += 2) {
        const float4 a0 = ra[c], a1 = ra[c + 1];
        const float2 b0 = rb[c], b1 = rb[c + 1];
#pragma unroll
        for (int i = 0; i < kExPx; ++i)
          m[i] = cs_min_abs(m[i], cs_pd<kAngle, kCap>(v[i], n[i], a0, b0, k), cs_pd<kAngle, kCap>(v[i], n[i], a1, b1, k));
      }
      for (; c <= e; ++c) edge(c);
      const int at = yy * k.W + g;
#pragma unroll
      for (int i = 0; i < kExPx; ++i)
        if ((unsigned)(yy - pv[i] + r) <= 2u * r && (m[i] < L[i] || (m[i] == L[i] && at < G[i]))) {
          L[i] = m[i];
          G[i] = at;
        }
    }
  }
}

// The reference's arithmetic on every candidate.  A lane's four pixels share each
// candidate's load; shared memory's data path (six cycles per 32 records) is
// what bounds it with two.  The CTA's halves take every second row each.  Leaves of each
// pixel the least distance and the first run in row-major order that has it.
// all: the whole frame; otherwise the chunks that the search has left.
template <bool kAngle>
__global__ void __launch_bounds__(kCsThreads, kExCtasPerSm)
    corr_exact_kernel(const CorrConsts k, const float4* A, const float2* B, const CsPix pix,
                      const CsBox* box, const int* flag, const CsPart part, int tiles_x,
                      int tiles, bool all) {
  cs_after_previous();
  extern __shared__ float4 cs_smem[];
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, half = wid >> 2, r = k.radius;
  const int items = all ? tiles * k.chunks : *part.todo;
  for (int item = blockIdx.x; item < items; item += gridDim.x) {
    const int what = all ? 2 * item : part.todo[1 + item];
    const int chunk = (what >> 1) / tiles, tile = (what >> 1) - chunk * tiles, ty = tile / tiles_x,
              tx = tile - ty * tiles_x;
    CsTile t;
    if (!cs_tile(k, box, flag, tx, ty, chunk, t)) continue;
    // columns [xs, xe] of the rows from yb on, asynchronously; the first of them come
    // while the boxes and pixels are read
    auto stage = [&](int xs, int yb) {
      const int wu = min(t.xhi, xs + kSlab - 1) - xs + 1, band = kExSmem / (wu * 24), rows = min(band, t.c1 - yb + 1);
      float2* sB = reinterpret_cast<float2*>(cs_smem + (size_t)band * wu);
      for (int j = tid; j < rows * wu; j += kCsThreads) {
        const int rr = j / wu, g = (yb + rr) * k.W + xs + j - rr * wu;
        cp_async16(cs_smem + j, A + g);
        cp_async8(sB + j, B + g);
      }
      cp_async_commit();
    };
    stage(t.xlo, t.c0);
    bool any = true, cap = what & 1;
    if (all) {
      const CsReach q = cs_reach(k, box, t);
      any = q.any;
      cap = q.cap;
    }
    const int x = tx * kCsTx + lane, y0 = ty * kCsTy + kExPx * (wid & 3), px = y0 * k.W + x;
    float3 v[kExPx], n[kExPx];
    int pu[kExPx], pv[kExPx], G[kExPx];
    float L[kExPx];
    unsigned on = 0;
    // the windows' union, the columns common to them, their rows
    int lo = k.W, hi = -1, il = 0, ih = k.W, pl = k.H, ph = -1;
#pragma unroll
    for (int i = 0; i < kExPx; ++i) {
      CsPixel p;
      p.search = p.special = false;
      if (x < k.W && y0 + i < k.H) p = cs_load_pixel(pix, px + i * k.W);
      v[i] = n[i] = make_float3(0.f, 0.f, 0.f);
      pu[i] = 0;
      pv[i] = -(1 << 30);
      if (p.search && !p.special) {
        on |= 1u << i;
        v[i] = p.vc;
        if (kAngle) n[i] = p.nc;
        pu[i] = p.pu;
        pv[i] = p.pv;
        lo = min(lo, max(0, p.pu - r));
        hi = max(hi, min(k.W - 1, p.pu + r));
        il = max(il, p.pu - r);
        ih = min(ih, p.pu + r);
        pl = min(pl, p.pv - r);
        ph = max(ph, p.pv + r);
      }
      L[i] = INFINITY;
      G[i] = -1;
    }
    for (int xs = t.xlo; xs <= t.xhi && any; xs += kSlab) {
      const int xe = min(t.xhi, xs + kSlab - 1), wu = xe - xs + 1, band = kExSmem / (wu * 24);
      const float2* sB = reinterpret_cast<const float2*>(cs_smem + (size_t)band * wu);
      for (int yb = t.c0; yb <= t.c1; yb += band) {
        const int rows = min(band, t.c1 - yb + 1);
        if (xs > t.xlo || yb > t.c0) {
          __syncthreads();
          stage(xs, yb);
        }
        cp_async_wait<0>();
        __syncthreads();
        if (cap) cs_scan_exact<kAngle, false>(cs_smem, sB, wu, xs, xe, yb, rows, half, lo, hi, il, ih, pl, ph, v, n, pu, pv, L, G, k);
        else cs_scan_exact<kAngle, true>(cs_smem, sB, wu, xs, xe, yb, rows, half, lo, hi, il, ih, pl, ph, v, n, pu, pv, L, G, k);
      }
    }
    // the halves together
    cp_async_wait<0>();
    __syncthreads();
    float2* both = reinterpret_cast<float2*>(cs_smem) + (tid & 127);
    if (half) {
#pragma unroll
      for (int i = 0; i < kExPx; ++i) both[128 * i] = make_float2(L[i], __int_as_float(G[i]));
    }
    __syncthreads();
    if (!half) {
#pragma unroll
      for (int i = 0; i < kExPx; ++i) {
        if (!((on >> i) & 1u)) continue;
        const float2 h = both[128 * i];
        const int g = __float_as_int(h.y);
        if (h.x < L[i] || (h.x == L[i] && g < G[i])) {
          L[i] = h.x;
          G[i] = g;
        }
        const size_t at = (size_t)chunk * k.P + px + i * k.W;
        part.a[at] = make_float4(L[i], INFINITY, INFINITY, 0.f);
        part.g[at] = make_int2(G[i], -1);
      }
    }
    __syncthreads();
  }
}

// A candidate taken so far; of equal distances the first in row-major order.
struct CsBest {
  float pd;
  int i;
  __device__ __forceinline__ void take(float d, int j) {
    if (j >= 0 && (d < pd || (d == pd && i >= 0 && j < i))) {
      pd = d;
      i = j;
    }
  }
};

constexpr int kFly = 6;  // loads in flight
// A pixel's n rows of w candidates from row0 (columns from l), all within the
// cap, the warp's lanes on consecutive ones of them: the lane's first least in
// row-major order.
__device__ __forceinline__ void cs_rows(const CorrConsts& k, const float3& v, int row0, int n, int l, int w, int lane,
                                        const float4* A, const float2* B, CsBest& b) {
  const int total = n * w, dy = 32 / w, dx = 32 - dy * w;
  int y = lane / w, x = lane - y * w;
  for (int t = lane; t < total; t += 32 * kFly) {
    int at[kFly];
    float4 a[kFly];
    float2 c[kFly];
#pragma unroll
    for (int h = 0; h < kFly; ++h) {  // the loads together (one by one they take three times as long)
      at[h] = t + 32 * h < total ? (row0 + y) * k.W + l + x : -1;
      a[h] = at[h] >= 0 ? A[at[h]] : make_float4(kCsFar, kCsFar, 0.f, kCsFar);
      c[h] = at[h] >= 0 ? B[at[h]] : make_float2(0.f, 0.f);
      x += dx;
      y += dy;
      if (x >= w) {
        x -= w;
        ++y;
      }
    }
#pragma unroll
    for (int h = 0; h < kFly; ++h) {
      const float d = cs_pd<false, false>(v, v, a[h], c[h], k);
      if (d < b.pd) {
        b.pd = d;
        b.i = at[h];
      }
    }
  }
}

// Eight lanes per pixel evaluate its runs (the loads of a run's columns are then
// in flight together, and four pixels' runs per warp; a warp per run took
// three times as long).  Pixels whose third value is within the bound have those
// chunks' rows evaluated by the CTA's warps.
// own: the exact scan saw every chunk, and a lane evaluates its own pixel's one
// run.  Shorter while the merge is at most two CTAs per SM and its chain of loads
// is what it takes (160 x 120 at radius 20: 70 us a call with eight lanes, 63), longer
// beyond (640 x 480: 282 and 290).
// kDirect: no scan went before, each lane scans its pixel's window (rule at
// kCsDirect).
constexpr int kMergeThreads = 256;
static_assert(kMergeThreads <= 256 && kCorrMaxChunks <= 8, "an item: pixel, chunk");
template <bool kAngle, bool kDirect>
__global__ void __launch_bounds__(kMergeThreads)
    corr_merge_kernel(const CorrConsts k, const float* lv, const float4* A,
                      const float2* B, const CsPix pix, const int* flag, const CsPart part,
                      const KnnSrc knn, bool own, cf_correspondence* __restrict__ out, int* __restrict__ num_valid,
                      int* __restrict__ stats) {
  after_previous();
  __shared__ float s_stage[kMergeThreads / 32][32 * kCsRecWords];
  __shared__ unsigned long long s_key[kMergeThreads];  // distance bits, candidate: the least first
  __shared__ unsigned short s_items[kMergeThreads * kCorrMaxChunks];
  __shared__ int s_count, s_next;
  const int tid = threadIdx.x, lane = tid & 31;
  const int px = blockIdx.x * kMergeThreads + tid;
  const bool inimg = px < k.P;
  CsPixel p;
  p.search = false;
  p.special = false;
  p.code = -1;
  p.pu = p.pv = 0;
  p.vl = p.vc = p.nc = make_float3(0.f, 0.f, 0.f);
  p.view_cos = 0.f;
  if (tid == 0) s_count = s_next = 0;
  if (!kDirect) __syncthreads();
  if (inimg) {
    p = cs_load_pixel(pix, px);
    if (p.search) {
      p.special |= *flag != 0;
      p.vl = make_float3(lv[3 * px], lv[3 * px + 1], lv[3 * px + 2]);
    }
  }
  const bool on = p.search && !p.special;
  // an upper bound of the winner's distance, and the runs that can hold it: bit
  // 2 c + s the chunk's s-th
  CsBest best = {k.dist_thr, -1};
  float U = k.dist_thr;
  unsigned runs = 0, again = 0;  // again: the chunks of which more runs could
  if (!kDirect && on) {
    for (int c = 0; c < k.chunks; ++c) {
      const float4 a = part.a[(size_t)c * k.P + px];
      U = fminf(U, a.x + 2.25f * a.w);
    }
    unsigned only = 0;
    float found = INFINITY;  // the least of the exact scan: one run, the first that has it
    for (int c = 0; c < k.chunks; ++c) {
      const float4 a = part.a[(size_t)c * k.P + px];
      if (a.w == 0.f) {
        if (a.x <= U && a.x < found) {
          found = a.x;
          runs &= ~only;
          only = 1u << (2 * c);
          runs |= only;
        }
        continue;
      }
      runs |= (a.x <= U ? 1u : 0u) << (2 * c) | (a.y <= U ? 2u : 0u) << (2 * c);
      again |= (a.z <= U ? 1u : 0u) << c;
    }
  }
  if (kDirect && on) {
    const int l = max(0, p.pu - k.radius), h = min(k.W - 1, p.pu + k.radius);
    const int ya = max(0, p.pv - k.radius), yz = min(k.H - 1, p.pv + k.radius);
    for (int yy = ya; yy <= yz; ++yy)
#pragma unroll 4
      for (int c = l; c <= h; ++c) {
        const float d = cs_pd<kAngle>(p.vc, p.nc, A[yy * k.W + c], B[yy * k.W + c], k);
        if (d < best.pd) {
          best.pd = d;
          best.i = yy * k.W + c;
        }
      }
  }
  if (!kDirect && own && runs) {  // the one run that the exact scan has found
    const int g = part.g[(size_t)((__ffs(runs) - 1) >> 1) * k.P + px].x, row0 = g / k.W * k.W, c0 = g - row0;
    const int l = max(c0, p.pu - k.radius), h = min(min(c0 + kGroup - 1, k.W - 1), p.pu + k.radius);
    for (int col = l; col <= h; col += kFly) {
      float4 a[kFly];
      float2 b[kFly];
#pragma unroll
      for (int j = 0; j < kFly; ++j) {
        const int i = row0 + min(col + j, h);
        a[j] = A[i];
        b[j] = B[i];
      }
#pragma unroll
      for (int j = 0; j < kFly; ++j) {
        const float d = cs_pd<kAngle>(p.vc, p.nc, a[j], b[j], k);
        if (d < best.pd) {
          best.pd = d;
          best.i = row0 + min(col + j, h);
        }
      }
    }
  }
  for (unsigned todo; !kDirect && !own && (todo = __ballot_sync(0xffffffffu, runs != 0)) != 0;) {
    const unsigned mine = (todo >> (lane & 24)) & 0xffu;  // of this lane's eight pixels
    const int src = (lane & 24) + (mine ? __ffs(mine) - 1 : 0);
    int gs = -1;
    if (mine && lane == src) {
      const int e = __ffs(runs) - 1;
      runs &= runs - 1;
      const int2 g = part.g[(size_t)(e >> 1) * k.P + px];
      gs = e & 1 ? g.y : g.x;
    }
    const int gg = __shfl_sync(0xffffffffu, gs, src), pu = __shfl_sync(0xffffffffu, p.pu, src);
    const float3 v = make_float3(__shfl_sync(0xffffffffu, p.vc.x, src), __shfl_sync(0xffffffffu, p.vc.y, src),
                                 __shfl_sync(0xffffffffu, p.vc.z, src));
    float3 nc = v;
    if (kAngle)
      nc = make_float3(__shfl_sync(0xffffffffu, p.nc.x, src), __shfl_sync(0xffffffffu, p.nc.y, src),
                       __shfl_sync(0xffffffffu, p.nc.z, src));
    CsBest b = {INFINITY, -1};
    if (mine && gg >= 0) {
      const int row0 = gg / k.W * k.W, c0 = gg - row0;
      const int l = max(c0, pu - k.radius), h = min(min(c0 + kGroup - 1, k.W - 1), pu + k.radius);
      const int first = l + (lane & 7);
      if (h - l < 8 * kFly) {  // all loads together (640 x 480 at radius 20: 280 us a call in fours, 271)
        float4 a[kFly];
        float2 c[kFly];
#pragma unroll
        for (int j = 0; j < kFly; ++j) {
          const int i = row0 + min(first + 8 * j, h);
          a[j] = A[i];
          c[j] = B[i];
        }
#pragma unroll
        for (int j = 0; j < kFly; ++j) {
          const float d = cs_pd<kAngle>(v, nc, a[j], c[j], k);
          if (d < b.pd) {
            b.pd = d;
            b.i = row0 + min(first + 8 * j, h);
          }
        }
      } else {
#pragma unroll 4
        for (int col = first; col <= h; col += 8) {
          const float d = cs_pd<kAngle>(v, nc, A[row0 + col], B[row0 + col], k);
          if (d < b.pd) {
            b.pd = d;
            b.i = row0 + col;
          }
        }
      }
    }
#pragma unroll
    for (int o = 4; o; o >>= 1) {
      const float d = __shfl_xor_sync(0xffffffffu, b.pd, o);
      const int i = __shfl_xor_sync(0xffffffffu, b.i, o);
      b.take(d, i);
    }
    if (mine && lane == src) best.take(b.pd, b.i);
  }
  // The pixels left: the rows of their chunks, a chunk at a time to the CTA's
  // next free warp (a surface of equal distances leaves whole CTAs of them).
  if (!kDirect && !kAngle && !own) {  // (only the search leaves such, and it knows no angle)
    float* q = s_stage[0] + 5 * tid;  // (the records' staging is not in use yet)
    if (again) {
      q[0] = p.vc.x; q[1] = p.vc.y; q[2] = p.vc.z;
      q[3] = __int_as_float(p.pu); q[4] = __int_as_float(p.pv);
      s_key[tid] = best.i < 0 ? ~0ull : (unsigned long long)__float_as_uint(best.pd) << 32 | (unsigned)best.i;
      for (unsigned m = again; m; m &= m - 1)
        s_items[atomicAdd(&s_count, 1)] = (unsigned short)(tid | (__ffs(m) - 1) << 8);
    }
    __syncthreads();
    const int items = s_count;
    for (;;) {
      int t = 0;
      if (lane == 0) t = atomicAdd(&s_next, 1);
      t = __shfl_sync(0xffffffffu, t, 0);
      if (t >= items) break;
      const int src = s_items[t] & 255, cc = s_items[t] >> 8;
      const float* r = s_stage[0] + 5 * src;
      const float3 v = make_float3(r[0], r[1], r[2]);
      const int pu = __float_as_int(r[3]), pv = __float_as_int(r[4]);
      const int spx = blockIdx.x * kMergeThreads + src, y = spx / k.W, x = spx - y * k.W;
      const int2 rw = part.rows[y / kCsTy * ((k.W + kCsTx - 1) / kCsTx) + x / kCsTx];
      const int l = max(0, pu - k.radius), w = min(k.W - 1, pu + k.radius) - l + 1;
      const int ya = max(max(0, pv - k.radius), rw.x + cc * rw.y),
                n = min(min(k.H - 1, pv + k.radius), rw.x + cc * rw.y + rw.y - 1) - ya + 1;
      CsBest b = {k.dist_thr, -1};
      cs_rows(k, v, ya, n, l, w, lane, A, B, b);
#pragma unroll
      for (int o = 16; o; o >>= 1) {
        const float d = __shfl_xor_sync(0xffffffffu, b.pd, o);
        const int i = __shfl_xor_sync(0xffffffffu, b.i, o);
        b.take(d, i);
      }
      if (lane == 0 && b.i >= 0)
        atomicMin(&s_key[src], (unsigned long long)__float_as_uint(b.pd) << 32 | (unsigned)b.i);
    }
    __syncthreads();
    if (again && s_key[tid] != ~0ull) {
      best.pd = __uint_as_float((unsigned)(s_key[tid] >> 32));
      best.i = (int)(unsigned)s_key[tid];
    }
    __syncthreads();  // (the staging is the records' again)
  }
  int code = p.code;
  int bi = -1;
  if (p.search) {
    bool saw_depth = false;
    if (p.special) {
      bi = cs_rescan(k, p, A, B, saw_depth);
    } else {
      bi = best.i;
      if (bi < 0 && stats) saw_depth = cs_any_depth(k, p, A);
    }
    code = bi >= 0 ? 5 : (saw_depth ? 3 : 2);
  }
  cs_emit(k, p, inimg, px, bi, code, A, B, knn, out, num_valid, stats, lane, s_stage[threadIdx.x >> 5]);
}

__global__ void pixel_knn_kernel(const int* hit, int P, const int* vk,
                                 const float* vw, long long num_voxels, int* __restrict__ pk,
                                 float* __restrict__ pw) {
  after_previous();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= P) return;
  const int v = hit[i];
  const bool ok = v >= 0 && (long long)v < num_voxels;
#pragma unroll
  for (int j = 0; j < CF_K_NEIGHBORS; ++j) {
    pk[(size_t)i * CF_K_NEIGHBORS + j] = ok ? vk[(size_t)v * CF_K_NEIGHBORS + j] : -1;
    pw[(size_t)i * CF_K_NEIGHBORS + j] = ok ? vw[(size_t)v * CF_K_NEIGHBORS + j] : 0.f;
  }
}

// Largest float s with sqrtf(s) <= cap (IEEE square roots on both sides), so
// that sqrtf(s) > cap exactly when s > bound.
float sqrt_bound(float cap) {
  if (std::isnan(cap)) return NAN;  // sqrtf(s) > NaN never holds; neither does s > NaN
  if (cap < 0.f) return -INFINITY;
  if (std::isinf(cap)) return INFINITY;
  float s = cap * cap;
  if (std::isinf(s)) s = FLT_MAX;
  while (s > 0.f && std::sqrt(s) > cap) s = std::nextafter(s, 0.f);
  for (;;) {
    const float up = std::nextafter(s, INFINITY);
    if (std::isinf(up) || !(std::sqrt(up) <= cap)) break;
    s = up;
  }
  return s;
}

}  // namespace

// Row chunks per tile.  Rough model in SM clocks, from 640 x 480 at radii 8, 20
// and 50 and 320 x 240 at 20, each with 1 to 8 chunks: a CTA's set-up takes 9000,
// its scan of 512 pixels x S/C candidates goes at 9 per clock beside two others,
// the last CTAs run with fewer beside them, so the waves count as
// tiles x C / slots + 0.4; the merge reads each chunk for 5000 at 640 x 480.
// The exact scan: 6000, 8 beside one other (80 x 60 to 1280 x 960 at radii 9 to 50:
// 1.5 % above the best number of chunks on average, 10 % at most).
int corr_pick_chunks(int tiles, int sms, int radius, int W, int H, bool filter) {
  const double slots = (double)(sms > 0 ? sms : 1) * (filter ? kCsCtasPerSm : kExCtasPerSm);
  const double side_x = std::fmin(2.0 * radius + 8.0, (double)W), side_y = std::fmin(2.0 * radius + 8.0, (double)H);
  const double setup = filter ? 9000.0 : 6000.0;
  const double scan = 512.0 * side_x * side_y / (filter ? 9.0 : 8.0), merge = 5000.0 * ((double)W * H / 307200.0);
  int best_c = 1;
  double best = 1e300;
  for (int c = 1; c <= kCorrMaxChunks; ++c) {
    const double t = ((double)tiles * c / slots + 0.4) * (setup + scan / c) + merge * c;
    if (t < best * (1.0 - 1e-9)) {
      best = t;
      best_c = c;
    }
  }
  return best_c;
}

// Row chunks that the partials of frames of up to P pixels have room for.
int corr_chunk_cap(size_t P) {
  return (int)std::fmax(1.0, std::fmin((double)kCorrMaxChunks, std::floor((double)(1u << 27) / (double)P)));
}

// Blocks of frames of up to P pixels, whatever their sides.
size_t corr_box_cap(size_t P) { return P / (kCsBlock * kCsBlock) + (P + 1) / kCsBlock + 2; }
size_t corr_box_bytes() { return sizeof(CsBox); }

cudaError_t launch_corr_search(const cf_corr_frame* f, const cf_camera* cam, const cf_mat4* Tcw, const cf_mat4* Twc,
                               const cf_corr_params* p, const CorrScratch& sc, int chunks, cf_correspondence* out,
                               int* num_valid, int* stats, cudaStream_t s, long long* launches) {
  cudaError_t e = cudaSuccess;
  const int W = cam->width, H = cam->height;
  CorrConsts k;
  k.fx = cam->fx;
  k.fy = cam->fy;
  k.cx = cam->cx;
  k.cy = cam->cy;
  k.W = W;
  k.H = H;
  k.P = W * H;
  // a window wider than the image reads the same pixels as the image itself
  const int span = W > H ? W : H;
  k.radius = p->search_radius_px < 0 ? 0 : (p->search_radius_px > span ? span : p->search_radius_px);
  for (int r = 0; r < 3; ++r)
    for (int c = 0; c < 4; ++c) {
      k.cw[4 * r + c] = Tcw->m[r][c];
      k.wc[4 * r + c] = Twc->m[r][c];
    }
  k.dist_thr = p->dist_threshold;
  k.angle_thr = p->angle_threshold;
  k.view_thr = p->view_threshold;
  // kernels/tsdf_kernels.cu:456-458
  const float d3 = 3.0f * p->dist_threshold, d2 = p->dist_threshold + 0.03f;
  k.cap = std::fmax(d3, d2);
  const float ne = 1.0f - p->angle_threshold, ve = 1.0f - p->view_threshold;
  k.normal_eps = std::fmax(ne, 1e-4f);
  k.view_eps = std::fmax(ve, 1e-4f);
  k.s_max = sqrt_bound(k.cap);

  KnnSrc knn;
  knn.pixel_knn = f->d_pixel_knn;
  knn.pixel_knn_w = f->d_pixel_knn_w;
  knn.hit = f->d_pixel_knn ? nullptr : f->d_hit_voxel_idx;
  knn.voxel_knn = f->d_voxel_knn;
  knn.voxel_knn_w = f->d_voxel_knn_w;
  knn.num_voxels = f->d_voxel_knn ? f->num_voxels : 0;
  knn.pixel_knn_out = f->d_pixel_knn ? nullptr : f->d_pixel_knn_out;
  knn.pixel_knn_w_out = f->d_pixel_knn ? nullptr : f->d_pixel_knn_w_out;

  if (W == 0 || H == 0) {
    e = cudaMemsetAsync(num_valid, 0, sizeof(int), s);
    if (e == cudaSuccess && stats) e = cudaMemsetAsync(stats, 0, 6 * sizeof(int), s);
    return e;
  }
  // a NaN bound defeats the strict-less rule (the reference then accepts every
  // candidate it reaches) and an infinite one lets a skip record pass the
  // Euclidean test: such calls take the sequential scan throughout
  e = cudaMemsetAsync(sc.flag, std::isfinite(p->dist_threshold) ? 0 : 1, sizeof(int), s);
  if (e != cudaSuccess) return e;

  const dim3 tiles((W + kCsTx - 1) / kCsTx, (H + kCsTy - 1) / kCsTy);
  const bool angle = p->angle_threshold > 0.f;
  const double side = 2.0 * k.radius + 1.0;
  const bool filter = !angle && (double)k.P * std::fmin(side, W) * std::fmin(side, H) > kCsFilter;
  const int want = chunks > 0 ? chunks : corr_pick_chunks((int)(tiles.x * tiles.y), sc.sms, k.radius, W, H, filter);
  k.chunks = want < sc.chunk_cap ? want : sc.chunk_cap;
  auto exact = angle ? corr_exact_kernel<true> : corr_exact_kernel<false>;
  const bool direct = k.radius <= (angle ? kCsDirectAngle : kCsDirect);
  auto merge = direct ? (angle ? corr_merge_kernel<true, true> : corr_merge_kernel<false, true>)
                      : (angle ? corr_merge_kernel<true, false> : corr_merge_kernel<false, false>);
  // per device and cheap: set on every call rather than cached per device
  e = cudaFuncSetAttribute(corr_search_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kCsSmem);
  if (e == cudaSuccess) e = cudaFuncSetAttribute(exact, cudaFuncAttributeMaxDynamicSharedMemorySize, kExSmem);
  if (e != cudaSuccess) return e;
  const CsPart part = {sc.part_a, sc.part_g, sc.rows, sc.todo};

  const CsPix pix = {sc.pix_v, sc.pix_n, sc.pix_row};
  CsBox* box = static_cast<CsBox*>(sc.box);
  launch_next(corr_prep_kernel, dim3((W + kCsBlock - 1) / kCsBlock, (H + kCsBlock - 1) / kCsBlock),
              kCsBlock * kCsBlock, 0, s, k, f->d_depth, f->d_depth_normals, f->d_live_vertices, f->d_live_normals,
              sc.A, sc.B, pix, box, sc.flag, sc.todo, num_valid, stats);
  // (launch_next only for the short calls: CTAs of the merge that wait beside a
  // running search cost 15 of 573 us at radius 50)
  const int mg = (k.P + kMergeThreads - 1) / kMergeThreads;
  if (direct) {
    launch_next(merge, mg, kMergeThreads, 0, s, k, f->d_live_vertices, sc.A, sc.B, pix, sc.flag, part, knn, true, out,
                num_valid, stats);
  } else {
    const dim3 grid(tiles.x, tiles.y, k.chunks);
    if (filter) corr_search_kernel<<<grid, kCsThreads, kCsSmem, s>>>(k, sc.A, sc.B, pix, box, sc.flag, part);
    const int n = (int)(tiles.x * tiles.y), items = n * k.chunks, slots = kExCtasPerSm * (sc.sms > 0 ? sc.sms : 1);
    launch_next(exact, filter && items > slots ? slots : items, kCsThreads, kExSmem, s, k, sc.A, sc.B, pix, box, sc.flag,
                part, (int)tiles.x, n, !filter);
    launch_next(merge, mg, kMergeThreads, 0, s, k, f->d_live_vertices, sc.A, sc.B, pix, sc.flag, part, knn,
                !filter && mg <= 2 * sc.sms, out, num_valid, stats);
  }
  *launches += direct ? 2 : filter ? 4 : 3;
  return cudaGetLastError();
}

cudaError_t launch_pixel_knn(const int* hit, int P, const int* vk, const float* vw, long long num_voxels, int* pk,
                             float* pw, cudaStream_t s) {
  if (P <= 0) return cudaSuccess;
  launch_next(pixel_knn_kernel, (P + 255) / 256, 256, 0, s, hit, P, vk, vw, num_voxels, pk, pw);
  return cudaGetLastError();
}

}  // namespace cf
