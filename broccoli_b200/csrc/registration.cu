// registration.cu -- the per-iteration kernels of batched linear registration
// and the volume helpers around it (warps, separable smoothing, rescale).
//
// Per affine iteration and instance:
//   normal_eq_partial_kernel  phase difference, certainty and phase gradient
//                             of the three filter pairs, reduced to the 42
//                             distinct sums of the 12x12 system (FP64).
//   solve_update_kernel       reduces the partial sums in a fixed order,
//                             solves the three decoupled 4x4 systems in FP64,
//                             applies the TRANSLATION / RIGID / AFFINE update
//                             and the convergence test.
//   warp_affine_kernel        exact-weight trilinear resampling of the
//                             original volume with the total parameters.
#include <math.h>

#include <type_traits>

#include "common.cuh"
#include "internal.h"

namespace brc {

// ---------------------------------------------------------------------------
// Normal equations
// ---------------------------------------------------------------------------

constexpr int kNEThreads = 256;
// Largest volume the 32-bit voxel indexing of the resampling kernels takes.
constexpr long long kMaxVoxels = 0x7fffff00LL;

// Phase difference and certainty of one response pair
// (CalculatePhaseDifferencesAndCertainties, kernelRegistration.cpp:173-211):
// dphi = arg(q1 q2*), c = |q1 q2| cos^2(dphi/2).  With cos^2(t/2) =
// (1 + cos t)/2 and cos dphi = Re(q1 q2*)/|q1 q2*|, c = (|q1 q2*| + Re(q1 q2*))/2:
// the same value without the cosine (|q1 q2| = |q1 q2*|).
__device__ __forceinline__ void phase_diff_cert(float2 a, float2 c, float& pd, float& cert) {
  // products rounded separately (no FMA contraction), as in the reference's
  // arithmetic: identical responses then give exactly zero phase difference
  const float re = __fadd_rn(__fmul_rn(a.x, c.x), __fmul_rn(a.y, c.y));
  const float im = __fsub_rn(__fmul_rn(a.y, c.x), __fmul_rn(a.x, c.y));
  pd = phase_atan2(im, re);
  cert = 0.5f * __fadd_rn(sqrt_approx(fmaf(re, re, __fmul_rn(im, im))), re);
}

// Phase gradient from the neighbours along one axis
// (CalculatePhaseGradientsX/Y/Z, kernelRegistration.cpp:213-382).
__device__ __forceinline__ float phase_grad(float2 a_p, float2 a_c, float2 a_m, float2 c_p,
                                            float2 c_c, float2 c_m) {
  float tr = 0.f, ti = 0.f;
  tr += a_p.x * a_c.x + a_p.y * a_c.y;
  ti += a_p.y * a_c.x - a_p.x * a_c.y;
  tr += a_c.x * a_m.x + a_c.y * a_m.y;
  ti += a_c.y * a_m.x - a_c.x * a_m.y;
  tr += c_p.x * c_c.x + c_p.y * c_c.y;
  ti += c_p.y * c_c.x - c_p.x * c_c.y;
  tr += c_c.x * c_m.x + c_c.y * c_m.y;
  ti += c_c.y * c_m.x - c_c.x * c_m.y;
  return phase_atan2(ti, tr);
}

// phase_grad with every rounding written out, for the kernel whose forms have
// to agree bit for bit (left to the compiler, the products that fuse with an
// addition differ from kernel to kernel).
__device__ __forceinline__ float phase_grad_rn(float2 a_p, float2 a_c, float2 a_m, float2 c_p,
                                               float2 c_c, float2 c_m) {
  // p conj(o) of each pair of neighbours, summed in order
  const auto re = [](float2 p, float2 o) { return fmaf(p.x, o.x, __fmul_rn(p.y, o.y)); };
  const auto im = [](float2 p, float2 o) { return fmaf(p.y, o.x, -__fmul_rn(p.x, o.y)); };
  const float tr = __fadd_rn(__fadd_rn(__fadd_rn(re(a_p, a_c), re(a_c, a_m)), re(c_p, c_c)), re(c_c, c_m));
  const float ti = __fadd_rn(__fadd_rn(__fadd_rn(im(a_p, a_c), im(a_c, a_m)), im(c_p, c_c)), im(c_c, c_m));
  return phase_atan2(ti, tr);
}

// Sum e (0..13) of one axis as (row moment) x y^py x z^pz: moments
// [sum w, sum w x, sum w x^2, sum v, sum v x] of the row, y and z relative
// to the volume centre.
__constant__ signed char c_sum_moment[14] = {0, 1, 0, 0, 2, 1, 1, 0, 0, 0, 3, 4, 3, 3};
__constant__ signed char c_sum_ypow[14] = {0, 0, 1, 0, 0, 1, 0, 2, 1, 0, 0, 0, 1, 0};
__constant__ signed char c_sum_zpow[14] = {0, 0, 0, 1, 0, 0, 1, 0, 1, 2, 0, 0, 0, 1};

__device__ __forceinline__ double pick_moment(const float (&m)[3][5], int sel) {
  float r = 0.f;
#pragma unroll
  for (int k = 0; k < 3; k++)
#pragma unroll
    for (int q = 0; q < 5; q++) r = (sel == 5 * k + q) ? m[k][q] : r;
  return (double)r;
}
__device__ __forceinline__ double ypow(double y, int e) {
  const int p = c_sum_ypow[e];
  return p == 0 ? 1.0 : (p == 1 ? y : y * y);
}
__device__ __forceinline__ double zpow(double z, int e) {
  const int p = c_sum_zpow[e];
  return p == 0 ? 1.0 : (p == 1 ? z : z * z);
}

// Sums over the interior (3 voxels from every face) of
//   c g^2 [1, x, y, z, xx, xy, xz, yy, yz, zz]  and  c g dphi [1, x, y, z]
// for each axis k (sum index 14k + e), coordinates relative to the volume
// centre: the 30 + 12 values that CalculateAMatrixAndHVector2DValuesX/Y/Z,
// CalculateAMatrix1DValues / HVector1DValues and CalculateAMatrix /
// HVector accumulate (kernelRegistration.cpp:387-800).  One CTA handles
// `zpb` interior slices of one instance and writes 42 FP64 partial sums.
//
// One warp walks one (y, z) row at a time, lanes along x (coalesced float2
// loads).  Within a row y and z are constant, so the 42 sums factor into 15
// row moments per lane, sum_x w [1, x, x^2] and sum_x v [1, x] for the three
// axes, reduced over the warp in FP32 and expanded into the 42 sums in FP64
// (lane j owns sums j and 32 + j).  The same order on every run: results
// are deterministic.
__global__ void __launch_bounds__(kNEThreads, 4)
normal_eq_partial_kernel(const float2* __restrict__ q1, long long q1_stride,
                         const float2* __restrict__ q2, int W, int H, int D, int zpb,
                         double* __restrict__ partials) {
  const int b = blockIdx.y;
  const long long V = (long long)W * H * D;
  const long long WH = (long long)W * H;
  const float2* Q1 = q1 + (long long)b * q1_stride;
  const float2* Q2 = q2 + (long long)b * 3 * V;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;

  const int nx = W - 6, ny = H - 6;
  const int z0 = 3 + blockIdx.x * zpb;
  const int z1 = min(D - 3, z0 + zpb);
  const int nrows = (nx > 0 && ny > 0 && z1 > z0) ? ny * (z1 - z0) : 0;
  const float cxf = 0.5f * (float)(W - 1);
  const double cy = 0.5 * (H - 1), cz = 0.5 * (D - 1);

  // lane j accumulates sums j and 32 + j (the latter for j < 10)
  double acc_lo = 0.0, acc_hi = 0.0;
  const int jlo = lane, jhi = 32 + lane;
  const int elo = jlo % 14, ehi = jhi % 14;
  const int slo = 5 * (jlo / 14) + c_sum_moment[elo];
  const int shi = jhi < kNSums ? 5 * (jhi / 14) + c_sum_moment[ehi] : 0;

  for (int r = warp; r < nrows; r += kNEThreads / 32) {
    const int y = 3 + r % ny;
    const int z = z0 + r / ny;
    const long long row = (long long)y * W + (long long)z * WH;
    // [k][0..4] = sum w, sum w x, sum w x^2, sum v, sum v x
    float m[3][5];
#pragma unroll
    for (int k = 0; k < 3; k++)
#pragma unroll
      for (int q = 0; q < 5; q++) m[k][q] = 0.f;
    // all lanes run every chunk (shuffles need the full warp); lanes past
    // the interior load their clamped centre for their neighbours' use and
    // add nothing
    for (int xb = 3; xb < W - 3; xb += 32) {
      const int x = xb + lane;
      const bool act = x < W - 3;
      const long long i = row + (x < W ? x : W - 1);
      const float xf = (float)x - cxf;
#pragma unroll
      for (int k = 0; k < 3; k++) {
        const float2* A = Q1 + k * V;
        const float2* C = Q2 + k * V;
        const float2 a = __ldg(A + i), c = __ldg(C + i);
        float2 ap, am, cp, cm;
        if (k == 0) {
          // x neighbours from the adjacent lanes; the warp's end lanes load
          ap = make_float2(__shfl_down_sync(0xffffffffu, a.x, 1), __shfl_down_sync(0xffffffffu, a.y, 1));
          cp = make_float2(__shfl_down_sync(0xffffffffu, c.x, 1), __shfl_down_sync(0xffffffffu, c.y, 1));
          am = make_float2(__shfl_up_sync(0xffffffffu, a.x, 1), __shfl_up_sync(0xffffffffu, a.y, 1));
          cm = make_float2(__shfl_up_sync(0xffffffffu, c.x, 1), __shfl_up_sync(0xffffffffu, c.y, 1));
          if (lane == 31 && act) {
            ap = __ldg(A + i + 1);
            cp = __ldg(C + i + 1);
          }
          if (lane == 0) {
            am = __ldg(A + i - 1);
            cm = __ldg(C + i - 1);
          }
        } else {
          const long long st = k == 1 ? (long long)W : WH;
          ap = act ? __ldg(A + i + st) : a;
          am = act ? __ldg(A + i - st) : a;
          cp = act ? __ldg(C + i + st) : c;
          cm = act ? __ldg(C + i - st) : c;
        }
        float pd, cert;
        phase_diff_cert(a, c, pd, cert);
        const float g = phase_grad(ap, a, am, cp, c, cm);
        const float cg = act ? cert * g : 0.f;
        const float w = cg * g;
        const float v = cg * pd;
        m[k][0] += w;
        m[k][1] += w * xf;
        m[k][2] += w * xf * xf;
        m[k][3] += v;
        m[k][4] += v * xf;
      }
    }
#pragma unroll
    for (int k = 0; k < 3; k++)
#pragma unroll
      for (int q = 0; q < 5; q++) {
        float t = m[k][q];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        m[k][q] = t;
      }
    const double yf = (double)y - cy, zf = (double)z - cz;
    acc_lo += pick_moment(m, slo) * ypow(yf, elo) * zpow(zf, elo);
    if (jhi < kNSums) acc_hi += pick_moment(m, shi) * ypow(yf, ehi) * zpow(zf, ehi);
  }

  // Deterministic block reduction: warps in order.
  __shared__ double s_part[kNEThreads / 32][kNSums];
  s_part[warp][jlo] = acc_lo;
  if (jhi < kNSums) s_part[warp][jhi] = acc_hi;
  __syncthreads();
  if (threadIdx.x < kNSums) {
    double v = 0.0;
#pragma unroll
    for (int w = 0; w < kNEThreads / 32; w++) v += s_part[w][threadIdx.x];
    partials[((long long)b * gridDim.x + blockIdx.x) * kNSums + threadIdx.x] = v;
  }
}

// ---------------------------------------------------------------------------
// Normal equations, z-marching form: certainty smoothing fused in.
//
// One CTA of 10 warps x 32 lanes covers a patch of 30 x 8 interior voxels
// (x, y) with a one-voxel halo (lanes 0 and 31, warps 0 and 9) and walks a
// slab of interior planes z0..z1-1, reading each plane's responses once:
//   * certainties of a plane are smoothed along x by shuffles, along y
//     through shared memory and along z through a three-plane window kept
//     in shared memory (the separable 3x3x3 Gaussian in the order x, y, z);
//   * phase-gradient neighbours come from the adjacent lanes (x), from the
//     shared-memory copy of the axis-1 responses of the adjacent warps (y)
//     and from the previous / next plane held in registers (z);
//   * each lane accumulates, over the planes, the FP32 moments
//     sum w [1, z, z^2] and sum v [1, z] of its (x, y) column per axis, which
//     are expanded once into the 42 FP64 sums.
// The next plane's responses are loaded while the current plane's sums are
// computed.  Without smoothing, the same sums as normal_eq_partial_kernel
// up to FP32 summation order.
// ---------------------------------------------------------------------------

constexpr int kMarchWarps = 10;              // 8 output rows + 2 halo rows
constexpr int kMarchCols = 30;               // output columns per warp
constexpr int kMarchThreads = kMarchWarps * 32;
constexpr int kMarchZs = 32;                 // at most this many planes per slab (14: 3.5 % slower for a series)
constexpr int kMarchMaxGs = 10;              // planes of a CTA of a shared slab (7.5 KB of shared memory each)

constexpr int kMarchRowSums = 27;            // 9 row moments per axis (below)
// Row moment of sum e (0..13) of an axis: [s0, x s0, xx s0, sz, x sz, szz, v0, x v0, vz].
__constant__ signed char c_row_moment[14] = {0, 1, 0, 3, 2, 1, 4, 0, 3, 5, 6, 7, 6, 8};

struct PlaneQ {
  float2 a[3], c[3];  // q1, q2 of the three filters at this lane's (x, y)
};

__device__ __forceinline__ void load_plane_q(const float2* __restrict__ Q1, const float2* __restrict__ Q2,
                                             long long V, long long i, bool in, PlaneQ& q) {
#pragma unroll
  for (int k = 0; k < 3; k++) {
    q.a[k] = in ? __ldg(Q1 + k * V + i) : make_float2(0.f, 0.f);
    q.c[k] = in ? __ldg(Q2 + k * V + i) : make_float2(0.f, 0.f);
  }
}

// All threads of the CTAs of a cluster.
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// A float at the address `p` of this CTA's shared memory, read from CTA `rank`.
__device__ __forceinline__ float cluster_load(const float* p, int rank) {
  uint32_t a;
  float v;
  asm("mapa.shared::cluster.u32 %0, %1, %2;"
      : "=r"(a)
      : "r"(static_cast<uint32_t>(__cvta_generic_to_shared(p))), "r"(rank));
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
  return v;
}

// Three-tap sum with the weights w1, w0, w1.
__device__ __forceinline__ float smooth3(float w0, float w1, float a, float b, float c) {
  return fmaf(w1, c, fmaf(w1, a, __fmul_rn(w0, b)));
}

// Adds a plane's w and v to the moments of an axis.
__device__ __forceinline__ void add_moments(float (&m)[5], float wv, float vv, float zf) {
  const float wz = __fmul_rn(wv, zf);
  m[0] = __fadd_rn(m[0], wv);
  m[1] = __fadd_rn(m[1], wz);
  m[2] = fmaf(wz, zf, m[2]);
  m[3] = __fadd_rn(m[3], vv);
  m[4] = fmaf(vv, zf, m[4]);
}

// SPLIT: a cluster of np CTAs shares a slab, gs planes each.  The CTAs keep the
// w and v of their planes in shared memory and the first one adds them all
// plane by plane, so that the FP32 moments are those of one CTA walking the
// slab, bit for bit, and a volume's result does not depend on the batch it is
// in.  Every rounding on the way from the responses to the sums is written
// out (which products fuse with an addition is the compiler's choice
// otherwise, in each form of the kernel for itself).
template <bool SMOOTH, bool SPLIT>
__global__ void __launch_bounds__(kMarchWarps * 32, 2)
normal_eq_march_kernel(const float2* __restrict__ q1, long long q1_stride, const float2* __restrict__ q2, int W,
                       int H, int D, int ntx, int nty, int zs, int gs, int np, double* __restrict__ partials,
                       const ActiveSet act, float cw0, float cw1) {
  extern __shared__ float s_wv[];  // SPLIT: [gs planes][3 axes][w, v][threads]
  if ((int)blockIdx.y >= active_count(act, (int)gridDim.y)) return;
  const int b = active_instance(act, blockIdx.y);
  // Shared slots are numbered by step: the plane of step s (p = z0 - 1 + s)
  // uses slot s % 3, a constant in each of the three unrolled copies below.
  __shared__ float sxr[kMarchWarps][3][32];     // x-smoothed certainties of the newest plane
  // x/y-smoothed certainties of the last three planes; each thread reads
  // back only its own entries, so no barrier guards them
  __shared__ float cxr[SMOOTH ? 3 : 1][kMarchWarps][3][32];
  __shared__ float2 qy1[3][kMarchWarps][32];    // axis-1 responses (q1) of the last planes
  __shared__ float2 qy2[3][kMarchWarps][32];    // axis-1 responses (q2)
  __shared__ double s_part[kMarchWarps][kMarchRowSums];
  const long long V = (long long)W * H * D;
  const long long WH = (long long)W * H;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int part = SPLIT ? blockIdx.x % np : 0;
  const int bx = SPLIT ? blockIdx.x / np : blockIdx.x, nbx = SPLIT ? gridDim.x / np : gridDim.x;
  const int zsl = bx / (ntx * nty), rem = bx - zsl * (ntx * nty);
  const int yt = rem / ntx, xt = rem - yt * ntx;
  const int x = 3 + xt * kMarchCols - 1 + lane;  // lanes 0 and 31: halo columns
  const int y = 3 + yt * 8 - 1 + warp;           // warps 0 and 9: halo rows
  const int zend = min(D - 3, 3 + (zsl + 1) * zs);
  const int z0 = 3 + zsl * zs + (SPLIT ? part * gs : 0);
  const int z1 = SPLIT ? min(zend, z0 + gs) : zend;
  const bool empty = W <= 6 || H <= 6 || z1 <= z0;  // no interior voxel: zero sums
  const float2* Q1 = q1 + (long long)b * q1_stride;
  const float2* Q2 = q2 + (long long)b * 3 * V;
  const bool in = x < W && y < H;                         // loads stay inside the volume
  const bool cin = x <= W - 3 && y <= H - 3;              // certainty defined (smoothing support)
  const bool out = lane >= 1 && lane <= kMarchCols && warp >= 1 && warp <= 8 && x <= W - 4 && y <= H - 4;
  const long long col = (long long)y * W + x;
  const float xf = (float)x - 0.5f * (float)(W - 1);
  const float w0 = cw0, w1 = cw1;

  // per-lane moments over the planes: [k][sum w, sum w z, sum w z^2, sum v, sum v z]
  float m[3][5];
#pragma unroll
  for (int k = 0; k < 3; k++)
#pragma unroll
    for (int q = 0; q < 5; q++) m[k][q] = 0.f;

  // Three plane buffers whose roles rotate by step: at step s (plane p) the
  // current one holds plane p - 1 (the output plane), the newest plane p,
  // and the third, which held plane p - 2, receives plane p + 1.  The loop
  // is unrolled three times so that the rotation costs no register moves.
  PlaneQ pb0, pb1, pb2;
  float2 prev_a2 = make_float2(0.f, 0.f), prev_c2 = make_float2(0.f, 0.f);  // axis 2 at z - 1
#pragma unroll
  for (int k = 0; k < 3; k++) pb0.a[k] = pb0.c[k] = pb2.a[k] = pb2.c[k] = make_float2(0.f, 0.f);
  if (!empty) load_plane_q(Q1, Q2, V, (long long)(z0 - 1) * WH + col, in, pb1);

  auto step = [&](auto slot, int p, PlaneQ& cur, PlaneQ& nw, PlaneQ& nxt) {
    constexpr int j = decltype(slot)::value;  // slot of plane p
    constexpr int j1 = (j + 2) % 3;            // plane p - 1
    constexpr int j2 = (j + 1) % 3;            // plane p - 2
    // [A] certainties of plane p, x pass, axis-1 responses to shared memory
    if (SMOOTH) {
#pragma unroll
      for (int k = 0; k < 3; k++) {
        float pd, cv = 0.f;
        phase_diff_cert(nw.a[k], nw.c[k], pd, cv);
        cv = cin ? cv : 0.f;
        const float cl = __shfl_up_sync(0xffffffffu, cv, 1), cr = __shfl_down_sync(0xffffffffu, cv, 1);
        sxr[warp][k][lane] = smooth3(w0, w1, cl, cv, cr);
      }
    }
    qy1[j][warp][lane] = nw.a[1];
    qy2[j][warp][lane] = nw.c[1];
    __syncthreads();
    // axis 2 of plane p - 2, then the next plane in flight during the rest
    // of this step
    prev_a2 = nxt.a[2];
    prev_c2 = nxt.c[2];
    if (p + 1 <= z1) load_plane_q(Q1, Q2, V, (long long)(p + 1) * WH + col, in, nxt);
    // [B] y pass: smoothed certainty of plane p in the register window
    if (SMOOTH && warp >= 1 && warp <= 8) {
#pragma unroll
      for (int k = 0; k < 3; k++)
        cxr[SMOOTH ? j : 0][warp][k][lane] =
            smooth3(w0, w1, sxr[warp - 1][k][lane], sxr[warp][k][lane], sxr[warp + 1][k][lane]);
    }
    // [C] sums of output plane z = p - 1
    if (p >= z0 + 1) {
      const int z = p - 1;
      const float zf = (float)z - 0.5f * (float)(D - 1);
      // x neighbours of axis 0 from the adjacent lanes (all lanes shuffle)
      const float2 a0p = make_float2(__shfl_down_sync(0xffffffffu, cur.a[0].x, 1),
                                     __shfl_down_sync(0xffffffffu, cur.a[0].y, 1));
      const float2 c0p = make_float2(__shfl_down_sync(0xffffffffu, cur.c[0].x, 1),
                                     __shfl_down_sync(0xffffffffu, cur.c[0].y, 1));
      const float2 a0m = make_float2(__shfl_up_sync(0xffffffffu, cur.a[0].x, 1),
                                     __shfl_up_sync(0xffffffffu, cur.a[0].y, 1));
      const float2 c0m = make_float2(__shfl_up_sync(0xffffffffu, cur.c[0].x, 1),
                                     __shfl_up_sync(0xffffffffu, cur.c[0].y, 1));
      if (out) {
        float2 ap[3], am[3], cp[3], cm[3];
        ap[0] = a0p; am[0] = a0m; cp[0] = c0p; cm[0] = c0m;
        ap[1] = qy1[j1][warp + 1][lane]; am[1] = qy1[j1][warp - 1][lane];
        cp[1] = qy2[j1][warp + 1][lane]; cm[1] = qy2[j1][warp - 1][lane];
        ap[2] = nw.a[2]; am[2] = prev_a2; cp[2] = nw.c[2]; cm[2] = prev_c2;
#pragma unroll
        for (int k = 0; k < 3; k++) {
          float pd, cert;
          phase_diff_cert(cur.a[k], cur.c[k], pd, cert);
          const float g = phase_grad_rn(ap[k], cur.a[k], am[k], cp[k], cur.c[k], cm[k]);
          if (SMOOTH)
            cert = smooth3(w0, w1, cxr[SMOOTH ? j2 : 0][warp][k][lane], cxr[SMOOTH ? j1 : 0][warp][k][lane],
                           cxr[SMOOTH ? j : 0][warp][k][lane]);  // planes z - 1, z, z + 1
          const float cg = __fmul_rn(cert, g);
          const float wv = __fmul_rn(cg, g);
          const float vv = __fmul_rn(cg, pd);
          if (SPLIT) {
            float* t = s_wv + ((z - z0) * 6 + 2 * k) * kMarchThreads + threadIdx.x;
            t[0] = wv;
            t[kMarchThreads] = vv;
          } else {
            add_moments(m[k], wv, vv, zf);
          }
        }
      }
    }
    __syncthreads();  // sxr and the qy slot of plane p - 2 are rewritten next step
  };

  if (!empty) {
    for (int p = z0 - 1;; p += 3) {
      step(std::integral_constant<int, 0>(), p, pb0, pb1, pb2);
      if (p + 1 > z1) break;
      step(std::integral_constant<int, 1>(), p + 1, pb1, pb2, pb0);
      if (p + 2 > z1) break;
      step(std::integral_constant<int, 2>(), p + 2, pb2, pb0, pb1);
      if (p + 3 > z1) break;
    }
  }

  if (SPLIT) {
    cluster_sync();
    if (part == 0 && out) {
      for (int r = 0; r < np; r++) {
        const int za = z0 + r * gs, zb = min(zend, za + gs);
#pragma unroll 2
        for (int z = za; z < zb; z++) {
          const float zf = (float)z - 0.5f * (float)(D - 1);
          const float* t = s_wv + (z - za) * (6 * kMarchThreads) + threadIdx.x;
          float v[6];
#pragma unroll
          for (int q = 0; q < 6; q++) v[q] = cluster_load(t + q * kMarchThreads, r);
#pragma unroll
          for (int k = 0; k < 3; k++) add_moments(m[k], v[2 * k], v[2 * k + 1], zf);
        }
      }
    }
    __syncwarp();
    cluster_sync();  // no CTA leaves while its planes are read
    if (part != 0) return;
  }
  // FP64 sums over the row of a warp (y is the same for its lanes): nine
  // moments per axis, sum s0 [1, x, xx], sz [1, x], szz, v0 [1, x], vz.  The 27
  // sums over 32 lanes take one transposing tree of 31 exchanges (lane l ends
  // with sum l), not five shuffles per sum: the expansion of every lane into
  // the 42 sums and their shuffles cost as much as two and a half planes
  // (199 volumes of 64x64x33: 470 -> 437 us).
  const double xd = (double)xf;
  double red[32];
#pragma unroll
  for (int k = 0; k < 3; k++) {
    const double s0 = m[k][0], sz = m[k][1], v0 = m[k][3];
    red[9 * k] = s0;
    red[9 * k + 1] = xd * s0;
    red[9 * k + 2] = xd * xd * s0;
    red[9 * k + 3] = sz;
    red[9 * k + 4] = xd * sz;
    red[9 * k + 5] = m[k][2];
    red[9 * k + 6] = v0;
    red[9 * k + 7] = xd * v0;
    red[9 * k + 8] = m[k][4];
  }
#pragma unroll
  for (int i = kMarchRowSums; i < 32; i++) red[i] = 0.0;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const bool upper = (lane & o) != 0;
#pragma unroll
    for (int i = 0; i < o; i++) {
      const double send = upper ? red[i] : red[i + o];
      const double keep = upper ? red[i + o] : red[i];
      red[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
  if (lane < kMarchRowSums) s_part[warp][lane] = red[0];
  __syncthreads();
  // the 42 sums from the eight output rows, in order
  if (threadIdx.x < kNSums) {
    const int k = threadIdx.x / 14, e = threadIdx.x - 14 * k;
    const int q = 9 * k + c_row_moment[e], py = c_sum_ypow[e];
    double v = 0.0;
#pragma unroll
    for (int w = 1; w <= 8; w++) {
      const double yd = (double)(3 + yt * 8 - 1 + w) - 0.5 * (double)(H - 1);
      v = fma(s_part[w][q], py == 0 ? 1.0 : (py == 1 ? yd : yd * yd), v);
    }
    partials[((long long)b * nbx + bx) * kNSums + threadIdx.x] = v;
  }
}

// (row, column) of the 10 A entries of one axis, monomial order
// [1, x, y, z, xx, xy, xz, yy, yz, zz]; axis k owns parameters
// {k, 3+3k, 4+3k, 5+3k} (the GetParameterIndices table,
// kernelRegistration.cpp:43-171).
__constant__ int c_mono_a[10] = {0, 1, 2, 3, 1, 2, 3, 2, 3, 3};
__constant__ int c_mono_b[10] = {0, 0, 0, 0, 1, 1, 1, 2, 2, 3};

__device__ __forceinline__ int axis_param(int k, int m) { return m == 0 ? k : 2 + 3 * k + m; }

// Sums the nblk partial rows of instance b into s, in a fixed order: kRedSegs
// threads per sum take every kRedSegs-th row, then the segments are added in
// order.  (One thread per sum made this a chain of nblk dependent loads and
// adds: 48 us at the 972 rows of a 182x218x182 volume.)
constexpr int kRedSegs = 8;
constexpr int kSolveThreads = 352;  // kRedSegs x 42 sums, whole warps
__device__ void reduce_partials(const double* __restrict__ partials, int nblk, int b, double* s) {
  __shared__ double seg_sum[kRedSegs][kNSums];
  const int seg = threadIdx.x / kNSums, j = threadIdx.x - seg * kNSums;
  if (seg < kRedSegs) {
    double v = 0.0;
#pragma unroll 4
    for (int r = seg; r < nblk; r += kRedSegs) v += partials[((long long)b * nblk + r) * kNSums + j];
    seg_sum[seg][j] = v;
  }
  __syncthreads();
  if (threadIdx.x < kNSums) {
    double v = 0.0;
#pragma unroll
    for (int q = 0; q < kRedSegs; q++) v += seg_sum[q][threadIdx.x];
    s[threadIdx.x] = v;
  }
  __syncthreads();
}

// Full symmetric 12x12 A (column-major) and h of one instance.
__global__ void assemble_kernel(const double* __restrict__ partials, int nblk, double* __restrict__ A,
                                double* __restrict__ h) {
  __shared__ double s[kNSums];
  const int b = blockIdx.x;
  reduce_partials(partials, nblk, b, s);
  double* Ab = A + (long long)b * 144;
  for (int j = threadIdx.x; j < 144; j += blockDim.x) Ab[j] = 0.0;
  __syncthreads();
  if (threadIdx.x < 30) {
    const int k = threadIdx.x / 10, e = threadIdx.x % 10;
    const int i = axis_param(k, c_mono_a[e]), j = axis_param(k, c_mono_b[e]);
    Ab[i + 12 * j] = s[14 * k + e];
    Ab[j + 12 * i] = s[14 * k + e];
  } else if (threadIdx.x >= 32 && threadIdx.x < 44) {
    const int t = threadIdx.x - 32, k = t / 4, m = t % 4;
    h[(long long)b * 12 + axis_param(k, m)] = s[14 * k + 10 + m];
  }
}

// Solves the 4x4 block of an axis by Gaussian elimination with complete
// pivoting.  Pivots at or below `thresh` end the elimination and the
// remaining unknowns are 0, the rank rule of the reference's full-pivoting
// QR solve (SolveEquationSystem, broccoli_lib.cpp:17157-17186).  Every index
// is a constant and the exchanges are selections, so that the matrix stays
// in registers.
__device__ __forceinline__ void swap_if(bool c, double& a, double& b) {
  const double t = a;
  a = c ? b : a;
  b = c ? t : b;
}
__device__ __forceinline__ void solve4(double (&M)[4][4], double (&r)[4], double thresh, double (&x)[4]) {
  int perm[4] = {0, 1, 2, 3};
  int rank = 0;
  bool on = true;
#pragma unroll
  for (int k = 0; k < 4; k++) {
    int pr = k, pc = k;
    double best = -1.0;
#pragma unroll
    for (int i = k; i < 4; i++)
#pragma unroll
      for (int j = k; j < 4; j++) {
        const double m = fabs(M[i][j]);
        const bool more = m > best;
        best = more ? m : best;
        pr = more ? i : pr;
        pc = more ? j : pc;
      }
    on = on && !(best <= thresh || best == 0.0);
    if (!on) continue;
    rank = k + 1;
#pragma unroll
    for (int i = k + 1; i < 4; i++) {
      const bool sw = pr == i;
#pragma unroll
      for (int j = 0; j < 4; j++) swap_if(sw, M[k][j], M[i][j]);
      swap_if(sw, r[k], r[i]);
    }
#pragma unroll
    for (int j = k + 1; j < 4; j++) {
      const bool sw = pc == j;
#pragma unroll
      for (int i = 0; i < 4; i++) swap_if(sw, M[i][k], M[i][j]);
      const int t = perm[k];
      perm[k] = sw ? perm[j] : perm[k];
      perm[j] = sw ? t : perm[j];
    }
#pragma unroll
    for (int i = k + 1; i < 4; i++) {
      const double m = M[i][k] / M[k][k];
      if (m != 0.0) {
#pragma unroll
        for (int j = k; j < 4; j++) M[i][j] -= m * M[k][j];
        r[i] -= m * r[k];
      }
    }
  }
  double y[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
  for (int i = 3; i >= 0; i--) {
    if (i < rank) {
      double s = r[i];
#pragma unroll
      for (int j = i + 1; j < 4; j++)
        if (j < rank) s -= M[i][j] * y[j];
      y[i] = s / M[i][i];
    }
  }
#pragma unroll
  for (int q = 0; q < 4; q++) {
    double v = 0.0;
#pragma unroll
    for (int i = 0; i < 4; i++) v = perm[i] == q ? y[i] : v;
    x[q] = v;
  }
}

// The four parameters of axis k from the 42 sums, FP64, rounded to float (the
// reference casts its Eigen solution to float): one thread per axis.
__device__ __forceinline__ void solve_axis_from_sums(const double* s, int k, float* p) {
  double maxabs = 0.0;
  for (int j = 0; j < kNSums; j++)
    if ((j % 14) < 10) maxabs = fmax(maxabs, fabs(s[j]));
  const double thresh = maxabs * 2.220446049250313e-16 * 12.0;
  const double* e = s + 14 * k;
  double M[4][4] = {{e[0], e[1], e[2], e[3]}, {e[1], e[4], e[5], e[6]}, {e[2], e[5], e[7], e[8]}, {e[3], e[6], e[8], e[9]}};
  double r[4] = {e[10], e[11], e[12], e[13]}, x[4];
  solve4(M, r, thresh, x);
#pragma unroll
  for (int m = 0; m < 4; m++) p[axis_param(k, m)] = (float)x[m];
}

// Orthogonal polar factor U V^T of a 3x3 matrix (row-major) from one-sided
// Jacobi sweeps, FP64 (the reference takes U V^T of Eigen's JacobiSVD in
// RemoveTransformationScaling, broccoli_lib.cpp:6153-6194).
__device__ __forceinline__ void polar3(const double* M, double* R) {
  double A[9], Vm[9] = {1, 0, 0, 0, 1, 0, 0, 0, 1};
  for (int i = 0; i < 9; i++) A[i] = M[i];
  for (int sweep = 0; sweep < 60; sweep++) {
    bool rotated = false;
#pragma unroll
    for (int p = 0; p < 2; p++)
#pragma unroll
      for (int q = p + 1; q < 3; q++) {
        double al = 0, be = 0, ga = 0;
#pragma unroll
        for (int i = 0; i < 3; i++) {
          al += A[i * 3 + p] * A[i * 3 + p];
          be += A[i * 3 + q] * A[i * 3 + q];
          ga += A[i * 3 + p] * A[i * 3 + q];
        }
        if (fabs(ga) <= 1e-300 || fabs(ga) <= 2.220446049250313e-16 * sqrt(al * be)) continue;
        rotated = true;
        const double zeta = (be - al) / (2.0 * ga);
        const double t = (zeta >= 0 ? 1.0 : -1.0) / (fabs(zeta) + sqrt(1.0 + zeta * zeta));
        const double c = 1.0 / sqrt(1.0 + t * t), sn = c * t;
#pragma unroll
        for (int i = 0; i < 3; i++) {
          const double ap = A[i * 3 + p], aq = A[i * 3 + q];
          A[i * 3 + p] = c * ap - sn * aq;
          A[i * 3 + q] = sn * ap + c * aq;
          const double vp = Vm[i * 3 + p], vq = Vm[i * 3 + q];
          Vm[i * 3 + p] = c * vp - sn * vq;
          Vm[i * 3 + q] = sn * vp + c * vq;
        }
      }
    if (!rotated) break;
  }
  double U[9], sig[3];
#pragma unroll
  for (int j = 0; j < 3; j++) {
    sig[j] = sqrt(A[j] * A[j] + A[3 + j] * A[3 + j] + A[6 + j] * A[6 + j]);
    for (int i = 0; i < 3; i++) U[i * 3 + j] = sig[j] > 0 ? A[i * 3 + j] / sig[j] : 0.0;
  }
#pragma unroll
  for (int j = 0; j < 3; j++)
    if (!(sig[j] > 0)) {
      const int a = (j + 1) % 3, bb = (j + 2) % 3;
      U[0 * 3 + j] = U[1 * 3 + a] * U[2 * 3 + bb] - U[2 * 3 + a] * U[1 * 3 + bb];
      U[1 * 3 + j] = U[2 * 3 + a] * U[0 * 3 + bb] - U[0 * 3 + a] * U[2 * 3 + bb];
      U[2 * 3 + j] = U[0 * 3 + a] * U[1 * 3 + bb] - U[1 * 3 + a] * U[0 * 3 + bb];
    }
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = 0; j < 3; j++) {
      double s = 0;
      for (int k = 0; k < 3; k++) s += U[i * 3 + k] * Vm[j * 3 + k];
      R[i * 3 + j] = s;
    }
}

__device__ void remove_scaling(float* p) {
  double M[9], R[9];
  for (int i = 0; i < 9; i++) M[i] = (double)p[3 + i];
  M[0] += 1.0;
  M[4] += 1.0;
  M[8] += 1.0;
  polar3(M, R);
  R[0] -= 1.0;
  R[4] -= 1.0;
  R[8] -= 1.0;
  for (int i = 0; i < 9; i++) p[3 + i] = (float)R[i];
}

// Total = New * Old on 4x4 homogeneous matrices in FP64, the diagonal ones
// added in float first (AddAffineRegistrationParameters,
// broccoli_lib.cpp:7252-7340).
__device__ void compose(float* old12, const float* n12) {
  double O[16], N[16], T[16];
  const float* src[2] = {old12, n12};
  double* dst[2] = {O, N};
  for (int m = 0; m < 2; m++) {
    const float* p = src[m];
    double* Mt = dst[m];
    Mt[0] = (double)(p[3] + 1.0f); Mt[1] = (double)p[4]; Mt[2] = (double)p[5]; Mt[3] = (double)p[0];
    Mt[4] = (double)p[6]; Mt[5] = (double)(p[7] + 1.0f); Mt[6] = (double)p[8]; Mt[7] = (double)p[1];
    Mt[8] = (double)p[9]; Mt[9] = (double)p[10]; Mt[10] = (double)(p[11] + 1.0f); Mt[11] = (double)p[2];
    Mt[12] = 0; Mt[13] = 0; Mt[14] = 0; Mt[15] = 1;
  }
  for (int i = 0; i < 4; i++)
    for (int j = 0; j < 4; j++) {
      double s = 0;
      for (int k = 0; k < 4; k++) s += N[i * 4 + k] * O[k * 4 + j];
      T[i * 4 + j] = s;
    }
  old12[0] = (float)T[3];
  old12[1] = (float)T[7];
  old12[2] = (float)T[11];
  old12[3] = (float)(T[0] - 1.0); old12[4] = (float)T[1]; old12[5] = (float)T[2];
  old12[6] = (float)T[4]; old12[7] = (float)(T[5] - 1.0); old12[8] = (float)T[6];
  old12[9] = (float)T[8]; old12[10] = (float)T[9]; old12[11] = (float)(T[10] - 1.0);
}

// Euler angles in degrees (CalculateRotationAnglesFromRotationMatrix,
// broccoli_lib.cpp:6199-6244).
__device__ void rotation_angles(const float* p, float* rot) {
  const double PI_ = 3.14159265358979323846;
  double m[9];
  for (int i = 0; i < 9; i++) m[i] = (double)p[3 + i];
  m[0] += 1.0;
  m[4] += 1.0;
  m[8] += 1.0;
  const double a1 = -atan2(m[5], m[8]) * 180.0 / PI_;
  const double c2 = sqrt(m[0] * m[0] + m[1] * m[1]);
  const double a2 = -atan2(-m[2], c2) * 180.0 / PI_;
  const double s1 = sin(a1 * PI_ / 180.0), c1 = cos(a1 * PI_ / 180.0);
  const double a3 = -atan2(s1 * m[6] - c1 * m[3], c1 * m[4] - s1 * m[7]) * 180.0 / PI_;
  rot[0] = (float)a1;
  rot[1] = (float)a2;
  rot[2] = (float)a3;
}

// Largest displacement (voxels) of the update p over the 8 volume corners.
__device__ double update_magnitude(const float* p, int W, int H, int D) {
  const double hx = 0.5 * (W - 1), hy = 0.5 * (H - 1), hz = 0.5 * (D - 1);
  double best = 0.0;
#pragma unroll
  for (int c = 0; c < 8; c++) {
    const double x = (c & 1) ? hx : -hx, y = (c & 2) ? hy : -hy, z = (c & 4) ? hz : -hz;
    const double dx = p[0] + p[3] * x + p[4] * y + p[5] * z;
    const double dy = p[1] + p[6] * x + p[7] * y + p[8] * z;
    const double dz = p[2] + p[9] * x + p[10] * y + p[11] * z;
    best = fmax(best, dx * dx + dy * dy + dz * dz);
  }
  return sqrt(best);
}

// One iteration's solve and parameter update for every active instance
// (AlignTwoVolumesLinear, broccoli_lib.cpp:5380-5421), iteration it of
// act; instances whose update is not yet below tol go to list
// (it + 1) % 3, and list (it + 2) % 3 (the one iteration it - 1 used) is
// emptied for the next solve.
//
// Two blocks per SM: with the registers of one, the 199 instances of a series
// took two rounds (25 us a launch, 16 now).
__global__ void __launch_bounds__(kSolveThreads, 2)
solve_update_kernel(const double* __restrict__ partials, int nblk, int type,
                                    float tol, int W, int H, int D, float* __restrict__ params,
                                    float* __restrict__ rotations, int* __restrict__ conv_iter,
                                    int* __restrict__ iterations, int* __restrict__ status,
                                    const ActiveSet act, int* __restrict__ lists, int* __restrict__ counts) {
  __shared__ double s[kNSums];
  const int it = active_iteration(act);
  int* next_list = lists + ((it + 1) % 3) * act.stride;
  int* next_count = counts + (it + 1) % 3;
  if (blockIdx.x == 0 && threadIdx.x == 0) counts[(it + 2) % 3] = 0;
  if ((int)blockIdx.x >= active_count(act, (int)gridDim.x)) return;
  const int b = active_instance(act, blockIdx.x);
  __shared__ float s_p[12];
  reduce_partials(partials, nblk, b, s);
  // three warps, one axis each; then thread 0
  if ((threadIdx.x & 31) == 0 && threadIdx.x < 96) solve_axis_from_sums(s, threadIdx.x >> 5, s_p);
  __syncthreads();
  if (threadIdx.x != 0) return;
  float p[12];
#pragma unroll
  for (int i = 0; i < 12; i++) p[i] = s_p[i];
  bool finite = true;
  for (int i = 0; i < 12; i++) finite = finite && isfinite(p[i]);
  if (!finite) {
    for (int i = 0; i < 12; i++) p[i] = 0.f;
    if (status) atomicOr(status, 1);
  }
  float* tot = params + (long long)b * 12;
  float t[12];
  for (int i = 0; i < 12; i++) t[i] = tot[i];
  if (type == 0) {
    t[0] += p[0];
    t[1] += p[1];
    t[2] += p[2];
    for (int i = 3; i < 12; i++) t[i] = 0.f;
    for (int i = 3; i < 12; i++) p[i] = 0.f;
  } else if (type == 1) {
    remove_scaling(p);
    compose(t, p);
  } else {
    compose(t, p);
  }
  for (int i = 0; i < 12; i++) tot[i] = t[i];
  if (iterations) iterations[b] = it + 1;
  if (rotations && type == 1) rotation_angles(t, rotations + (long long)b * 3);
  const bool converged = tol > 0.f && update_magnitude(p, W, H, D) < (double)tol;
  if (converged && conv_iter != nullptr) conv_iter[b] = it;
  if (!converged) next_list[atomicAdd(next_count, 1)] = b;
}

// End of an iteration of the loop: advances the device iteration counter,
// and, when the loop runs as a graph's conditional WHILE node, sets its
// condition: another iteration while iterations remain and the list the
// solve just filled is not empty (then *iters_run counts the iteration).
__global__ void iteration_control_kernel(int* __restrict__ iter, const int* __restrict__ counts, int max_it,
                                         cudaGraphConditionalHandle cond, int use_cond,
                                         unsigned long long* __restrict__ iters_run) {
  const int next = *iter + 1;
  *iter = next;
  if (use_cond) {
    atomicAdd(iters_run, 1ull);
    cudaGraphSetConditional(cond, (next < max_it && counts[next % 3] > 0) ? 1u : 0u);
  }
}

__global__ void active_init_kernel(int* __restrict__ list0, int* __restrict__ counts, int batch) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < batch; i += gridDim.x * blockDim.x) list0[i] = i;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    counts[0] = batch;
    counts[1] = 0;
    counts[2] = 0;
  }
}

// Plain solve of given A/h (brc_solve_affine_fp64): A column-major 12x12.
__global__ void solve_given_kernel(const double* __restrict__ A, const double* __restrict__ h,
                                   float* __restrict__ p) {
  const int b = blockIdx.x;
  if (threadIdx.x != 0) return;
  const double* Ab = A + (long long)b * 144;
  const double* hb = h + (long long)b * 12;
  // The 12x12 of this path is block diagonal; solve it as a general 12x12
  // with complete pivoting so that any symmetric system is handled.
  double M[144], r[12], x[12];
  int perm[12];
  for (int i = 0; i < 12; i++) {
    r[i] = hb[i];
    perm[i] = i;
    for (int j = 0; j < 12; j++) M[i * 12 + j] = Ab[i + 12 * j];
  }
  double maxpiv = 0.0;
  int rank = 0;
  for (int k = 0; k < 12; k++) {
    int pr = k, pc = k;
    double best = -1.0;
    for (int i = k; i < 12; i++)
      for (int j = k; j < 12; j++)
        if (fabs(M[i * 12 + j]) > best) {
          best = fabs(M[i * 12 + j]);
          pr = i;
          pc = j;
        }
    if (k == 0) maxpiv = best;
    if (best <= maxpiv * 2.220446049250313e-16 * 12.0 || best == 0.0) break;
    rank++;
    if (pr != k) {
      for (int j = 0; j < 12; j++) {
        const double t = M[k * 12 + j];
        M[k * 12 + j] = M[pr * 12 + j];
        M[pr * 12 + j] = t;
      }
      const double t = r[k];
      r[k] = r[pr];
      r[pr] = t;
    }
    if (pc != k) {
      for (int i = 0; i < 12; i++) {
        const double t = M[i * 12 + k];
        M[i * 12 + k] = M[i * 12 + pc];
        M[i * 12 + pc] = t;
      }
      const int t = perm[k];
      perm[k] = perm[pc];
      perm[pc] = t;
    }
    for (int i = k + 1; i < 12; i++) {
      const double m = M[i * 12 + k] / M[k * 12 + k];
      if (m == 0.0) continue;
      for (int j = k; j < 12; j++) M[i * 12 + j] -= m * M[k * 12 + j];
      r[i] -= m * r[k];
    }
  }
  double y[12];
  for (int i = 0; i < 12; i++) y[i] = 0.0;
  for (int i = rank - 1; i >= 0; i--) {
    double s = r[i];
    for (int j = i + 1; j < rank; j++) s -= M[i * 12 + j] * y[j];
    y[i] = s / M[i * 12 + i];
  }
  for (int i = 0; i < 12; i++) x[perm[i]] = y[i];
  for (int i = 0; i < 12; i++) p[(long long)b * 12 + i] = (float)x[i];
}

// ---------------------------------------------------------------------------
// Trilinear sampling
// ---------------------------------------------------------------------------

// out_b(x) = src_b(x + t + (A - I)(x - centre)), params_b of instance b
// (InterpolateVolumeLinearLinear, kernelRegistration.cpp:1066-1101).
// VEC: params is 16-byte aligned, and the 12 parameters of an instance are
// read as three 16-byte loads.
//
// Bound by instruction issue (one voxel per thread: 84 % of the slots at 178
// instructions per warp and voxel row; LSU 44 %, DRAM 8 %).  A thread takes the same
// voxel of two planes: the instance's part and the x and y terms once, the
// positions and interpolations as packed pairs.  One plane to two, us:
// 199 x 64x64x33 135.0 -> 123.2-125.0, 59 x 80x80x37 88.3 -> 77.5-77.9, 24 x
// 64x64x33 22.9 -> 18.7, one 182x218x182 53.5 -> 39.2.  56 registers, four blocks
// per SM; five and six blocks are slower (130.6 and 139.5 us at the first size),
// as is clamping x alone where y and z are inside (121.8 us there, but 43.3 at
// 182x218x182).
template <bool VEC, int NZ>
__global__ void __launch_bounds__(256)
warp_affine_kernel(const float* __restrict__ src, long long src_stride, int W, int H, int D, int ntx, int batch,
                   const float* __restrict__ params, float* __restrict__ out, long long out_stride,
                   const ActiveSet act) {
  // block: 32 x 8 voxels of NZ planes, a voxel of each per thread; grid (x-y
  // tiles, groups of planes, a share of the instances: blockIdx.z, + gridDim.z, ...)
  const int ty = blockIdx.x / ntx, tx = blockIdx.x - ty * ntx;
  const int x = tx * 32 + threadIdx.x, y = ty * 8 + threadIdx.y, z = NZ * blockIdx.y;
  const bool on = (x < W) & (y < H);
  const unsigned mask = __ballot_sync(0xffffffffu, on);  // the sampler's lanes
  if (!on) return;
  const int z2 = min(z + 1, D - 1);
  const long long WH = (long long)W * H;
  const int n = active_count(act, batch);
  const int* list = act.list ? act.list + (active_iteration(act) % 3) * act.stride : nullptr;
  float* o = out + z * WH + (y * W + x);
  for (int li = blockIdx.z; li < n; li += gridDim.z) {
    const int b = list ? __ldg(list + li) : li;
    float p[12];
    if (VEC) {
      const float4* p4 = reinterpret_cast<const float4*>(params + (long long)b * 12);
#pragma unroll
      for (int q = 0; q < 3; q++) {
        const float4 v = __ldg(p4 + q);
        p[4 * q] = v.x;
        p[4 * q + 1] = v.y;
        p[4 * q + 2] = v.z;
        p[4 * q + 3] = v.w;
      }
    } else {
#pragma unroll
      for (int q = 0; q < 12; q++) p[q] = __ldg(params + (long long)b * 12 + q);
    }
    const float* s = src + (long long)b * src_stride;
    float* ob = o + (long long)b * out_stride;
    if constexpr (NZ == 2) {
      const float2 r = affine_sample_pair(s, W, H, D, p, x, y, z, z2, mask);
      ob[0] = r.x;
      if (z + 1 < D) ob[WH] = r.y;
    } else {
      ob[0] = affine_sample(s, W, H, D, p, x, y, z, mask);
    }
  }
}

// Displacement-field warp (InterpolateVolumeLinearNonLinear,
// kernelRegistration.cpp:1111-1140).
__global__ void __launch_bounds__(256)
warp_field_kernel(const float* __restrict__ src, int W, int H, int D, const float* __restrict__ dx,
                  const float* __restrict__ dy, const float* __restrict__ dz, float* __restrict__ out,
                  long long src_stride, long long field_stride, long long out_stride) {
  const int V = W * H * D;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const unsigned mask = __ballot_sync(0xffffffffu, i < V);  // the sampler's lanes
  if (i >= V) return;
  // instance blockIdx.y
  const long long b = blockIdx.y;
  src += b * src_stride;
  dx += b * field_stride;
  dy += b * field_stride;
  dz += b * field_stride;
  out += b * out_stride;
  int x, y, z;
  voxel_of(i, W, H, x, y, z);
  out[i] = sample_linear(src, W, H, D, (float)x + dx[i] + 0.5f, (float)y + dy[i] + 0.5f,
                         (float)z + dz[i] + 0.5f, mask);
}

// Linear resample with spacing (N-1)/(N'-1) (RescaleVolumeLinear,
// kernelRegistration.cpp:1340-1366).
__global__ void __launch_bounds__(256)
rescale_linear_kernel(const float* __restrict__ src, int W, int H, int D, float* __restrict__ out,
                      int W2, int H2, int D2, float vx, float vy, float vz) {
  const int V2 = W2 * H2 * D2;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const unsigned mask = __ballot_sync(0xffffffffu, i < V2);  // the sampler's lanes
  if (i >= V2) return;
  int x, y, z;
  voxel_of(i, W2, H2, x, y, z);
  out[i] = sample_linear(src, W, H, D, x * vx + 0.5f, y * vy + 0.5f, z * vz + 0.5f, mask);
}

// ---------------------------------------------------------------------------
// Separable 9-tap smoothing (three passes)
// ---------------------------------------------------------------------------

// The three separable 9-tap passes in one kernel: y over (vol * cert), then
// x, then z, divided by the smoothed certainty (SeparableConvolutionRows /
// Columns / Rods, kernelConvolution.cpp:52-91, :531-569, :1201-1240, zero
// padding).  Each output is the same sequence of terms as three separate
// passes (o = -4..4 in order, out-of-volume terms 0), and the volume is read
// from HBM once and written once.
//
// A block owns a column tile of up to 32 x 8 outputs and marches along z
// through a chunk of planes, eight planes (a group) at a time:
//   y  a thread takes one pair of window columns of a plane: sixteen 8-byte
//      loads straight from global memory, 72 packed FMAs, eight 8-byte stores
//      to the shared y buffer;
//   x  a thread takes eight consecutive outputs of a row: four 16-byte
//      shared loads, 36 packed FMAs on aligned and shifted pairs, two 16-byte
//      stores into a ring of sixteen planes.  Its lanes run along the rows,
//      whose pitches (12 and 4 modulo 32 banks) keep the 16-byte accesses
//      free of conflicts;
//   z  a thread takes one column pair: sixteen 8-byte loads from the ring, the
//      eight output planes of the group in 72 packed FMAs, stored coalesced.
// The z pass of a group runs in the same interval as the y pass of the next,
// so a group has two barriers.  What a thread works on is decoded once: the
// groups differ only by the plane offset.  This layout is for instruction
// issue, which bounds the kernel: a form with a shared-memory window per
// plane and a register ring for z issued 109 thread instructions per voxel
// for its 27 FMAs.  Packed FP32 FMAs (two lanes per instruction, rounded as
// two scalar ones) halve the issue slots of the arithmetic.
// Measured (CUDA events, passes back to back): 9 volumes of 182x218x182 278 ->
// 168 us (3.1 TB/s; 172-174 with the inputs of several passes in turn, 188 for a
// pass that starts on an idle GPU),
// 9 of 91x109x91 (odd width) 59 -> 36 us, 200 of 64x64x33 175 -> 73 us (3.0
// TB/s), the same with certainty, division and mask product in the kernel
// 360 -> 160 us.  Tiles of 64 columns with 288 threads: 174, 37, 73, 173 us
// (fewer, larger blocks wait longer at a group's barriers); 48 columns 182, 40,
// 83, 218.
// `out` must not overlap the inputs.
constexpr int kSmTX = 32, kSmTY = 8;    // largest output tile (the width is chosen per volume)
constexpr int kSmG = 8;                 // planes per group
constexpr int kSmThreads = 160;         // y units of a 32-wide tile: 20 column pairs x 8 planes
constexpr int kSmPY = kSmTX + 12;       // y buffer pitch: 44 floats, 12 modulo 32
constexpr int kSmPR = kSmTX + 4;        // ring pitch: 36 floats, 4 modulo 32
constexpr int kSmYPlane = kSmTY * kSmPY, kSmRPlane = kSmTY * kSmPR;
constexpr int kSmRGroup = kSmG * kSmRPlane;
constexpr size_t kSmSmem = sizeof(float) * (kSmG * kSmYPlane + 2 * kSmRGroup);
static_assert(kSmTY == 8 && kSmG == 8, "the unit decodes assume 8 rows and groups of 8 planes");
static_assert(kSmSmem <= 48 * 1024, "more needs a function attribute on every device");

// The taps of the three passes, each twice (both lanes of a packed FMA), in
// the order of the samples (o = -4..4 meets taps 8..0).
struct SmoothTaps {
  F2 x[9], y[9], z[9];
};

// Output width of a block's tile: W in equal parts of at most 32, rounded up to
// whole octets of the x pass.
__host__ __device__ inline int smooth_tile_width(int W) {
  const int n = (W + kSmTX - 1) / kSmTX;
  return ((W + n - 1) / n + 7) / 8 * 8;
}

// VEC: pairs move as 8 bytes (an even W, so that no pair straddles the edge,
// and 8-byte aligned volumes); DIV: divide by the smoothed certainty scert;
// MUL: then multiply by the certainty; ACC: add into `out`.
template <bool CERT, bool VEC, bool DIV, bool MUL, bool ACC>
// Five blocks per SM where pairs move and there is no certainty (of these the two
// that divide spill 12 bytes); the certainty forms take four (194 us with five,
// 160 with four), and so do single accesses.
__global__ void __launch_bounds__(kSmThreads, VEC && !CERT ? 5 : 4)
smooth3d_kernel(const float* __restrict__ in, const float* __restrict__ cert, const float* __restrict__ scert,
                int W, int H, int D, int tw, int zc, const __grid_constant__ SmoothTaps taps,
                float* __restrict__ out) {
  extern __shared__ __align__(16) float smem[];
  float* s_y = smem;                       // [8 planes][8 rows][kSmPY]
  float* s_r = smem + kSmG * kSmYPlane;    // [2 groups][8 planes][8 rows][kSmPR]
  const int tid = threadIdx.x;
  const int ntx = (W + tw - 1) / tw;
  const int x0 = (int)(blockIdx.x % ntx) * tw, y0 = (int)(blockIdx.x / ntx) * kSmTY;
  const int z0 = blockIdx.y * zc, z1 = min(D, z0 + zc);
  const int ngroups = (z1 - z0 + 8 + kSmG - 1) / kSmG;
  const int WH = W * H;
  const float* src = in + (long long)blockIdx.z * WH * D;
  float* dst = out + (long long)blockIdx.z * WH * D;

  // y unit: plane yp of the group, window rows y0 - 4 .. y0 + 11, columns gx, gx + 1
  const int ncp = (tw + 8) / 2;
  const int yp = tid / ncp, yc = tid - yp * ncp;
  const int gx = x0 - 4 + 2 * yc, gy = y0 - 4;
  unsigned rows = 0;  // window rows inside the volume
#pragma unroll
  for (int i = 0; i < 16; i++)
    if (gy + i >= 0 && gy + i < H) rows |= 1u << i;
  const bool in0 = gx >= 0 && gx < W, in1 = gx + 1 >= 0 && gx + 1 < W;
  if ((!in0 && !in1) || yp >= kSmG) rows = 0;
  const int yoff = gy * W + gx;  // in-plane offset of the first row (rows outside are not loaded)
  float* const yb = s_y + yp * kSmYPlane + 2 * yc;
  auto load = [&](const float* __restrict__ p, F2 (&a)[16]) {
    const float* q = p + yoff;
    if (VEC && rows == 0xffffu) {
#pragma unroll
      for (int i = 0; i < 16; i++) a[i] = __ldg(reinterpret_cast<const F2*>(q + i * W));
    } else {
#pragma unroll
      for (int i = 0; i < 16; i++) {
        float2 v = make_float2(0.f, 0.f);
        if ((rows >> i) & 1u) {
          if (VEC) {
            v = __ldg(reinterpret_cast<const float2*>(q + i * W));
          } else {
            if (in0) v.x = __ldg(q + i * W);
            if (in1) v.y = __ldg(q + i * W + 1);
          }
        }
        a[i] = f2_pack(v.x, v.y);
      }
    }
  };
  // x units: row (lanes along the rows), plane and octet; at most two per thread
  const int noct = tw / 8, nx = kSmG * kSmTY * noct;
  int xp[2], xs[2], xd[2];
#pragma unroll
  for (int k = 0; k < 2; k++) {
    const int u = tid + k * kSmThreads, row = u & 7, t = u >> 3;
    const int pl = t / noct, oct = t - pl * noct;
    xp[k] = u < nx ? pl : -1;
    xs[k] = pl * kSmYPlane + row * kSmPY + 8 * oct;
    xd[k] = pl * kSmRPlane + row * kSmPR + 8 * oct;
  }
  // z unit: one column pair of a row
  const int ncz = tw / 2, zrow = tid / ncz, zcol = tid - zrow * ncz;
  const int zx = x0 + 2 * zcol, zy = y0 + zrow;
  const bool zon = zrow < kSmTY && zx < W && zy < H;
  const bool two = VEC || zx + 1 < W;
  const float* const zb = s_r + zrow * kSmPR + 2 * zcol;

  // the group's z pass: chunk planes 8 (g - 1) .. 8 g + 7 sit in ring halves
  // (g + 1) & 1 and g & 1; output plane i of the group sums planes i .. i + 8
  // of those sixteen
  auto zpass = [&](int g) {
    if (!zon) return;
    const int zo = z0 + kSmG * (g - 1);
    F2 a[16];
    const float* r0 = zb + ((g + 1) & 1) * kSmRGroup;
    const float* r1 = zb + (g & 1) * kSmRGroup;
#pragma unroll
    for (int i = 0; i < 8; i++) {
      a[i] = *reinterpret_cast<const F2*>(r0 + i * kSmRPlane);
      a[8 + i] = *reinterpret_cast<const F2*>(r1 + i * kSmRPlane);
    }
    int o = zo * WH + zy * W + zx;
#pragma unroll
    for (int i = 0; i < kSmG; i++, o += WH) {
      if (zo + i < z1) {
        F2 sum = 0;
#pragma unroll
        for (int j = 0; j < 9; j++) sum = f2_fma(a[i + j], taps.z[j], sum);
        float2 v = f2_unpack(sum);
        if (DIV) {
          v.x = v.x / __ldg(scert + o);
          if (two) v.y = v.y / __ldg(scert + o + 1);
        }
        if (MUL) {
          v.x *= __ldg(cert + o);
          if (two) v.y *= __ldg(cert + o + 1);
        }
        if (VEC) {
          float2* d = reinterpret_cast<float2*>(dst + o);
          if (ACC) {
            const float2 old = *d;
            v.x = old.x + v.x;
            v.y = old.y + v.y;
          }
          *d = v;
        } else {
          dst[o] = ACC ? dst[o] + v.x : v.x;
          if (two) dst[o + 1] = ACC ? dst[o + 1] + v.y : v.y;
        }
      }
    }
  };

  for (int g = 0; g <= ngroups; g++) {
    // the z pass of the group before, then this group's loads and y pass
    const int p = z0 - 4 + kSmG * g + yp;
    const bool yin = g < ngroups && yp < kSmG && p >= 0 && p < D;
    F2 a[16];
    if (g >= 2) zpass(g - 1);
    if (yin) {
      load(src + (long long)p * WH, a);
      if (CERT) {
        F2 w[16];
        load(cert + (long long)p * WH, w);
#pragma unroll
        for (int i = 0; i < 16; i++) a[i] = f2_mul(a[i], w[i]);
      }
    }
    if (g == ngroups) break;
    if (yin) {
#pragma unroll
      for (int i = 0; i < 8; i++) {
        F2 sum = 0;
#pragma unroll
        for (int j = 0; j < 9; j++) sum = f2_fma(a[i + j], taps.y[j], sum);
        *reinterpret_cast<F2*>(yb + i * kSmPY) = sum;
      }
    }
    __syncthreads();
    // x pass into ring half g & 1 (planes outside the volume: zeros)
    float* const ring = s_r + (g & 1) * kSmRGroup;
#pragma unroll
    for (int k = 0; k < 2; k++) {
      if (xp[k] >= 0) {
        const int zp = z0 - 4 + kSmG * g + xp[k];
        F2 s[4] = {0, 0, 0, 0};
        if (zp >= 0 && zp < D) {
          const ulonglong2* r = reinterpret_cast<const ulonglong2*>(s_y + xs[k]);
          F2 e[8], o[7];
#pragma unroll
          for (int q = 0; q < 4; q++) {
            const ulonglong2 v = r[q];
            e[2 * q] = v.x;
            e[2 * q + 1] = v.y;
          }
#pragma unroll
          for (int q = 0; q < 7; q++) o[q] = f2_pack(f2_unpack(e[q]).y, f2_unpack(e[q + 1]).x);
#pragma unroll
          for (int j = 0; j < 9; j++)
#pragma unroll
            for (int q = 0; q < 4; q++) s[q] = f2_fma(j % 2 == 0 ? e[q + j / 2] : o[q + j / 2], taps.x[j], s[q]);
        }
        ulonglong2* d = reinterpret_cast<ulonglong2*>(ring + xd[k]);
        d[0] = make_ulonglong2(s[0], s[1]);
        d[1] = make_ulonglong2(s[2], s[3]);
      }
    }
    __syncthreads();
  }
}

// Planes per z chunk of smooth3d_kernel: enough chunks that the grid fills
// the 148 SMs about six blocks deep, at least 16 planes per chunk.
static int smooth_chunk(int D, long long tiles_x_batch) {
  const long long want = 148LL * 6;
  long long chunks = (want + tiles_x_batch - 1) / tiles_x_batch;
  const long long maxc = (D + 15) / 16;
  if (chunks > maxc) chunks = maxc;
  if (chunks < 1) chunks = 1;
  return (int)((D + chunks - 1) / chunks);
}

// ---------------------------------------------------------------------------
// Host launchers
// ---------------------------------------------------------------------------

cudaError_t normal_eq_partials(const float* q1, long long q1_stride_floats, const float* q2, int W,
                               int H, int D, int batch, double* partials, int nblk, int zpb, cudaStream_t st) {
  dim3 grid(nblk, batch);
  normal_eq_partial_kernel<<<grid, kNEThreads, 0, st>>>(
      reinterpret_cast<const float2*>(q1), q1_stride_floats / 2, reinterpret_cast<const float2*>(q2),
      W, H, D, zpb, partials);
  return cudaGetLastError();
}

int normal_eq_march_blocks(int W, int H, int D, int* ntx, int* nty, int* zs) {
  const int nx = W - 6, ny = H - 6, nz = D - 6;
  *ntx = nx > 0 ? (nx + kMarchCols - 1) / kMarchCols : 1;
  *nty = ny > 0 ? (ny + 7) / 8 : 1;
  const int nzs = nz > 0 ? (nz + kMarchZs - 1) / kMarchZs : 1;
  *zs = nz > 0 ? (nz + nzs - 1) / nzs : 0;
  return *ntx * *nty * nzs;
}

// CTAs that share a slab: the most, up to a cluster's 8 and with six planes or more each,
// that all run at once (two per SM); 1 where they would not.  Such a launch is a
// chain of plane steps, which the parts shorten (one 64x64x33 volume: 16 CTAs of
// 29 steps, or 80 of 8; 20 iterations 952 -> 827 us, with four planes each 835);
// a larger one fills the chip with whole slabs, which step over two halo planes
// once and not per part.
static int march_parts(long long blocks, int zs) {
  for (int np = 8; np > 1; np--) {
    const int gs = (zs + np - 1) / np;
    if (gs >= 6 && gs <= kMarchMaxGs && (np - 1) * gs < zs && blocks * np <= 2 * 148) return np;
  }
  return 1;
}

template <bool SMOOTH, bool SPLIT>
static cudaError_t launch_march(const float2* q1, long long q1_stride, const float2* q2, int W, int H, int D, int ntx,
                                int nty, int nblk, int zs, int np, int batch, double* partials, ActiveSet act,
                                float w0, float w1, cudaStream_t st) {
  const int gs = SPLIT ? (zs + np - 1) / np : zs;
  const size_t plane = sizeof(float) * 6 * kMarchThreads;
  if (SPLIT) {
    // shared memory above 48 KB is a per-device function attribute
    static bool attr_set[64] = {false};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    if (!attr_set[dev]) {
      const cudaError_t e = cudaFuncSetAttribute(normal_eq_march_kernel<SMOOTH, SPLIT>,
                                                 cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 (int)(plane * kMarchMaxGs));
      if (e != cudaSuccess) return e;
      attr_set[dev] = true;
    }
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(nblk * np), (unsigned)batch);
  cfg.blockDim = dim3(kMarchThreads);
  cfg.dynamicSmemBytes = SPLIT ? plane * gs : 0;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)np;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = SPLIT ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, normal_eq_march_kernel<SMOOTH, SPLIT>, q1, q1_stride, q2, W, H, D, ntx, nty, zs, gs,
                            np, partials, act, w0, w1);
}

cudaError_t normal_eq_march(const float* q1, long long q1_stride_floats, const float* q2, int W, int H, int D,
                            int batch, double* partials, int nblk, ActiveSet act, cudaStream_t st,
                            float cert_sigma) {
  int ntx, nty, zs;
  if (normal_eq_march_blocks(W, H, D, &ntx, &nty, &zs) != nblk) return cudaErrorInvalidValue;
  const float2* a = reinterpret_cast<const float2*>(q1);
  const float2* c = reinterpret_cast<const float2*>(q2);
  const int np = march_parts((long long)nblk * batch, zs);
  // 3-tap Gaussian of the certainties, weights normalised to sum 1
  float w0 = 1.f, w1 = 0.f;
  if (cert_sigma > 0.f) {
    const float e = (float)exp(-1.0 / (2.0 * (double)cert_sigma * (double)cert_sigma));
    w0 = 1.0f / (1.0f + 2.0f * e);
    w1 = e * w0;
  }
  const auto launch = [&](auto smooth, auto split) {
    return launch_march<decltype(smooth)::value, decltype(split)::value>(
        a, q1_stride_floats / 2, c, W, H, D, ntx, nty, nblk, zs, np, batch, partials, act, w0, w1, st);
  };
  if (cert_sigma > 0.f)
    return np > 1 ? launch(std::true_type(), std::true_type()) : launch(std::true_type(), std::false_type());
  return np > 1 ? launch(std::false_type(), std::true_type()) : launch(std::false_type(), std::false_type());
}

cudaError_t assemble_normal_eq(const double* partials, int nblk, int batch, double* A, double* h,
                               cudaStream_t st) {
  assemble_kernel<<<batch, kSolveThreads, 0, st>>>(partials, nblk, A, h);
  return cudaGetLastError();
}

cudaError_t solve_update(const double* partials, int nblk, int batch, int type, float tol, int W,
                         int H, int D, float* params, float* rotations, int* conv_iter,
                         int* iterations, int* status, ActiveSet act, int* lists, int* counts, cudaStream_t st) {
  if (!act.list) return cudaErrorInvalidValue;
  solve_update_kernel<<<batch, kSolveThreads, 0, st>>>(partials, nblk, type, tol, W, H, D, params, rotations,
                                            conv_iter, iterations, status, act, lists, counts);
  return cudaGetLastError();
}

cudaError_t iteration_control(int* iter, const int* counts, int max_it, cudaGraphConditionalHandle cond,
                              bool use_cond, unsigned long long* iters_run, cudaStream_t st) {
  iteration_control_kernel<<<1, 1, 0, st>>>(iter, counts, max_it, cond, use_cond ? 1 : 0, iters_run);
  return cudaGetLastError();
}

cudaError_t active_init(int* list0, int* counts, int batch, cudaStream_t st) {
  active_init_kernel<<<(batch + 255) / 256, 256, 0, st>>>(list0, counts, batch);
  return cudaGetLastError();
}

cudaError_t solve_given(const double* A, const double* h, int batch, float* p, cudaStream_t st) {
  solve_given_kernel<<<batch, 32, 0, st>>>(A, h, p);
  return cudaGetLastError();
}

cudaError_t warp_affine(const float* src, long long src_stride, int W, int H, int D, int batch,
                        const float* params, float* out, long long out_stride, ActiveSet act,
                        cudaStream_t st) {
  const long long V = (long long)W * H * D;
  if (V > kMaxVoxels) return cudaErrorInvalidValue;
  if (D > 65535 || batch > 65535 || batch <= 0) return cudaErrorInvalidValue;
  const int ntx = (W + 31) / 32, nty = (H + 7) / 8;
  // at most 16 instance shares: a launch whose instances have mostly
  // converged does not pay for blocks with nothing to do
  const int shares = batch < 16 ? batch : 16;
  // Two planes per thread where their blocks fill the chip (four per SM are
  // resident); a smaller launch is as long as its busiest SM's chain, and half
  // the blocks are spread less evenly (one 64x64x33: a registration of 20 such
  // launches 767 us with two planes per thread, 762 with one).
  const bool two = (long long)ntx * nty * ((D + 1) / 2) * shares >= 4 * 148;
  const bool vec = (reinterpret_cast<uintptr_t>(params) & 15) == 0;
  dim3 grid((unsigned)(ntx * nty), (unsigned)(two ? (D + 1) / 2 : D), (unsigned)shares);
  auto* k = two ? (vec ? warp_affine_kernel<true, 2> : warp_affine_kernel<false, 2>)
                : (vec ? warp_affine_kernel<true, 1> : warp_affine_kernel<false, 1>);
  k<<<grid, dim3(32, 8), 0, st>>>(src, src_stride, W, H, D, ntx, batch, params, out, out_stride, act);
  return cudaGetLastError();
}

cudaError_t warp_field(const float* src, int W, int H, int D, const float* dx, const float* dy,
                       const float* dz, float* out, cudaStream_t st, int batch, long long src_stride,
                       long long field_stride, long long out_stride) {
  const long long V = (long long)W * H * D;
  if (V > kMaxVoxels || batch <= 0 || batch > 65535) return cudaErrorInvalidValue;
  warp_field_kernel<<<dim3((unsigned)((V + 255) / 256), (unsigned)batch), 256, 0, st>>>(
      src, W, H, D, dx, dy, dz, out, src_stride, field_stride, out_stride);
  return cudaGetLastError();
}

cudaError_t rescale_linear(const float* src, int W, int H, int D, float* out, int W2, int H2, int D2,
                           cudaStream_t st) {
  const long long V2 = (long long)W2 * H2 * D2;
  if (V2 > kMaxVoxels || (long long)W * H * D > kMaxVoxels) return cudaErrorInvalidValue;
  const float vx = (float)(W - 1) / (float)(W2 - 1);
  const float vy = (float)(H - 1) / (float)(H2 - 1);
  const float vz = (float)(D - 1) / (float)(D2 - 1);
  rescale_linear_kernel<<<(unsigned)((V2 + 255) / 256), 256, 0, st>>>(src, W, H, D, out, W2, H2, D2,
                                                                     vx, vy, vz);
  return cudaGetLastError();
}

// vols[b][i] *= mask[i] for every volume b (MultiplyVolumes,
// kernelMisc.cpp, as PerformSmoothingNormalized ends, broccoli_lib.cpp:11359-11450).
__global__ void __launch_bounds__(256)
multiply_mask_kernel(float* __restrict__ vols, const float* __restrict__ mask, long long V) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= V) return;
  vols[(long long)blockIdx.y * V + i] *= __ldg(mask + i);
}

__global__ void phase_atan2_kernel(const float* __restrict__ y, const float* __restrict__ x,
                                   float* __restrict__ out, long long n) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    out[i] = phase_atan2(y[i], x[i]);
}

// The reference's linear phase quantities of one filter pair, volume by
// volume (CalculatePhaseDifferencesAndCertainties, CalculatePhaseGradients
// X/Y/Z, kernelRegistration.cpp:173-382), with the library's own atan2f,
// cosf and sqrtf and no contraction into FMAs (the reference's order of
// operations).  Used for the debug outputs, not in the registration loop.
__global__ void __launch_bounds__(256)
phase_volumes_kernel(const float2* __restrict__ q1, const float2* __restrict__ q2, int W, int H, int D, int axis,
                     float* __restrict__ pd, float* __restrict__ cert, float* __restrict__ grad) {
  const long long V = (long long)W * H * D;
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= V) return;
  if (pd || cert) {
    const float2 a = q1[i], c = q2[i];
    const float re = __fadd_rn(__fmul_rn(a.x, c.x), __fmul_rn(a.y, c.y));
    const float im = __fsub_rn(__fmul_rn(a.y, c.x), __fmul_rn(a.x, c.y));
    const float d = atan2f(im, re);
    if (pd) pd[i] = d;
    if (cert) {
      const float pr = __fsub_rn(__fmul_rn(a.x, c.x), __fmul_rn(a.y, c.y));
      const float pi = __fadd_rn(__fmul_rn(a.y, c.x), __fmul_rn(a.x, c.y));
      const float cc = cosf(__fmul_rn(d, 0.5f));
      cert[i] = __fmul_rn(__fmul_rn(sqrtf(__fadd_rn(__fmul_rn(pr, pr), __fmul_rn(pi, pi))), cc), cc);
    }
  }
  if (grad) {
    int x, y, z;
    voxel_of(i, W, H, x, y, z);
    const int c = axis == 0 ? x : (axis == 1 ? y : z);
    const int n = axis == 0 ? W : (axis == 1 ? H : D);
    const long long step = axis == 0 ? 1 : (axis == 1 ? (long long)W : (long long)W * H);
    if (c - 1 < 0 || c + 1 >= n) {
      grad[i] = 0.f;
      return;
    }
    float tr = 0.f, ti = 0.f;
    const float2* qs[2] = {q1, q2};
#pragma unroll
    for (int k = 0; k < 2; k++) {
      const float2 p = qs[k][i + step], o = qs[k][i], m = qs[k][i - step];
      tr = __fadd_rn(tr, __fadd_rn(__fmul_rn(p.x, o.x), __fmul_rn(p.y, o.y)));
      ti = __fadd_rn(ti, __fsub_rn(__fmul_rn(p.y, o.x), __fmul_rn(p.x, o.y)));
      tr = __fadd_rn(tr, __fadd_rn(__fmul_rn(o.x, m.x), __fmul_rn(o.y, m.y)));
      ti = __fadd_rn(ti, __fsub_rn(__fmul_rn(o.y, m.x), __fmul_rn(o.x, m.y)));
    }
    grad[i] = atan2f(ti, tr);
  }
}

cudaError_t phase_volumes(const float* q1, const float* q2, int W, int H, int D, int axis, float* pd, float* cert,
                          float* grad, cudaStream_t st) {
  const long long V = (long long)W * H * D;
  if (V <= 0 || V > kMaxVoxels || axis < 0 || axis > 2) return cudaErrorInvalidValue;
  phase_volumes_kernel<<<(unsigned)((V + 255) / 256), 256, 0, st>>>(reinterpret_cast<const float2*>(q1),
                                                                   reinterpret_cast<const float2*>(q2), W, H, D,
                                                                   axis, pd, cert, grad);
  return cudaGetLastError();
}

cudaError_t phase_atan2_eval(const float* y, const float* x, float* out, long long n, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  const long long nb = (n + 255) / 256;
  phase_atan2_kernel<<<(unsigned)(nb < 148 * 16 ? nb : 148 * 16), 256, 0, st>>>(y, x, out, n);
  return cudaGetLastError();
}

cudaError_t multiply_mask(float* vols, const float* mask, long long V, int batch, cudaStream_t st) {
  dim3 grid((unsigned)((V + 255) / 256), batch);
  multiply_mask_kernel<<<grid, 256, 0, st>>>(vols, mask, V);
  return cudaGetLastError();
}

// smooth3d_kernel instantiations indexed by (cert << 3) | (pairs << 2) |
// (divide << 1) | accumulate, then the two of the normalised smoothing
// (certainty, division, product with the certainty) by pairs.
static const void* smooth_kernel_of(int v) {
#define BRC_SK(C, P, Q, M, A) reinterpret_cast<const void*>(smooth3d_kernel<C, P, Q, M, A>)
  static const void* const table[18] = {
      BRC_SK(false, false, false, false, false), BRC_SK(false, false, false, false, true),
      BRC_SK(false, false, true, false, false),  BRC_SK(false, false, true, false, true),
      BRC_SK(false, true, false, false, false),  BRC_SK(false, true, false, false, true),
      BRC_SK(false, true, true, false, false),   BRC_SK(false, true, true, false, true),
      BRC_SK(true, false, false, false, false),  BRC_SK(true, false, false, false, true),
      BRC_SK(true, false, true, false, false),   BRC_SK(true, false, true, false, true),
      BRC_SK(true, true, false, false, false),   BRC_SK(true, true, false, false, true),
      BRC_SK(true, true, true, false, false),    BRC_SK(true, true, true, false, true),
      BRC_SK(true, false, true, true, false),    BRC_SK(true, true, true, true, false)};
#undef BRC_SK
  return table[v];
}

static long long smooth_tiles(int W, int H) {
  const int tw = smooth_tile_width(W);
  return (long long)((W + tw - 1) / tw) * ((H + kSmTY - 1) / kSmTY);
}

int smooth3d_default_chunk(int W, int H, int D, int batch) {
  return smooth_chunk(D, smooth_tiles(W, H) * batch);
}

int smooth3d_chunk_candidates(int D, int* zc, int max_n) {
  // D split into 1, 2, 3, 4, 6 or 8 chunks of at least 8 planes
  static const int parts[] = {1, 2, 3, 4, 6, 8};
  int n = 0;
  for (int c : parts) {
    const int z = (D + c - 1) / c;
    if (n >= max_n || (c > 1 && z < 8)) break;
    if (n == 0 || zc[n - 1] != z) zc[n++] = z;
  }
  return n;
}

cudaError_t smooth3d(const float* vol, int W, int H, int D, int batch, const float* fx,
                     const float* fy, const float* fz, const float* cert, const float* scert,
                     float* tmp1, float* tmp2, float* out, cudaStream_t st, int accumulate, int zchunk,
                     bool times_cert) {
  const long long V = (long long)W * H * D;
  SmoothTaps taps;
  for (int i = 0; i < 9; i++) {
    taps.x[i] = f2_twice(fx[8 - i]);
    taps.y[i] = f2_twice(fy[8 - i]);
    taps.z[i] = f2_twice(fz[8 - i]);
  }
  if (times_cert && (!cert || !scert || accumulate)) return cudaErrorInvalidValue;
  (void)tmp2;  // the fused kernel needs no second temporary
  // an output overlapping an input is computed into tmp1, then moved
  const size_t bytes = sizeof(float) * (size_t)V * batch;
  auto overlaps = [&](const float* a, size_t na) {
    const char *o0 = reinterpret_cast<const char*>(out), *a0 = reinterpret_cast<const char*>(a);
    return a != nullptr && o0 < a0 + na && a0 < o0 + bytes;
  };
  const bool alias = overlaps(vol, bytes) || overlaps(cert, sizeof(float) * (size_t)V) ||
                     overlaps(scert, sizeof(float) * (size_t)V);
  float* dst = alias ? tmp1 : out;
  const long long ntiles = smooth_tiles(W, H);
  if (ntiles > 0x7fffffffLL || batch > 65535 || V > kMaxVoxels) return cudaErrorInvalidValue;
  const int tw = smooth_tile_width(W);
  const int zc = zchunk > 0 ? (zchunk < D ? zchunk : D) : smooth_chunk(D, ntiles * batch);
  const dim3 grid((unsigned)ntiles, (unsigned)((D + zc - 1) / zc), (unsigned)batch);
  // 8-byte accesses need an even W (pairs never straddle the edge) and 8-byte
  // aligned volumes
  const bool pairs = (W & 1) == 0 &&
                     ((reinterpret_cast<uintptr_t>(vol) | reinterpret_cast<uintptr_t>(cert) |
                       reinterpret_cast<uintptr_t>(dst)) & 7) == 0;
  const bool acc = !alias && accumulate != 0;
  const int variant = times_cert ? 16 + (pairs ? 1 : 0)
                                 : (cert ? 8 : 0) | (pairs ? 4 : 0) | (scert ? 2 : 0) | (acc ? 1 : 0);
  void* args[] = {(void*)&vol, (void*)&cert, (void*)&scert, (void*)&W, (void*)&H,
                  (void*)&D,   (void*)&tw,   (void*)&zc,    (void*)&taps, (void*)&dst};
  {
    const cudaError_t e0 = cudaLaunchKernel(smooth_kernel_of(variant), grid, dim3(kSmThreads), args, kSmSmem, st);
    if (e0 != cudaSuccess) return e0;
  }
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess || !alias) return e;
  if (accumulate) return add_volumes(out, out, tmp1, V * batch, st);
  return cudaMemcpyAsync(out, tmp1, bytes, cudaMemcpyDeviceToDevice, st);
}

}  // namespace brc
