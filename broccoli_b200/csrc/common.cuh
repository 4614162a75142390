// common.cuh -- shared definitions of the B200 registration/filtering kernels.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace brc {

constexpr int kTaps = 343;          // 7 x 7 x 7
constexpr int kFilterFloats = 686;  // re[343] + im[343]
constexpr int kNParam = 12;
constexpr int kNSums = 42;          // 3 axes x (10 A sums + 4 h sums)
constexpr int kMaxFilters = 6;

// Filter bank passed to kernels by value (kernel parameter space).  Stored
// tap-major with the taps already reversed, so that coef[t][2k+c] is the
// weight that the sample at offset (dx,dy,dz) = (t%7-3, t/7%7-3, t/49-3)
// contributes to filter k's component c (0 re, 1 im): the reference's
// convolution uses F[(3-dx) + 7(3-dy) + 49(3-dz)] for that sample
// (kernelConvolution.cpp:2840-2858, broccoli_lib.cpp:5016-5017).
template <int NF>
struct FilterBank {
  float coef[kTaps * 2 * NF];
};

// The instances a kernel of the batched registration loop works on.  The
// loop keeps three lists of `stride` entries and their lengths; iteration
// it works on list it % 3, written by the solve of the previous iteration
// (instances whose update has not yet fallen below the tolerance).  The
// iteration is `it`, or *iter when iter is set (a device counter, so that
// one captured iteration serves every iteration of a graph's loop).  With
// list null: every instance 0 .. batch-1.
struct ActiveSet {
  const int* list;
  const int* count;
  const int* iter;
  int it;
  int stride;
};

inline ActiveSet all_instances() { return ActiveSet{nullptr, nullptr, nullptr, 0, 0}; }

__device__ __forceinline__ int active_iteration(const ActiveSet& a) { return a.iter ? *a.iter : a.it; }
__device__ __forceinline__ int active_count(const ActiveSet& a, int batch) {
  return a.list ? a.count[active_iteration(a) % 3] : batch;
}
__device__ __forceinline__ int active_instance(const ActiveSet& a, int i) {
  return a.list ? a.list[(active_iteration(a) % 3) * a.stride + i] : i;
}

// Four-quadrant arctangent of the phase kernels.  t = min(|x|,|y|) /
// max(|x|,|y|) with the hardware reciprocal (rcp.approx, about 1 ulp), atan(t)
// = t P(t^2) with P of degree 8 (a relative-error minimax fit made by
// broccoli_b200/fit_atan.py with Lawson's iteration, float32 relative error
// 1.4e-7 on [0, 1]), then pi/2 - r when |y| > |x|, pi - r when x < 0, and the sign
// of y.  Largest error about 2.5e-7 rad.  (0, 0) gives 0, and so does (+-0,
// -0), where atan2 gives +-pi; a larger magnitude below 2^-126 or from 2^126
// on gives a finite angle of lower accuracy.
__device__ __forceinline__ float phase_atan2(float y, float x) {
  const float ax = fabsf(x), ay = fabsf(y);
  const float mx = fmaxf(ax, ay), mn = fminf(ax, ay);
  float rmx;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(rmx) : "f"(fmaxf(mx, 1e-30f)));
  const float t = mn * rmx;
  const float s = t * t;
  float p = 2.849935787e-03f;
  p = fmaf(p, s, -1.606882550e-02f);
  p = fmaf(p, s, 4.269186407e-02f);
  p = fmaf(p, s, -7.504326850e-02f);
  p = fmaf(p, s, 1.064095125e-01f);
  p = fmaf(p, s, -1.420364976e-01f);
  p = fmaf(p, s, 1.999261975e-01f);
  p = fmaf(p, s, -3.333307207e-01f);
  p = fmaf(p, s, 1.0f);
  float r = __fmul_rn(p, t);
  r = ay > ax ? __fsub_rn(1.57079632679489662f, r) : r;
  r = x < 0.f ? __fsub_rn(3.14159265358979324f, r) : r;
  return copysignf(r, y);
}

// Square root by the hardware approximation (sqrt.approx, relative error
// about 2^-23); denormal inputs count as 0.
__device__ __forceinline__ float sqrt_approx(float v) {
  float r;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
  return r;
}

// Two floats in one 64-bit register, and the packed operations on them; each
// lane rounds as the scalar instruction does.
typedef unsigned long long F2;
__host__ __device__ __forceinline__ F2 f2_twice(float v) {
  union {
    float f[2];
    F2 u;
  } r;
  r.f[0] = r.f[1] = v;
  return r.u;
}
__device__ __forceinline__ F2 f2_pack(float lo, float hi) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ float2 f2_unpack(F2 v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ F2 f2_fma(F2 a, F2 b, F2 c) {
  F2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ F2 f2_mul(F2 a, F2 b) {
  F2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

__device__ __forceinline__ F2 f2_add(F2 a, F2 b) {
  F2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ F2 f2_add_rm(F2 a, F2 b) {
  F2 r;
  asm("add.rm.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ F2 f2_sub(F2 a, F2 b) {
  F2 r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

// Voxel i of a volume as (x, y, z): 32-bit divisions where the index allows
// them (a 64-bit division by a runtime size is some hundred instructions,
// more than the rest of an elementwise kernel).
__device__ __forceinline__ void voxel_of(long long i, int W, int H, int& x, int& y, int& z) {
  if ((i >> 32) == 0) {
    const unsigned r = (unsigned)i / (unsigned)W;
    x = (int)((unsigned)i - r * (unsigned)W);
    z = (int)(r / (unsigned)H);
    y = (int)(r - (unsigned)z * (unsigned)H);
  } else {
    x = (int)(i % W);
    y = (int)((i / W) % H);
    z = (int)(i / ((long long)W * H));
  }
}

// floor(v) as a float and an integer, for |v| < 2^22: adding 1.5 x 2^23 with
// rounding towards minus infinity leaves floor(v) in the low mantissa bits.
// (floorf and the conversion to int are one operation each of the
// quarter-rate unit; these are two additions and an integer subtraction.)
__device__ __forceinline__ void floor_small(float v, float& f, int& i) {
  const float t = __fadd_rd(v, 12582912.0f);
  f = t - 12582912.0f;
  i = __float_as_int(t) - 0x4B400000;
}

// OpenCL 1.2 section 8.2 linear filtering with unnormalised coordinates and
// clamp-to-edge addressing, exact float weights (the sampler of
// kernelRegistration.cpp:1064).  u, v, w include the +0.5 texel offset.
//
// The lanes of `mask` (those of the warp that sample at all, the same value on
// each of them) choose together: where the eight neighbours of every one are
// inside the volume they take one base address and constant offsets, else
// they all clamp every index (at W = 64 every warp of a moved volume holds an
// edge, and lanes that took two paths one after the other doubled its
// instructions).  Every lane of the mask comes to the vote once per call.
__device__ __forceinline__ float sample_linear(const float* __restrict__ T, int W, int H, int D,
                                              float u, float v, float w, unsigned mask) {
  // volumes hold fewer than 2^31 voxels (checked by the launchers)
  const float uu = u - 0.5f, vv = v - 0.5f, ww = w - 0.5f;
  float fu, fv, fw;
  int i0, j0, k0;
  if (fmaxf(fmaxf(fabsf(uu), fabsf(vv)), fabsf(ww)) < 4194304.0f) {
    floor_small(uu, fu, i0);
    floor_small(vv, fv, j0);
    floor_small(ww, fw, k0);
  } else {
    fu = floorf(uu);
    fv = floorf(vv);
    fw = floorf(ww);
    i0 = (int)fu;
    j0 = (int)fv;
    k0 = (int)fw;
  }
  const float a = uu - fu, bb = vv - fv, c = ww - fw;
  const int WH = W * H;
  float t000, t100, t010, t110, t001, t101, t011, t111;
  const bool inside =
      ((unsigned)i0 < (unsigned)(W - 1)) & ((unsigned)j0 < (unsigned)(H - 1)) & ((unsigned)k0 < (unsigned)(D - 1));
  if (__all_sync(mask, inside)) {
    const float* p0 = T + (i0 + j0 * W + k0 * WH);
    const float* p1 = p0 + WH;
    t000 = __ldg(p0);
    t100 = __ldg(p0 + 1);
    t010 = __ldg(p0 + W);
    t110 = __ldg(p0 + W + 1);
    t001 = __ldg(p1);
    t101 = __ldg(p1 + 1);
    t011 = __ldg(p1 + W);
    t111 = __ldg(p1 + W + 1);
  } else {
    // i0 + 1 of the largest int (a saturated conversion) clamps as i0 does
    const int xi0 = min(max(i0, 0), W - 1), xi1 = min(max(i0, -1) + (i0 < W), W - 1);
    const int yj0 = min(max(j0, 0), H - 1), yj1 = min(max(j0, -1) + (j0 < H), H - 1);
    const int zk0 = min(max(k0, 0), D - 1), zk1 = min(max(k0, -1) + (k0 < D), D - 1);
    const int r00 = yj0 * W + zk0 * WH;
    const int r10 = yj1 * W + zk0 * WH;
    const int r01 = yj0 * W + zk1 * WH;
    const int r11 = yj1 * W + zk1 * WH;
    t000 = __ldg(T + xi0 + r00);
    t100 = __ldg(T + xi1 + r00);
    t010 = __ldg(T + xi0 + r10);
    t110 = __ldg(T + xi1 + r10);
    t001 = __ldg(T + xi0 + r01);
    t101 = __ldg(T + xi1 + r01);
    t011 = __ldg(T + xi0 + r11);
    t111 = __ldg(T + xi1 + r11);
  }
  // trilinear weights applied as seven linear interpolations
  const float c00 = fmaf(a, t100 - t000, t000), c10 = fmaf(a, t110 - t010, t010);
  const float c01 = fmaf(a, t101 - t001, t001), c11 = fmaf(a, t111 - t011, t011);
  const float c0 = fmaf(bb, c10 - c00, c00), c1 = fmaf(bb, c11 - c01, c01);
  return fmaf(c, c1 - c0, c0);
}

// The eight neighbours of (i0, j0, k0), every index clamped to the volume:
// t[0] at (i0, j0, k0), + 1 for x, + 2 for y, + 4 for z.
__device__ __forceinline__ void load_clamped(const float* __restrict__ T, int W, int H, int D, int i0, int j0,
                                             int k0, float (&t)[8]) {
  // clamped to [-1, W - 1] first: a saturated index then has a successor
  const int ic = min(max(i0, -1), W - 1), jc = min(max(j0, -1), H - 1), kc = min(max(k0, -1), D - 1);
  const int x0 = max(ic, 0), x1 = min(ic + 1, W - 1);
  const int y0 = max(jc, 0), y1 = min(jc + 1, H - 1);
  const int z0 = max(kc, 0) * H, z1 = min(kc + 1, D - 1) * H;
  const int r00 = (y0 + z0) * W, r10 = (y1 + z0) * W, r01 = (y0 + z1) * W, r11 = (y1 + z1) * W;
  t[0] = __ldg(T + (x0 + r00));
  t[1] = __ldg(T + (x1 + r00));
  t[2] = __ldg(T + (x0 + r10));
  t[3] = __ldg(T + (x1 + r10));
  t[4] = __ldg(T + (x0 + r01));
  t[5] = __ldg(T + (x1 + r01));
  t[6] = __ldg(T + (x0 + r11));
  t[7] = __ldg(T + (x1 + r11));
}

// sample_linear of one lane, for positions of any size.
__device__ __forceinline__ float sample_clamped(const float* __restrict__ T, int W, int H, int D, float u, float v,
                                                float w) {
  const float uu = u - 0.5f, vv = v - 0.5f, ww = w - 0.5f;
  const float fu = floorf(uu), fv = floorf(vv), fw = floorf(ww);
  const float a = uu - fu, b = vv - fv, c = ww - fw;
  float t[8];
  load_clamped(T, W, H, D, (int)fu, (int)fv, (int)fw, t);
#pragma unroll
  for (int q = 0; q < 8; q += 2) t[q] = fmaf(a, t[q + 1] - t[q], t[q]);
  t[0] = fmaf(b, t[2] - t[0], t[0]);
  t[4] = fmaf(b, t[6] - t[4], t[4]);
  return fmaf(c, t[4] - t[0], t[0]);
}

// sample_linear at two positions at once (the halves of u, v, w), the
// arithmetic as packed pairs: the same operations in the same order per half.
// One vote, as there; a lane with a position that floor_small does not take
// votes against the unclamped loads.
__device__ __forceinline__ float2 sample_linear_pair(const float* __restrict__ T, int W, int H, int D, F2 u, F2 v,
                                                     F2 w, unsigned mask) {
  const F2 half = f2_twice(0.5f), magic = f2_twice(12582912.0f);
  const F2 uu = f2_sub(u, half), vv = f2_sub(v, half), ww = f2_sub(w, half);
  const float2 us = f2_unpack(uu), vs = f2_unpack(vv), ws = f2_unpack(ww);
  const float far = fmaxf(fmaxf(fmaxf(fabsf(us.x), fabsf(us.y)), fmaxf(fabsf(vs.x), fabsf(vs.y))),
                          fmaxf(fabsf(ws.x), fabsf(ws.y)));
  const bool near = far < 4194304.0f;
  // floor_small of the six coordinates
  const F2 tu = f2_add_rm(uu, magic), tv = f2_add_rm(vv, magic), tw = f2_add_rm(ww, magic);
  const F2 a = f2_sub(uu, f2_sub(tu, magic)), b = f2_sub(vv, f2_sub(tv, magic)), c = f2_sub(ww, f2_sub(tw, magic));
  const float2 iu = f2_unpack(tu), iv = f2_unpack(tv), iw = f2_unpack(tw);
  const int ia = __float_as_int(iu.x) - 0x4B400000, ib = __float_as_int(iu.y) - 0x4B400000;
  const int ja = __float_as_int(iv.x) - 0x4B400000, jb = __float_as_int(iv.y) - 0x4B400000;
  const int ka = __float_as_int(iw.x) - 0x4B400000, kb = __float_as_int(iw.y) - 0x4B400000;
  float ta[8], tb[8];
  const bool inside = near & ((unsigned)ia < (unsigned)(W - 1)) & ((unsigned)ja < (unsigned)(H - 1)) &
                      ((unsigned)ka < (unsigned)(D - 1)) & ((unsigned)ib < (unsigned)(W - 1)) &
                      ((unsigned)jb < (unsigned)(H - 1)) & ((unsigned)kb < (unsigned)(D - 1));
  if (__all_sync(mask, inside)) {
    const long long WH = (long long)W * H;
    const float* pa = T + (ia + (ja + ka * H) * W);
    const float* pb = T + (ib + (jb + kb * H) * W);
#pragma unroll
    for (int q = 0; q < 8; q++) {
      const long long o = ((q & 4) ? WH : 0) + ((q & 2) ? W : 0);
      ta[q] = __ldg(pa + o + (q & 1));
      tb[q] = __ldg(pb + o + (q & 1));
    }
  } else if (near) {
    load_clamped(T, W, H, D, ia, ja, ka, ta);
    load_clamped(T, W, H, D, ib, jb, kb, tb);
  } else {
    const float2 u2 = f2_unpack(u), v2 = f2_unpack(v), w2 = f2_unpack(w);
    return make_float2(sample_clamped(T, W, H, D, u2.x, v2.x, w2.x), sample_clamped(T, W, H, D, u2.y, v2.y, w2.y));
  }
  F2 t[8];
#pragma unroll
  for (int q = 0; q < 8; q++) t[q] = f2_pack(ta[q], tb[q]);
#pragma unroll
  for (int q = 0; q < 8; q += 2) t[q] = f2_fma(a, f2_sub(t[q + 1], t[q]), t[q]);
  t[0] = f2_fma(b, f2_sub(t[2], t[0]), t[0]);
  t[4] = f2_fma(b, f2_sub(t[6], t[4]), t[4]);
  return f2_unpack(f2_fma(c, f2_sub(t[4], t[0]), t[0]));
}

// The affine warp's sample of voxel (x, y, z): src at x + t + (A - I)(x -
// centre) with p = {t, A - I} (InterpolateVolumeLinearLinear,
// kernelRegistration.cpp:1066-1101).
__device__ __forceinline__ float affine_sample(const float* __restrict__ src, int W, int H, int D,
                                               const float* __restrict__ p, int x, int y, int z,
                                               unsigned mask) {
  const float xf = (float)x - ((float)W - 1.0f) * 0.5f;
  const float yf = (float)y - ((float)H - 1.0f) * 0.5f;
  const float zf = (float)z - ((float)D - 1.0f) * 0.5f;
  const float u = fmaf(p[5], zf, fmaf(p[4], yf, fmaf(p[3], xf, (float)x + p[0]))) + 0.5f;
  const float v = fmaf(p[8], zf, fmaf(p[7], yf, fmaf(p[6], xf, (float)y + p[1]))) + 0.5f;
  const float w = fmaf(p[11], zf, fmaf(p[10], yf, fmaf(p[9], xf, (float)z + p[2]))) + 0.5f;
  return sample_linear(src, W, H, D, u, v, w, mask);
}

// affine_sample of voxels (x, y, z) and (x, y, z2): the same operations, each
// rounded alike, so that a volume's result does not depend on which of the two
// a launch takes.
__device__ __forceinline__ float2 affine_sample_pair(const float* __restrict__ src, int W, int H, int D,
                                                     const float* __restrict__ p, int x, int y, int z, int z2,
                                                     unsigned mask) {
  const float xf = (float)x - ((float)W - 1.0f) * 0.5f;
  const float yf = (float)y - ((float)H - 1.0f) * 0.5f;
  const F2 zz = f2_pack((float)z, (float)z2);
  const F2 zf = f2_sub(zz, f2_twice(((float)D - 1.0f) * 0.5f));
  const F2 half = f2_twice(0.5f);
  const float pu = fmaf(p[4], yf, fmaf(p[3], xf, (float)x + p[0]));
  const float pv = fmaf(p[7], yf, fmaf(p[6], xf, (float)y + p[1]));
  const F2 pw = f2_fma(f2_pack(p[10], p[10]), f2_pack(yf, yf),
                       f2_fma(f2_pack(p[9], p[9]), f2_pack(xf, xf), f2_add(zz, f2_pack(p[2], p[2]))));
  const F2 u = f2_add(f2_fma(f2_pack(p[5], p[5]), zf, f2_pack(pu, pu)), half);
  const F2 v = f2_add(f2_fma(f2_pack(p[8], p[8]), zf, f2_pack(pv, pv)), half);
  const F2 w = f2_add(f2_fma(f2_pack(p[11], p[11]), zf, pw), half);
  return sample_linear_pair(src, W, H, D, u, v, w, mask);
}

}  // namespace brc
