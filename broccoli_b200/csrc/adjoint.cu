// adjoint.cu -- adjoint (backward) kernels of the differentiable pieces of
// the path: the 7^3 complex filtering, the affine and displacement-field
// trilinear warps.  The separable smoothing is its own adjoint up to
// reversing the taps (smooth3d with reversed taps).
//
// Filtering: q_k(x) = sum_d V(x+d) W_k(d), W_k(d) = F_k[3-d].  With
// g_k = dL/dq_k (re, im as two real channels),
//   dL/dV(y) = sum_k sum_e [g_re,k(y+e) W_re,k(-e) + g_im,k(y+e) W_im,k(-e)],
// a correlation of the 2*NF gradient channels with the unflipped filters.
//
// Warps: out(x) = S(c(x)), c = x + t + (A-I)(x-centre) (affine) or x + u(x)
// (field); dL/dc(x) = g(x) grad S(c(x)) with the exact derivative of the
// clamp-to-edge trilinear interpolant, dL/du = dL/dc, dL/dp = sum_x dL/dc
// d c/d p, and dL/dS is scattered with atomics onto the 8 clamped corners.
#include "common.cuh"

namespace brc {

// One CTA computes a 32 x 16 x 4 block of outputs; a thread owns 4 (x) x 4
// (y) of them.  The gradient of one filter at a time is staged in shared
// memory as (re, im) pairs with its +-3 halo, and each pair meets the tap
// pair (W_re, W_im) in one packed FMA whose lanes accumulate the real and
// the imaginary channel's part of the sum, added at the end.
//
// Every staged sample feeds one real output per tap only, so shared-memory
// bandwidth, not the FMA pipe, bounds the plain form (a row segment per
// (dz, dy): 16 samples loaded for 56 FMAs, and the two channels of a filter
// staged one after the other with stride-2 reads).  Four output rows per
// thread reuse a loaded row for up to four dy: 6 + 16 shared loads (40
// wavefronts) per 112 packed FMAs (224 cycles of a scheduler's FMA pipe).
// The rows yr = 0..9 of a thread's window meet output y with dy = yr - y in
// 0..6; the rows 3..6 meet all four outputs and run as a loop, the three
// before and after are unrolled (one body for all ten would be half zeros,
// ten bodies would not fit the instruction cache).
//
// Bank conflicts: a quarter-warp's 16-byte loads come from four x groups (2
// slots of 16 bytes apart) of two slices, whose pitch is odd in slots.
//
// The copies of a filter's block (70 KB) are all in flight at once (cp.async);
// loading it through registers, four at a time, took 58 us of 228.
// Three filters at 128x128x96: 276 us (one row segment per (dz, dy)) -> 228
// (four rows per thread) -> 170 (cp.async).  At this size the grid is 1.7
// waves of three blocks per SM.
constexpr int kAdjTX = 32, kAdjTY = 16, kAdjTZ = 4;
constexpr int kAdjR = 4, kAdjY = 4;
constexpr int kAdjThreads = (kAdjTX / kAdjR) * (kAdjTY / kAdjY) * kAdjTZ;  // 128
constexpr int kAdjRow = kAdjTX + 8;                                        // pairs of a staged row (38 used)
constexpr int kAdjRows = kAdjTY + 6, kAdjSlices = kAdjTZ + 6;
constexpr int kAdjSlice = kAdjRows * kAdjRow + 2;  // pairs: 441 slots of 16 bytes
constexpr int kAdjWRow = 8;                        // tap pairs of a (dz, dy) row (7 used)
constexpr size_t kAdjSmem = 8 * ((size_t)kAdjSlices * kAdjSlice + 49 * kAdjWRow);
static_assert((kAdjSlice / 2) % 2 == 1 && kAdjThreads == 128, "bank layout / thread decode");

template <int NF>
struct AdjBank {
  float2 w[NF][kTaps];  // (re, im) of filter k; index (ex+3) + 7(ey+3) + 49(ez+3)
};

template <int NF>
__global__ void __launch_bounds__(kAdjThreads, 3)
filter3d_adjoint_kernel(const float* __restrict__ grad, int W, int H, int D,
                        const __grid_constant__ AdjBank<NF> bank, float* __restrict__ out,
                        const float* __restrict__ scale) {
  extern __shared__ __align__(16) F2 adj_smem[];
  F2* s_g = adj_smem;
  F2* s_w = adj_smem + kAdjSlices * kAdjSlice;
  const int b = blockIdx.z;
  const int z_tiles = (D + kAdjTZ - 1) / kAdjTZ;
  const int tile_x0 = blockIdx.x * kAdjTX;
  const int tile_y0 = (blockIdx.y / z_tiles) * kAdjTY;
  const int tile_z0 = (blockIdx.y % z_tiles) * kAdjTZ;
  const long long V = (long long)W * H * D;
  // lanes: x group (low two bits), slice (low bit), x group (high bit), slice (high bit)
  const int lane = threadIdx.x & 31, yg = threadIdx.x >> 5;
  const int tx = (lane & 3) | ((lane >> 1) & 4), tz = ((lane >> 2) & 1) | ((lane >> 3) & 2);
  const int xl = threadIdx.x & 7;
  // pairs move as 8 bytes where the gradient is 8-byte aligned
  const bool pairs = (reinterpret_cast<uintptr_t>(grad) & 7) == 0;

  F2 acc[kAdjY][kAdjR];
#pragma unroll
  for (int y = 0; y < kAdjY; y++)
#pragma unroll
    for (int r = 0; r < kAdjR; r++) acc[y][r] = 0;

#pragma unroll 1
  for (int k = 0; k < NF; k++) {
    const float* g = grad + ((long long)b * NF + k) * 2 * V;
    __syncthreads();
    for (int i = threadIdx.x; i < 49 * kAdjWRow; i += kAdjThreads) {
      const int row = i / kAdjWRow, dx = i % kAdjWRow;
      const float2 w = dx < 7 ? bank.w[k][row * 7 + dx] : make_float2(0.f, 0.f);
      s_w[i] = f2_pack(w.x, w.y);
    }
    // eight threads copy a row, every copy in flight at once
    for (int row = threadIdx.x >> 3; row < kAdjSlices * kAdjRows; row += kAdjThreads / 8) {
      const int zs = row / kAdjRows, ys = row - zs * kAdjRows;
      const int y = tile_y0 - 3 + ys, z = tile_z0 - 3 + zs;
      const bool rowok = y >= 0 && y < H && z >= 0 && z < D;
      const float* q = g + 2 * ((long long)(rowok ? y : 0) * W + (long long)(rowok ? z : 0) * W * H);
      const uint32_t d = static_cast<uint32_t>(__cvta_generic_to_shared(s_g + zs * kAdjSlice + ys * kAdjRow)) + 8 * xl;
#pragma unroll
      for (int m = 0; m < kAdjRow / 8; m++) {
        const int x = tile_x0 - 4 + xl + 8 * m;
        const bool ok = rowok && x >= 0 && x < W;
        const float* p = q + (ok ? 2 * x : 0);
        if (pairs) {
          asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d + 64 * m), "l"(p), "r"(ok ? 8 : 0) : "memory");
        } else {
          asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d + 64 * m), "l"(p), "r"(ok ? 4 : 0) : "memory");
          asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d + 64 * m + 4), "l"(p + 1), "r"(ok ? 4 : 0)
                       : "memory");
        }
      }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
#pragma unroll 1
    for (int dz = 0; dz < 7; dz++) {
      const F2* rows = s_g + (tz + dz) * kAdjSlice + (kAdjY * yg) * kAdjRow + kAdjR * tx;
      const F2* taps = s_w + dz * 7 * kAdjWRow;
      F2 d[12];
      // sample at offset ex of output r sits at d[4 + r + ex]
      auto load_row = [&](int yr) {
        const ulonglong2* q = reinterpret_cast<const ulonglong2*>(rows + yr * kAdjRow);
#pragma unroll
        for (int s = 0; s < 6; s++) {
          const ulonglong2 v = q[s];
          d[2 * s] = v.x;
          d[2 * s + 1] = v.y;
        }
      };
      auto add = [&](F2 (&o)[kAdjR], int dy) {
        const ulonglong2* q = reinterpret_cast<const ulonglong2*>(taps + dy * kAdjWRow);
#pragma unroll
        for (int s = 0; s < 4; s++) {
          const ulonglong2 w = q[s];
#pragma unroll
          for (int r = 0; r < kAdjR; r++) o[r] = f2_fma(d[1 + r + 2 * s], w.x, o[r]);
          if (s < 3) {
#pragma unroll
            for (int r = 0; r < kAdjR; r++) o[r] = f2_fma(d[2 + r + 2 * s], w.y, o[r]);
          }
        }
      };
#pragma unroll
      for (int yr = 0; yr < 3; yr++) {
        load_row(yr);
#pragma unroll
        for (int y = 0; y <= yr; y++) add(acc[y], yr - y);
      }
#pragma unroll 1
      for (int yr = 3; yr < 7; yr++) {
        load_row(yr);
#pragma unroll
        for (int y = 0; y < kAdjY; y++) add(acc[y], yr - y);
      }
#pragma unroll
      for (int yr = 7; yr < 10; yr++) {
        load_row(yr);
#pragma unroll
        for (int y = yr - 6; y < kAdjY; y++) add(acc[y], yr - y);
      }
    }
  }
  const int x0 = tile_x0 + kAdjR * tx, z = tile_z0 + tz;
  if (z >= D) return;
  const float f = scale ? 2.0f * *scale : 1.0f;  // 1: the sum itself, bit for bit
#pragma unroll
  for (int yy = 0; yy < kAdjY; yy++) {
    const int y = tile_y0 + kAdjY * yg + yy;
    if (y >= H) break;
    float* o = out + (long long)b * V + x0 + (long long)y * W + (long long)z * W * H;
#pragma unroll
    for (int r = 0; r < kAdjR; r++)
      if (x0 + r < W) {
        const float2 v = f2_unpack(acc[yy][r]);
        o[r] = f * (v.x + v.y);
      }
  }
}

// Value and gradient (d/du, d/dv, d/dw) of the clamp-to-edge trilinear
// interpolant at (u, v, w) (with the +0.5 texel convention).
__device__ __forceinline__ void sample_grad(const float* __restrict__ T, int W, int H, int D, float u, float v,
                                            float w, float& gx, float& gy, float& gz, long long* idx,
                                            float* wt) {
  const float uu = u - 0.5f, vv = v - 0.5f, ww = w - 0.5f;
  const float fu = floorf(uu), fv = floorf(vv), fw = floorf(ww);
  const float a = uu - fu, bb = vv - fv, c = ww - fw;
  const int i0 = (int)fu, j0 = (int)fv, k0 = (int)fw;
  const int xi0 = min(max(i0, 0), W - 1), xi1 = min(max(i0 + 1, 0), W - 1);
  const int yj0 = min(max(j0, 0), H - 1), yj1 = min(max(j0 + 1, 0), H - 1);
  const int zk0 = min(max(k0, 0), D - 1), zk1 = min(max(k0 + 1, 0), D - 1);
  const long long WH = (long long)W * H;
  idx[0] = xi0 + yj0 * (long long)W + zk0 * WH;
  idx[1] = xi1 + yj0 * (long long)W + zk0 * WH;
  idx[2] = xi0 + yj1 * (long long)W + zk0 * WH;
  idx[3] = xi1 + yj1 * (long long)W + zk0 * WH;
  idx[4] = xi0 + yj0 * (long long)W + zk1 * WH;
  idx[5] = xi1 + yj0 * (long long)W + zk1 * WH;
  idx[6] = xi0 + yj1 * (long long)W + zk1 * WH;
  idx[7] = xi1 + yj1 * (long long)W + zk1 * WH;
  float t[8];
#pragma unroll
  for (int k = 0; k < 8; k++) t[k] = __ldg(T + idx[k]);
  wt[0] = (1.f - a) * (1.f - bb) * (1.f - c);
  wt[1] = a * (1.f - bb) * (1.f - c);
  wt[2] = (1.f - a) * bb * (1.f - c);
  wt[3] = a * bb * (1.f - c);
  wt[4] = (1.f - a) * (1.f - bb) * c;
  wt[5] = a * (1.f - bb) * c;
  wt[6] = (1.f - a) * bb * c;
  wt[7] = a * bb * c;
  gx = (1.f - bb) * (1.f - c) * (t[1] - t[0]) + bb * (1.f - c) * (t[3] - t[2]) + (1.f - bb) * c * (t[5] - t[4]) +
       bb * c * (t[7] - t[6]);
  gy = (1.f - a) * (1.f - c) * (t[2] - t[0]) + a * (1.f - c) * (t[3] - t[1]) + (1.f - a) * c * (t[6] - t[4]) +
       a * c * (t[7] - t[5]);
  gz = (1.f - a) * (1.f - bb) * (t[4] - t[0]) + a * (1.f - bb) * (t[5] - t[1]) + (1.f - a) * bb * (t[6] - t[2]) +
       a * bb * (t[7] - t[3]);
}

constexpr int kWBThreads = 256;

// Affine warp backward: per-CTA FP64 partial sums of dL/dp (12 per
// instance) and, optionally, dL/dsrc scattered with atomics.
__global__ void __launch_bounds__(kWBThreads)
warp_affine_backward_kernel(const float* __restrict__ src, int W, int H, int D,
                            const float* __restrict__ params, const float* __restrict__ gout,
                            double* __restrict__ partials, float* __restrict__ gsrc) {
  const int b = blockIdx.y;
  const long long V = (long long)W * H * D;
  const float* S = src + (long long)b * V;
  const float* p = params + (long long)b * 12;
  double acc[12];
#pragma unroll
  for (int j = 0; j < 12; j++) acc[j] = 0.0;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < V;
       i += (long long)gridDim.x * blockDim.x) {
    int x, y, z;
    voxel_of(i, W, H, x, y, z);
    const float xf = (float)x - ((float)W - 1.0f) * 0.5f;
    const float yf = (float)y - ((float)H - 1.0f) * 0.5f;
    const float zf = (float)z - ((float)D - 1.0f) * 0.5f;
    const float u = (float)x + p[0] + p[3] * xf + p[4] * yf + p[5] * zf + 0.5f;
    const float v = (float)y + p[1] + p[6] * xf + p[7] * yf + p[8] * zf + 0.5f;
    const float w = (float)z + p[2] + p[9] * xf + p[10] * yf + p[11] * zf + 0.5f;
    float gx, gy, gz, wt[8];
    long long idx[8];
    sample_grad(S, W, H, D, u, v, w, gx, gy, gz, idx, wt);
    const float g = gout[(long long)b * V + i];
    const double cx = (double)g * gx, cy = (double)g * gy, cz = (double)g * gz;
    acc[0] += cx;
    acc[1] += cy;
    acc[2] += cz;
    acc[3] += cx * xf;
    acc[4] += cx * yf;
    acc[5] += cx * zf;
    acc[6] += cy * xf;
    acc[7] += cy * yf;
    acc[8] += cy * zf;
    acc[9] += cz * xf;
    acc[10] += cz * yf;
    acc[11] += cz * zf;
    if (gsrc != nullptr) {
      float* gs = gsrc + (long long)b * V;
#pragma unroll
      for (int k = 0; k < 8; k++) atomicAdd(gs + idx[k], g * wt[k]);
    }
  }
  __shared__ double red[kWBThreads / 32][12];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int j = 0; j < 12; j++) {
    double v = acc[j];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (lane == 0) red[warp][j] = v;
  }
  __syncthreads();
  if (threadIdx.x < 12) {
    double v = 0.0;
    for (int k = 0; k < kWBThreads / 32; k++) v += red[k][threadIdx.x];
    partials[((long long)b * gridDim.x + blockIdx.x) * 12 + threadIdx.x] = v;
  }
}

// out[b][j] = sum of the nblk partial rows, one warp per sum: lane l takes
// rows l, l + 32, .., then a fixed shuffle tree (the same order on every run).
__global__ void reduce12_kernel(const double* __restrict__ partials, int nblk, double* __restrict__ out) {
  const int b = blockIdx.x, j = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double v = 0.0;
  for (int r = lane; r < nblk; r += 32) v += partials[((long long)b * nblk + r) * 12 + j];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  if (lane == 0) out[(long long)b * 12 + j] = v;
}

// Field warp backward: dL/du per voxel and optionally dL/dsrc.
__global__ void __launch_bounds__(256)
warp_field_backward_kernel(const float* __restrict__ src, int W, int H, int D, const float* __restrict__ dx,
                           const float* __restrict__ dy, const float* __restrict__ dz,
                           const float* __restrict__ gout, float* __restrict__ gfield,
                           float* __restrict__ gsrc) {
  const long long V = (long long)W * H * D;
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= V) return;
  int x, y, z;
  voxel_of(i, W, H, x, y, z);
  float gx, gy, gz, wt[8];
  long long idx[8];
  sample_grad(src, W, H, D, (float)x + dx[i] + 0.5f, (float)y + dy[i] + 0.5f, (float)z + dz[i] + 0.5f, gx, gy,
              gz, idx, wt);
  const float g = gout[i];
  if (gfield != nullptr) {
    gfield[i] = g * gx;
    gfield[V + i] = g * gy;
    gfield[2 * V + i] = g * gz;
  }
  if (gsrc != nullptr) {
#pragma unroll
    for (int k = 0; k < 8; k++) atomicAdd(gsrc + idx[k], g * wt[k]);
  }
}

// ---------------------------------------------------------------------------

template <int NF>
static cudaError_t launch_adjoint(const float* grad, int W, int H, int D, int batch, const float* h_filters,
                                  float* out, const float* scale, cudaStream_t st) {
  AdjBank<NF> bank;
  for (int k = 0; k < NF; k++)
    for (int ez = -3; ez <= 3; ez++)
      for (int ey = -3; ey <= 3; ey++)
        for (int ex = -3; ex <= 3; ex++) {
          // weight W(-e) = F[3 + e]
          const float* f = h_filters + k * kFilterFloats + (3 + ex) + 7 * (3 + ey) + 49 * (3 + ez);
          bank.w[k][(ex + 3) + 7 * (ey + 3) + 49 * (ez + 3)] = make_float2(f[0], f[kTaps]);
        }
  // the dynamic shared memory above 48 KB is a per-device function attribute
  static bool attr_set[64] = {false};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  if (!attr_set[dev]) {
    const cudaError_t e = cudaFuncSetAttribute(filter3d_adjoint_kernel<NF>,
                                               cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kAdjSmem);
    if (e != cudaSuccess) return e;
    attr_set[dev] = true;
  }
  const int z_tiles = (D + kAdjTZ - 1) / kAdjTZ;
  dim3 grid((W + kAdjTX - 1) / kAdjTX, ((H + kAdjTY - 1) / kAdjTY) * z_tiles, batch);
  filter3d_adjoint_kernel<NF><<<grid, kAdjThreads, kAdjSmem, st>>>(grad, W, H, D, bank, out, scale);
  return cudaGetLastError();
}

cudaError_t filter3d_adjoint(const float* grad, int W, int H, int D, int batch, const float* h_filters, int nfilt,
                             float* out, cudaStream_t st, const float* scale) {
  if (nfilt == 3) return launch_adjoint<3>(grad, W, H, D, batch, h_filters, out, scale, st);
  if (nfilt == 6) return launch_adjoint<6>(grad, W, H, D, batch, h_filters, out, scale, st);
  return cudaErrorInvalidValue;
}

// Sum of squared differences.  q becomes q - ref in place (the backward pass
// needs the difference, and 2 g times it goes through the adjoint filtering
// as a factor of its output), and each block writes the FP64 sum of its
// squares; sum_partials_kernel adds the blocks in order.  Bound by memory:
// two reads and a write per value, one pass where subtraction, square, sum and
// their backward products were six (128x128x96, three filters: objective and
// gradient 432 -> 367 us).
constexpr int kSsdThreads = 256, kSsdBlocks = 148 * 8;

template <bool VEC>
__global__ void __launch_bounds__(kSsdThreads)
ssd_residual_kernel(float* __restrict__ q, const float* __restrict__ ref, long long n, double* __restrict__ partials) {
  double sum = 0.0;
  const long long step = (long long)gridDim.x * kSsdThreads;
  const long long i0 = (long long)blockIdx.x * kSsdThreads + threadIdx.x;
  if (VEC) {
    float4* q4 = reinterpret_cast<float4*>(q);
    const float4* r4 = reinterpret_cast<const float4*>(ref);
#pragma unroll 4
    for (long long i = i0; i < n / 4; i += step) {
      const float4 a = q4[i], b = __ldg(r4 + i);
      const float4 d = make_float4(a.x - b.x, a.y - b.y, a.z - b.z, a.w - b.w);
      q4[i] = d;
      sum += (double)(d.x * d.x + d.y * d.y + d.z * d.z + d.w * d.w);
    }
  } else {
    for (long long i = i0; i < n; i += step) {
      const float d = q[i] - __ldg(ref + i);
      q[i] = d;
      sum += (double)(d * d);
    }
  }
  __shared__ double s[kSsdThreads / 32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_down_sync(0xffffffffu, sum, o);
  if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = sum;
  __syncthreads();
  if (threadIdx.x == 0) {
#pragma unroll
    for (int w = 1; w < kSsdThreads / 32; w++) sum += s[w];
    partials[blockIdx.x] = sum;
  }
}

// *out = sum of n partial sums (one warp, a fixed order).
__global__ void sum_partials_kernel(const double* __restrict__ partials, int n, float* __restrict__ out) {
  double v = 0.0;
#pragma unroll 4
  for (int r = threadIdx.x; r < n; r += 32) v += partials[r];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  if (threadIdx.x == 0) *out = (float)v;
}

int ssd_blocks(long long n) {
  const long long b = (n / 4 + kSsdThreads) / kSsdThreads;
  return (int)(b < kSsdBlocks ? b : kSsdBlocks);
}

cudaError_t ssd_residual(float* q, const float* ref, long long n, double* partials, float* out, cudaStream_t st) {
  const int nb = ssd_blocks(n);
  // 16-byte accesses where both arrays allow them and no value is left over
  if ((n & 3) == 0 && ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(ref)) & 15) == 0)
    ssd_residual_kernel<true><<<nb, kSsdThreads, 0, st>>>(q, ref, n, partials);
  else
    ssd_residual_kernel<false><<<nb, kSsdThreads, 0, st>>>(q, ref, n, partials);
  sum_partials_kernel<<<1, 32, 0, st>>>(partials, nb, out);
  return cudaGetLastError();
}

int warp_affine_backward_blocks(long long V) {
  long long n = (V + kWBThreads - 1) / kWBThreads;
  return (int)(n < 148 * 4 ? n : 148 * 4);
}

cudaError_t warp_affine_backward(const float* src, int W, int H, int D, int batch, const float* params,
                                 const float* gout, double* partials, int nblk, double* gparams, float* gsrc,
                                 cudaStream_t st) {
  dim3 grid(nblk, batch);
  warp_affine_backward_kernel<<<grid, kWBThreads, 0, st>>>(src, W, H, D, params, gout, partials, gsrc);
  reduce12_kernel<<<batch, 12 * 32, 0, st>>>(partials, nblk, gparams);
  return cudaGetLastError();
}

cudaError_t warp_field_backward(const float* src, int W, int H, int D, const float* dx, const float* dy,
                                const float* dz, const float* gout, float* gfield, float* gsrc,
                                cudaStream_t st) {
  const long long V = (long long)W * H * D;
  warp_field_backward_kernel<<<(unsigned)((V + 255) / 256), 256, 0, st>>>(src, W, H, D, dx, dy, dz, gout,
                                                                          gfield, gsrc);
  return cudaGetLastError();
}

}  // namespace brc
