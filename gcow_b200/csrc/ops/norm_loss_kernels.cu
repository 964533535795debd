// Memory-bound training kernels (sm_100a): LayerNorm forward/backward, exact-erf
// GELU forward/backward, fused softmax cross-entropy (loss + in-place gradient),
// column sums (bias gradients) and the uint8 -> bf16 image normalisation.
// All of them stream their operands once with 16-byte accesses and keep row
// statistics in fp32; reductions that cross CTAs are two-stage with a fixed
// order, so results are run-to-run deterministic.
//
// The reference's models get these from ATen/cuDNN through PyTorch
// (hw/models/resenet.py:12-22,80-89; cross-entropy at hw/models/train_imagenet.py:249).
#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "pdl.cuh"
#include <atomic>
#include <stdint.h>

namespace gcow {
namespace nl {

typedef __nv_bfloat16 bf16;

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int d = 16; d; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
  return v;
}
__device__ __forceinline__ float warp_max(float v) {
#pragma unroll
  for (int d = 16; d; d >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, d));
  return v;
}
__device__ __forceinline__ void load8(const bf16* p, float (&v)[8]) {
  uint4 u = *reinterpret_cast<const uint4*>(p);
  const __nv_bfloat162* b = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
  for (int i = 0; i < 4; i++) { float2 f = __bfloat1622float2(b[i]); v[2 * i] = f.x; v[2 * i + 1] = f.y; }
}
__device__ __forceinline__ void unpack8(const uint4& u, float (&v)[8]) {
  const __nv_bfloat162* b = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
  for (int i = 0; i < 4; i++) { float2 f = __bfloat1622float2(b[i]); v[2 * i] = f.x; v[2 * i + 1] = f.y; }
}
__device__ __forceinline__ void store8(bf16* p, const float (&v)[8]) {
  uint4 u;
  __nv_bfloat162* b = reinterpret_cast<__nv_bfloat162*>(&u);
#pragma unroll
  for (int i = 0; i < 4; i++) b[i] = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
  *reinterpret_cast<uint4*>(p) = u;
}

// ------------------------------------------------------------------ LayerNorm
// One warp per row; H a multiple of 8. The row (a few KB) is re-read from L1.
__global__ void __launch_bounds__(128)
layernorm_fwd_kernel(const bf16* __restrict__ x, const float* __restrict__ gamma, const float* __restrict__ beta,
                     bf16* __restrict__ y, float* __restrict__ mean, float* __restrict__ rstd, int rows, int H,
                     float eps) {
  pdl_wait();
  pdl_trigger();
  const int lane = threadIdx.x & 31;
  for (int r = blockIdx.x * 4 + (threadIdx.x >> 5); r < rows; r += gridDim.x * 4) {
    const bf16* xr = x + (size_t)r * H;
    float s = 0;
    for (int c = lane * 8; c < H; c += 256) { float v[8]; load8(xr + c, v);
#pragma unroll
      for (int i = 0; i < 8; i++) s += v[i]; }
    const float mu = warp_sum(s) / H;
    float q = 0;
    for (int c = lane * 8; c < H; c += 256) { float v[8]; load8(xr + c, v);
#pragma unroll
      for (int i = 0; i < 8; i++) { float d = v[i] - mu; q += d * d; } }
    const float rs = rsqrtf(warp_sum(q) / H + eps);
    if (lane == 0) { mean[r] = mu; rstd[r] = rs; }
    bf16* yr = y + (size_t)r * H;
    for (int c = lane * 8; c < H; c += 256) {
      float v[8];
      load8(xr + c, v);
      const float4 g0 = *reinterpret_cast<const float4*>(gamma + c), g1 = *reinterpret_cast<const float4*>(gamma + c + 4);
      const float4 b0 = *reinterpret_cast<const float4*>(beta + c), b1 = *reinterpret_cast<const float4*>(beta + c + 4);
      const float g[8] = {g0.x, g0.y, g0.z, g0.w, g1.x, g1.y, g1.z, g1.w};
      const float b[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
#pragma unroll
      for (int i = 0; i < 8; i++) v[i] = (v[i] - mu) * rs * g[i] + b[i];
      store8(yr + c, v);
    }
  }
}

// The same for H <= 256 * CH: a row stays in registers (CH chunks of 8 values per lane) and the next one is on its way while
// this one is worked on. The form above reads a row three times, each time behind a reduction across
// the warp (16384 x 1024: 16.8 us, now 14.6; 67 MB take 10).
template <int CH> constexpr int kRowCtas = CH == 1 ? 10 : CH == 2 ? 9 : CH == 3 ? 8 : 6;   // CTAs per SM, as the registers allow: the grid
template <int CH>
__global__ void __launch_bounds__(128, kRowCtas<CH>)
layernorm_fwd_rows_kernel(const bf16* x, const float* gamma, const float* beta,
                          bf16* __restrict__ y, float* __restrict__ mean, float* __restrict__ rstd, int rows, int H, float eps) {
  pdl_wait();
  pdl_trigger();
  const int lane = threadIdx.x & 31, stride = gridDim.x * 4;
  int r = blockIdx.x * 4 + (threadIdx.x >> 5);
  uint4 next[CH];
  auto fetch = [&](int row) {
    const bf16* const xr = x + (size_t)row * H;
#pragma unroll
    for (int k = 0; k < CH; k++) {
      const int c = lane * 8 + 256 * k;
      next[k] = c < H ? *reinterpret_cast<const uint4*>(xr + c) : make_uint4(0, 0, 0, 0);
    }
  };
  if (r < rows) fetch(r);
  for (; r < rows; r += stride) {
    float v[CH][8];
#pragma unroll
    for (int k = 0; k < CH; k++) unpack8(next[k], v[k]);
    if (r + stride < rows) fetch(r + stride);
    float s = 0;
#pragma unroll
    for (int k = 0; k < CH; k++)
#pragma unroll
      for (int i = 0; i < 8; i++) s += v[k][i];
    const float mu = warp_sum(s) / H;
    float q = 0;
#pragma unroll
    for (int k = 0; k < CH; k++)
      if (lane * 8 + 256 * k < H) {
#pragma unroll
        for (int i = 0; i < 8; i++) { const float d = v[k][i] - mu; q += d * d; }
      }
    const float rs = rsqrtf(warp_sum(q) / H + eps);
    if (lane == 0) { mean[r] = mu; rstd[r] = rs; }
    bf16* const yr = y + (size_t)r * H;
#pragma unroll
    for (int k = 0; k < CH; k++) {
      const int c = lane * 8 + 256 * k;
      if (c < H) {
        const float4 g0 = *reinterpret_cast<const float4*>(gamma + c), g1 = *reinterpret_cast<const float4*>(gamma + c + 4);
        const float4 b0 = *reinterpret_cast<const float4*>(beta + c), b1 = *reinterpret_cast<const float4*>(beta + c + 4);
        const float g[8] = {g0.x, g0.y, g0.z, g0.w, g1.x, g1.y, g1.z, g1.w};
        const float b[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
#pragma unroll
        for (int i = 0; i < 8; i++) v[k][i] = (v[k][i] - mu) * rs * g[i] + b[i];
        store8(yr + c, v[k]);
      }
    }
  }
}

// LayerNorm backward: dx per row; per-CTA partial sums of dgamma/dbeta go to part[blockIdx.x][2][H].
// Rows of up to 1024 columns, H <= 256 * CH. A warp takes a row; a lane always works on the same columns (lane * 8 + 256 * k), so its
// dgamma/dbeta contributions stay in registers over all its rows and touch shared memory once at the end. The next row is on its way into
// shared memory (cp.async; each lane fetches and reads its own 16-byte pieces, so nothing has to be synchronised) while this one is worked
// on. What bounds it is how many rows an SM has in flight: with the next row in registers it was 12 warps (168 registers at 1024 columns,
// some of them spilled), now 16. Two rows ahead are 4 % slower at 16384 x 1024.
// T threads a CTA, 512 / T CTAs per SM: with 512 threads the SM's partial sums are added up before they are written, with 128 few rows spread
// over more SMs. Both passes together, against the rows in registers: 16384 x 1024 36.1 -> 24.7 us (100 MB take 15.4), x 768 23.1 -> 20.3,
// x 512 18.6 -> 15.6, x 256 13.5 -> 10.7, 2048 x 1024 12.7 -> 8.5, 512 x 1024 8.1 -> 6.7.
constexpr int kLnWide = 512, kLnNarrow = 128;
__device__ __forceinline__ void copy16(void* smem, const void* g) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(g) : "memory");
}
template <int CH, int T> constexpr size_t kLnBwdSmem = (size_t)CH * (256 * 4 + 2 * 2 * T * 16);      // gamma, two rows' x and dy of every lane
template <int CH, int T>
__global__ void __launch_bounds__(T, 512 / T)
layernorm_bwd_rows_kernel(const bf16* dy, const bf16* x, const float* gamma, const float* mean, const float* rstd, bf16* __restrict__ dx,
                          float* __restrict__ part, int rows, int H) {
  pdl_trigger();
  pdl_wait();
  extern __shared__ __align__(16) float sm[];          // gamma [256 * CH], the rows on their way; in the end [warps][2][H]
  constexpr int kWarps = T / 32;
  static_assert(kLnBwdSmem<CH, T> >= (size_t)kWarps * 2 * 256 * CH * 4, "the warps' sums lie over the gamma copy and the rows");
  uint4* const ring = reinterpret_cast<uint4*>(sm + 256 * CH) + threadIdx.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, stride = gridDim.x * kWarps;
  auto fetch = [&](int row, int slot) {
    if (row < rows) {
      const bf16* const xr = x + (size_t)row * H;
      const bf16* const gr = dy + (size_t)row * H;
#pragma unroll
      for (int k = 0; k < CH; k++) {
        const int c = lane * 8 + 256 * k;
        if (c < H) {
          copy16(ring + (slot * 2 * CH + 2 * k) * T, xr + c);
          copy16(ring + (slot * 2 * CH + 2 * k + 1) * T, gr + c);
        }
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  int r = blockIdx.x * kWarps + warp, slot = 0;
  fetch(r, 0);
  for (int c = threadIdx.x; c < 256 * CH; c += T) sm[c] = c < H ? gamma[c] : 0.0f;
  float rg[CH][8], rb[CH][8], next_mu = 0.0f, next_rs = 0.0f;
#pragma unroll
  for (int k = 0; k < CH; k++)
#pragma unroll
    for (int i = 0; i < 8; i++) { rg[k][i] = 0; rb[k][i] = 0; }
  if (r < rows) { next_mu = mean[r]; next_rs = rstd[r]; }
  __syncthreads();
  for (; r < rows; r += stride, slot ^= 1) {
    fetch(r + stride, slot ^ 1);
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    const float mu = next_mu, rs = next_rs;
    if (r + stride < rows) { next_mu = mean[r + stride]; next_rs = rstd[r + stride]; }
    const uint4* const row = ring + slot * 2 * CH * T;
    float s1 = 0, s2 = 0;
#pragma unroll
    for (int k = 0; k < CH; k++) {
      const int c = lane * 8 + 256 * k;
      if (c < H) {
        float xv[8], gv[8], gam[8];
        unpack8(row[2 * k * T], xv); unpack8(row[(2 * k + 1) * T], gv);
        *reinterpret_cast<float4*>(gam) = *reinterpret_cast<const float4*>(sm + c);
        *reinterpret_cast<float4*>(gam + 4) = *reinterpret_cast<const float4*>(sm + c + 4);
#pragma unroll
        for (int i = 0; i < 8; i++) {
          const float xh = (xv[i] - mu) * rs, gg = gv[i] * gam[i];
          s1 += gg; s2 += gg * xh;
          rg[k][i] += gv[i] * xh;
          rb[k][i] += gv[i];
        }
      }
    }
    s1 = warp_sum(s1) / H; s2 = warp_sum(s2) / H;
    bf16* const dr = dx + (size_t)r * H;
    // the row is unpacked again: cheaper than keeping 2 x 8 x CH floats
#pragma unroll
    for (int k = 0; k < CH; k++) {
      const int c = lane * 8 + 256 * k;
      if (c < H) {
        float xv[8], gv[8], gam[8], o[8];
        unpack8(row[2 * k * T], xv); unpack8(row[(2 * k + 1) * T], gv);
        *reinterpret_cast<float4*>(gam) = *reinterpret_cast<const float4*>(sm + c);
        *reinterpret_cast<float4*>(gam + 4) = *reinterpret_cast<const float4*>(sm + c + 4);
#pragma unroll
        for (int i = 0; i < 8; i++) o[i] = rs * (gv[i] * gam[i] - s1 - (xv[i] - mu) * rs * s2);
        store8(dr + c, o);
      }
    }
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();      // every warp is done with the gamma copy and the rows that these sums overwrite
  float* const dg = sm + (size_t)warp * 2 * H;
  float* const db = dg + H;
#pragma unroll
  for (int k = 0; k < CH; k++)
#pragma unroll
    for (int i = 0; i < 8; i += 4) {
      const int c = lane * 8 + 256 * k + i;
      if (c < H) {
        *reinterpret_cast<float4*>(dg + c) = make_float4(rg[k][i], rg[k][i + 1], rg[k][i + 2], rg[k][i + 3]);
        *reinterpret_cast<float4*>(db + c) = make_float4(rb[k][i], rb[k][i + 1], rb[k][i + 2], rb[k][i + 3]);
      }
    }
  __syncthreads();
  float* const out = part + (size_t)blockIdx.x * 2 * H;
  const bool wide = ((uintptr_t)part & 15) == 0;       // 2 H is a multiple of 16
  for (int c = threadIdx.x * 4; c < 2 * H; c += T * 4) {
    float4 t = *reinterpret_cast<const float4*>(sm + c);
#pragma unroll
    for (int w = 1; w < kWarps; w++) {
      const float4 u = *reinterpret_cast<const float4*>(sm + (size_t)w * 2 * H + c);
      t.x += u.x; t.y += u.y; t.z += u.z; t.w += u.w;
    }
    if (wide) {
      *reinterpret_cast<float4*>(out + c) = t;
    } else {
      out[c] = t.x; out[c + 1] = t.y; out[c + 2] = t.z; out[c + 3] = t.w;
    }
  }
}

// Wider rows: dgamma/dbeta are summed up in shared memory.
__global__ void __launch_bounds__(128)
layernorm_bwd_kernel(const bf16* __restrict__ dy, const bf16* __restrict__ x, const float* __restrict__ gamma,
                     const float* __restrict__ mean, const float* __restrict__ rstd, bf16* __restrict__ dx,
                     float* __restrict__ part, int rows, int H) {
  pdl_trigger();
  pdl_wait();
  extern __shared__ __align__(16) float sm[];          // [4 warps][2][H]
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float* dg = sm + (size_t)warp * 2 * H;
  float* db = dg + H;
  for (int c = lane; c < H; c += 32) { dg[c] = 0; db[c] = 0; }
  __syncwarp();
  for (int r = blockIdx.x * 4 + warp; r < rows; r += gridDim.x * 4) {
    const bf16* xr = x + (size_t)r * H;
    const bf16* gr = dy + (size_t)r * H;
    const float mu = mean[r], rs = rstd[r];
    float s1 = 0, s2 = 0;
    for (int c = lane * 8; c < H; c += 256) {
      float xv[8], gv[8];
      load8(xr + c, xv); load8(gr + c, gv);
#pragma unroll
      for (int i = 0; i < 8; i++) {
        const float xh = (xv[i] - mu) * rs, gg = gv[i] * gamma[c + i];
        s1 += gg; s2 += gg * xh;
        dg[c + i] += gv[i] * xh;
        db[c + i] += gv[i];
      }
    }
    s1 = warp_sum(s1) / H; s2 = warp_sum(s2) / H;
    bf16* dr = dx + (size_t)r * H;
    for (int c = lane * 8; c < H; c += 256) {
      float xv[8], gv[8], o[8];
      load8(xr + c, xv); load8(gr + c, gv);
#pragma unroll
      for (int i = 0; i < 8; i++) {
        const float xh = (xv[i] - mu) * rs;
        o[i] = rs * (gv[i] * gamma[c + i] - s1 - xh * s2);
      }
      store8(dr + c, o);
    }
  }
  __syncthreads();
  float* out = part + (size_t)blockIdx.x * 2 * H;
  for (int c = threadIdx.x; c < 2 * H; c += blockDim.x)
    out[c] = sm[c] + sm[2 * H + c] + sm[4 * H + c] + sm[6 * H + c];
}

// out[c] = sum_p part[p][c]  (fixed order)
__global__ void reduce_partials_kernel(const float* __restrict__ part, float* __restrict__ out, int parts, int n) {
  pdl_wait();       // launched as a dependent of the kernel that writes `part`
  pdl_trigger();
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= n) return;
  float s = 0;
  for (int p = 0; p < parts; p++) s += part[(size_t)p * n + c];
  out[c] = s;
}

// The same, four columns per thread, for long vectors: one column per thread needs 12288 CTAs for 3 M columns, and starting them takes
// longer than their reads, which the L2 still holds. 3 partials of 3 M columns 14.0 -> 5.1 us, 4 of 1 M 5.3 -> 3.4, 8 of 2.4 M 11.4 -> 7.4.
__global__ void __launch_bounds__(256)
reduce_partials_wide_kernel(const float4* part, float4* __restrict__ out, int parts, int n4) {
  pdl_wait();
  pdl_trigger();
  const int c = blockIdx.x * 256 + threadIdx.x;
  if (c >= n4) return;
  float4 s = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll 4
  for (int p = 0; p < parts; p++) {
    const float4 v = part[(size_t)p * n4 + c];
    s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
  }
  out[c] = s;
}

// The same for many partials of a short vector (LayerNorm's 148 to 444 x 2H): 32 x 32 threads per 32 columns, thread (cx, py)
// adds partials py, py + 32, ..., then the 32 rows are added in a fixed order. One thread per column walking all the
// partials serially took longer than the LayerNorm backward sweep it follows.
__global__ void __launch_bounds__(1024)
reduce_partials_tall_kernel(const float* __restrict__ part, float* __restrict__ out, int parts, int n) {
  pdl_wait();
  pdl_trigger();
  __shared__ float sm[32][33];
  const int cx = threadIdx.x, py = threadIdx.y;
  const int c = blockIdx.x * 32 + cx;
  float s = 0;
  if (c < n)
    for (int p = py; p < parts; p += 32) s += part[(size_t)p * n + c];
  sm[py][cx] = s;
  __syncthreads();
  if (py == 0 && c < n) {
    float t = 0;
#pragma unroll
    for (int j = 0; j < 32; j++) t += sm[j][cx];
    out[c] = t;
  }
}

// ----------------------------------------------------------------------- GELU
__device__ __forceinline__ float gelu_f(float x) { return 0.5f * x * (1.0f + erff(x * 0.70710678118654752f)); }
__device__ __forceinline__ float gelu_grad_f(float x) {
  const float cdf = 0.5f * (1.0f + erff(x * 0.70710678118654752f));
  return cdf + x * 0.3989422804014327f * __expf(-0.5f * x * x);
}
__global__ void gelu_fwd_kernel(const bf16* __restrict__ x, bf16* __restrict__ y, size_t n8) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n8; i += (size_t)gridDim.x * blockDim.x) {
    float v[8];
    load8(x + i * 8, v);
#pragma unroll
    for (int k = 0; k < 8; k++) v[k] = gelu_f(v[k]);
    store8(y + i * 8, v);
  }
}
__global__ void gelu_bwd_kernel(const bf16* __restrict__ dy, const bf16* __restrict__ x, bf16* __restrict__ dx, size_t n8) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n8; i += (size_t)gridDim.x * blockDim.x) {
    float v[8], g[8];
    load8(x + i * 8, v); load8(dy + i * 8, g);
#pragma unroll
    for (int k = 0; k < 8; k++) g[k] *= gelu_grad_f(v[k]);
    store8(dx + i * 8, g);
  }
}

// ------------------------------------------------------- softmax cross-entropy
// One CTA per row of `logits` [rows, ld] (V valid columns, bf16). Writes the
// row loss (0 for ignored rows) and overwrites the row with
// (softmax - onehot) * scale, scale = 1 / max(1, *valid_count).
__global__ void __launch_bounds__(256)
softmax_xent_kernel(bf16* __restrict__ logits, const int64_t* __restrict__ target, float* __restrict__ row_loss,
                    const float* __restrict__ valid_count, int V, int ld, int ignore_index) {
  __shared__ float red[16];
  const int r = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  bf16* row = logits + (size_t)r * ld;
  const int64_t t = target[r];
  const int V8 = V & ~7;
  if (t == ignore_index) {
    for (int c = tid * 8; c < ld; c += 256 * 8) *reinterpret_cast<uint4*>(row + c) = make_uint4(0, 0, 0, 0);
    if (tid == 0) row_loss[r] = 0;
    return;
  }
  float mx = -INFINITY;
  for (int c = tid * 8; c < V8; c += 256 * 8) { float v[8]; load8(row + c, v);
#pragma unroll
    for (int i = 0; i < 8; i++) mx = fmaxf(mx, v[i]); }
  for (int c = V8 + tid; c < V; c += 256) mx = fmaxf(mx, __bfloat162float(row[c]));
  mx = warp_max(mx);
  if (lane == 0) red[warp] = mx;
  __syncthreads();
  mx = red[0];
#pragma unroll
  for (int i = 1; i < 8; i++) mx = fmaxf(mx, red[i]);
  float s = 0;
  for (int c = tid * 8; c < V8; c += 256 * 8) { float v[8]; load8(row + c, v);
#pragma unroll
    for (int i = 0; i < 8; i++) s += __expf(v[i] - mx); }
  for (int c = V8 + tid; c < V; c += 256) s += __expf(__bfloat162float(row[c]) - mx);
  s = warp_sum(s);
  if (lane == 0) red[8 + warp] = s;
  __syncthreads();
  s = 0;
#pragma unroll
  for (int i = 0; i < 8; i++) s += red[8 + i];
  const float lse = mx + __logf(s);
  const float scale = 1.0f / fmaxf(1.0f, *valid_count);
  const float inv = scale / s;
  if (tid == 0) row_loss[r] = (lse - __bfloat162float(row[t])) * scale;
  __syncthreads();   // row[t] read before it is overwritten
  for (int c = tid * 8; c < V8; c += 256 * 8) {
    float v[8];
    load8(row + c, v);
#pragma unroll
    for (int i = 0; i < 8; i++) v[i] = __expf(v[i] - mx) * inv - ((int64_t)(c + i) == t ? scale : 0.0f);
    store8(row + c, v);
  }
  for (int c = V8 + tid; c < ld; c += 256)
    row[c] = c < V ? __float2bfloat16(__expf(__bfloat162float(row[c]) - mx) * inv - ((int64_t)c == t ? scale : 0.0f))
                   : __float2bfloat16(0.0f);
}

// -------------------------------------------------------------------- softmax
// Row softmax of scale * x (one warp per row, the row is re-read from L1), and its
// backward ds = scale * p * (dp - sum(dp * p)). Used by the unfused attention path.
__global__ void __launch_bounds__(128)
softmax_fwd_kernel(const bf16* __restrict__ x, bf16* __restrict__ y, int64_t rows, int S, float scale) {
  const int lane = threadIdx.x & 31;
  for (int64_t r = (int64_t)blockIdx.x * 4 + (threadIdx.x >> 5); r < rows; r += (int64_t)gridDim.x * 4) {
    const bf16* xr = x + r * S;
    float mx = -INFINITY;
    for (int c = lane * 8; c < S; c += 256) { float v[8]; load8(xr + c, v);
#pragma unroll
      for (int i = 0; i < 8; i++) mx = fmaxf(mx, v[i]); }
    mx = warp_max(mx) * scale;
    float sum = 0;
    for (int c = lane * 8; c < S; c += 256) { float v[8]; load8(xr + c, v);
#pragma unroll
      for (int i = 0; i < 8; i++) sum += __expf(v[i] * scale - mx); }
    const float inv = 1.0f / warp_sum(sum);
    bf16* yr = y + r * S;
    for (int c = lane * 8; c < S; c += 256) {
      float v[8];
      load8(xr + c, v);
#pragma unroll
      for (int i = 0; i < 8; i++) v[i] = __expf(v[i] * scale - mx) * inv;
      store8(yr + c, v);
    }
  }
}
__global__ void __launch_bounds__(128)
softmax_bwd_kernel(const bf16* __restrict__ dp, const bf16* __restrict__ p, bf16* __restrict__ ds, int64_t rows, int S,
                   float scale) {
  const int lane = threadIdx.x & 31;
  for (int64_t r = (int64_t)blockIdx.x * 4 + (threadIdx.x >> 5); r < rows; r += (int64_t)gridDim.x * 4) {
    const bf16 *gr = dp + r * S, *pr = p + r * S;
    float dot = 0;
    for (int c = lane * 8; c < S; c += 256) { float g[8], q[8]; load8(gr + c, g); load8(pr + c, q);
#pragma unroll
      for (int i = 0; i < 8; i++) dot += g[i] * q[i]; }
    dot = warp_sum(dot);
    bf16* dr = ds + r * S;
    for (int c = lane * 8; c < S; c += 256) {
      float g[8], q[8];
      load8(gr + c, g); load8(pr + c, q);
#pragma unroll
      for (int i = 0; i < 8; i++) g[i] = scale * q[i] * (g[i] - dot);
      store8(dr + c, g);
    }
  }
}

// -------------------------------------------------------------- column sums
// part[blockIdx.y][c] = sum over this CTA's row range of g[r][c]  (bf16 in, fp32 out)
__global__ void __launch_bounds__(256)
colsum_partial_kernel(const bf16* __restrict__ g, float* __restrict__ part, int rows, int cols, int ld, int rows_per) {
  pdl_trigger();
  pdl_wait();
  const int c = (blockIdx.x * 256 + threadIdx.x) * 2;
  if (c >= cols) return;
  const int r0 = blockIdx.y * rows_per, r1 = min(rows, r0 + rows_per);
  float s0 = 0, s1 = 0;
  for (int r = r0; r < r1; r++) {
    const __nv_bfloat162 v = *reinterpret_cast<const __nv_bfloat162*>(g + (size_t)r * ld + c);
    const float2 f = __bfloat1622float2(v);
    s0 += f.x; s1 += f.y;
  }
  part[(size_t)blockIdx.y * cols + c] = s0;
  if (c + 1 < cols) part[(size_t)blockIdx.y * cols + c + 1] = s1;
}

// Wide variant: 16-byte loads (8 columns per thread), 8 row lanes per CTA with independent accumulators,
// folded through shared memory. One CTA covers 256 columns x rows_per rows.
__global__ void __launch_bounds__(256)
colsum_partial8_kernel(const bf16* __restrict__ g, float* __restrict__ part, int rows, int cols, int ld, int rows_per) {
  pdl_trigger();
  pdl_wait();
  __shared__ float red[8][256 + 8];
  const int cg = threadIdx.x & 31, rl = threadIdx.x >> 5;       // column group (8 columns), row lane
  const int c = blockIdx.x * 256 + cg * 8;
  const int r0 = blockIdx.y * rows_per, r1 = min(rows, r0 + rows_per);
  float acc[8];
#pragma unroll
  for (int j = 0; j < 8; j++) acc[j] = 0.0f;
  if (c < cols) {
#pragma unroll 4
    for (int r = r0 + rl; r < r1; r += 8) {
      const uint4 v = *reinterpret_cast<const uint4*>(g + (size_t)r * ld + c);
      const __nv_bfloat162* b = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
      for (int e = 0; e < 4; e++) { const float2 f = __bfloat1622float2(b[e]); acc[2 * e] += f.x; acc[2 * e + 1] += f.y; }
    }
  }
#pragma unroll
  for (int j = 0; j < 8; j++) red[rl][cg * 8 + j] = acc[j];
  __syncthreads();
  const int col = blockIdx.x * 256 + threadIdx.x;
  if (col < cols) {
    float s = 0.0f;
#pragma unroll
    for (int l = 0; l < 8; l++) s += red[l][threadIdx.x];     // fixed order
    part[(size_t)blockIdx.y * cols + col] = s;
  }
}

// Few rows, one launch: a cluster of eight CTAs takes 64 columns, an eighth of the rows each; 16-byte loads (8 columns per thread, 32
// row lanes per CTA), folded through shared memory, then CTA r adds up columns 8 r .. 8 r + 7 of all eight in their order. Bound by latency,
// of which a second launch is the larger part. The lines (us, the two kernels above -> this one): with more rows a CTA has too many to itself,
// 4096 x 768 4.9 -> 3.6, 4096 x 3072 8.8 -> 7.4, 5120 x 1024 5.9 -> 5.6, 5120 x 3072 9.7 both, 7168 x 1024 8.9 -> 9.4, 8192 x 1024 8.1 -> 9.5; with more
// columns the clusters are not all resident, 256 x 6144 4.3 -> 3.6, 2048 x 6144 8.5 -> 6.9, 4096 x 6144 11.2 -> 10.3, but 256 x 8192 4.3 -> 5.7,
// 2048 x 8192 9.2 -> 11.0, 64 x 30528 3.3 -> 12.8. Within them this one is faster but for a few (3584 x 4096 8.8 -> 9.4).
constexpr int kSumCols = 64, kSumCtas = 8, kSumLanes = 32, kSumMostRows = 4096, kSumMostCols = 6144;
__global__ void __cluster_dims__(1, kSumCtas, 1) __launch_bounds__(256)
colsum_cluster_kernel(const bf16* g, float* __restrict__ out, int rows, int cols, int ld) {
  __shared__ float red[kSumLanes][kSumCols + 4], quarter[4][kSumCols], sum[kSumCols];
  pdl_trigger();
  pdl_wait();
  const int tid = threadIdx.x, cg = tid & 7, rl = tid >> 3;      // column group (8 columns), row lane
  const int c = blockIdx.x * kSumCols + cg * 8;
  const int r0 = (int)((int64_t)rows * blockIdx.y / kSumCtas), r1 = (int)((int64_t)rows * (blockIdx.y + 1) / kSumCtas);
  float acc[8];
#pragma unroll
  for (int j = 0; j < 8; j++) acc[j] = 0.0f;
  if (c < cols) {
#pragma unroll 8
    for (int r = r0 + rl; r < r1; r += kSumLanes) {
      const uint4 v = *reinterpret_cast<const uint4*>(g + (size_t)r * ld + c);
      const __nv_bfloat162* b = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
      for (int e = 0; e < 4; e++) { const float2 f = __bfloat1622float2(b[e]); acc[2 * e] += f.x; acc[2 * e + 1] += f.y; }
    }
  }
#pragma unroll
  for (int j = 0; j < 8; j++) red[rl][cg * 8 + j] = acc[j];
  __syncthreads();
  {
    const int col = tid & (kSumCols - 1), q = tid / kSumCols;
    float s = 0.0f;
#pragma unroll
    for (int l = 0; l < kSumLanes / 4; l++) s += red[q * (kSumLanes / 4) + l][col];   // fixed order
    quarter[q][col] = s;
  }
  __syncthreads();
  if (tid < kSumCols) sum[tid] = (quarter[0][tid] + quarter[1][tid]) + (quarter[2][tid] + quarter[3][tid]);
  const cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
  cluster.sync();
  const int mine = (int)blockIdx.y * 8 + tid, col = blockIdx.x * kSumCols + mine;
  if (tid < 8 && col < cols) {
    float s = 0.0f;
#pragma unroll
    for (int k = 0; k < kSumCtas; k++) s += cluster.map_shared_rank(sum, k)[mine];
    out[col] = s;
  }
  cluster.sync();                                                // the others' sums are read until here
}

// Both of a linear layer's sums in one launch, each in the order that it has by itself: the first CTAs four columns of the weight gradient a
// thread, the others 32 columns of the bias gradient each, 8 threads to a column.
__global__ void __launch_bounds__(256)
reduce_weight_bias_kernel(const float4* part, float4* __restrict__ out, int parts, int n4, const float* bias_part, float* __restrict__ bias_out,
                          int bias_parts, int bias_n, unsigned first) {
  pdl_wait();
  pdl_trigger();
  if (blockIdx.x < first) {
    const int c = blockIdx.x * 256 + threadIdx.x;
    if (c >= n4) return;
    float4 s = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll 4
    for (int p = 0; p < parts; p++) {
      const float4 v = part[(size_t)p * n4 + c];
      s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
    }
    out[c] = s;
    return;
  }
  __shared__ float sm[8][33];
  const int cx = threadIdx.x & 31, py = threadIdx.x >> 5, c = (blockIdx.x - first) * 32 + cx;
  float s = 0;
  if (c < bias_n)
    for (int p = py; p < bias_parts; p += 8) s += bias_part[(size_t)p * bias_n + c];
  sm[py][cx] = s;
  __syncthreads();
  if (py == 0 && c < bias_n) {
    float t = 0;
#pragma unroll
    for (int j = 0; j < 8; j++) t += sm[j][cx];
    bias_out[c] = t;
  }
}

// ------------------------------------------------------------ weights to bf16
// y = bf16(x), rounded to nearest even. Stands between two dependent kernels where a weight has no bf16 copy; as one of them its launch
// and start are hidden, and torch's cast took 10 us of the host (1024 -> 512, 1 x 1 and 7 x 7, batch 16: 180 -> 171 us, all host).
__global__ void __launch_bounds__(256) cast_bf16_kernel(const float* x, bf16* __restrict__ y, size_t n, int wide) {
  pdl_trigger();
  pdl_wait();
  const size_t i = ((size_t)blockIdx.x * 256 + threadIdx.x) * 8;
  if (i + 8 <= n && wide) {
    const float4 a = reinterpret_cast<const float4*>(x + i)[0], b = reinterpret_cast<const float4*>(x + i)[1];
    const float v[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    store8(y + i, v);
  } else {
    for (size_t k = i; k < i + 8 && k < n; k++) y[k] = __float2bfloat16(x[k]);
  }
}

// ------------------------------------------------------- image normalisation
// uint8 NHWC [n, 3] pixels -> bf16 NHWC padded to `cpad` channels (extra channels 0):
// y = (x - mean_c) / std_c with mean/std given in 0..255 units.
__global__ void u8_to_bf16_norm_kernel(const uint8_t* __restrict__ x, bf16* __restrict__ y, size_t pixels, int cpad,
                                       float m0, float m1, float m2, float i0, float i1, float i2) {
  for (size_t p = (size_t)blockIdx.x * blockDim.x + threadIdx.x; p < pixels; p += (size_t)gridDim.x * blockDim.x) {
    const uint8_t* s = x + p * 3;
    bf16* d = y + p * cpad;
    d[0] = __float2bfloat16(((float)s[0] - m0) * i0);
    d[1] = __float2bfloat16(((float)s[1] - m1) * i1);
    d[2] = __float2bfloat16(((float)s[2] - m2) * i2);
    for (int c = 3; c < cpad; c++) d[c] = __float2bfloat16(0.0f);
  }
}

}  // namespace nl
}  // namespace gcow

using namespace gcow::nl;

extern "C" {

int gcow_layernorm_fwd(const void* x, const float* gamma, const float* beta, void* y, float* mean, float* rstd,
                       int rows, int H, float eps, void* stream) {
  if (H % 8 || rows <= 0) return -1;
  const int want = (rows + 3) / 4;
#define GCOW_LN_FWD(K, CTAS) gcow::launch_dependent(K, dim3(want < 148 * (CTAS) ? want : 148 * (CTAS)), dim3(128), 0, (cudaStream_t)stream, \
                                                    (const bf16*)x, gamma, beta, (bf16*)y, mean, rstd, rows, H, eps)
  // As many CTAs as are resident: with six for every width, which is the widest rows' number, 65536 x 128 took 22.7 us (now 14.6), x
  // 256 25.1 (16.1), x 512 38.8 (28.0), x 768 51.0 (39.5); x 1024 51.6 as before.
  switch ((H + 255) / 256) {
    case 1: GCOW_LN_FWD(layernorm_fwd_rows_kernel<1>, kRowCtas<1>); break;
    case 2: GCOW_LN_FWD(layernorm_fwd_rows_kernel<2>, kRowCtas<2>); break;
    case 3: GCOW_LN_FWD(layernorm_fwd_rows_kernel<3>, kRowCtas<3>); break;
    case 4: GCOW_LN_FWD(layernorm_fwd_rows_kernel<4>, kRowCtas<4>); break;
    default: GCOW_LN_FWD(layernorm_fwd_kernel, 16); break;
  }
#undef GCOW_LN_FWD
  return (int)cudaGetLastError();
}

// Number of partial rows the backward writes at most; `part` must hold parts * 2 * H floats.
int gcow_layernorm_bwd_parts(int rows) { int g = (rows + 3) / 4; return g < 148 * 3 ? g : 148 * 3; }

int gcow_layernorm_bwd(const void* dy, const void* x, const float* gamma, const float* mean, const float* rstd,
                       void* dx, float* part, float* dgamma_dbeta, int rows, int H, void* stream) {
  if (H % 8 || rows <= 0 || H > 4096) return -1;
  const int most = gcow_layernorm_bwd_parts(rows);
  // 512 threads from where their sums' way through shared memory is less than what fewer partial sums save: 1024 x 1024 7.4 us with 128,
  // 8.5 with 512; 1280 8.8, 8.5; 2048 9.5, 8.7; the other widths change sides at the same place.
  const bool wide = rows > 1280;
  const int fit = (rows + 15) / 16, grid = H > 1024 || !wide ? most : fit < 148 ? fit : 148;
#define GCOW_LN_BWD(K, T, SMEM) do { \
    if ((SMEM) > 48 * 1024) { \
      static std::atomic<bool> allowed[64]; \
      int dev = 0; \
      cudaGetDevice(&dev); \
      if (dev >= 64 || !allowed[dev].load(std::memory_order_acquire)) { \
        const int e = (int)cudaFuncSetAttribute(K, cudaFuncAttributeMaxDynamicSharedMemorySize, 160 * 1024); \
        if (e) return e; \
        if (dev < 64) allowed[dev].store(true, std::memory_order_release); \
      } \
    } \
    gcow::launch_dependent(K, dim3(grid), dim3(T), SMEM, (cudaStream_t)stream, (const bf16*)dy, (const bf16*)x, gamma, mean, rstd, (bf16*)dx, part, rows, H); \
  } while (0)
#define GCOW_LN_ROWS(CH) do { \
    if (wide) GCOW_LN_BWD((layernorm_bwd_rows_kernel<CH, kLnWide>), kLnWide, (kLnBwdSmem<CH, kLnWide>)); \
    else GCOW_LN_BWD((layernorm_bwd_rows_kernel<CH, kLnNarrow>), kLnNarrow, (kLnBwdSmem<CH, kLnNarrow>)); \
  } while (0)
  switch ((H + 255) / 256) {
    case 1: GCOW_LN_ROWS(1); break;
    case 2: GCOW_LN_ROWS(2); break;
    case 3: GCOW_LN_ROWS(3); break;
    case 4: GCOW_LN_ROWS(4); break;
    default: GCOW_LN_BWD(layernorm_bwd_kernel, 128, (size_t)8 * H * sizeof(float)); break;
  }
#undef GCOW_LN_ROWS
#undef GCOW_LN_BWD
  gcow::launch_dependent(reduce_partials_tall_kernel, dim3((2 * H + 31) / 32), dim3(32, 32), 0, (cudaStream_t)stream, (const float*)part,
                   dgamma_dbeta, grid, 2 * H);
  return (int)cudaGetLastError();
}

int gcow_gelu_fwd(const void* x, void* y, uint64_t n, void* stream) {
  if (n % 8) return -1;
  if (!n) return 0;
  uint64_t n8 = n / 8; int grid = (int)((n8 + 255) / 256 < 148 * 16 ? (n8 + 255) / 256 : 148 * 16);
  gelu_fwd_kernel<<<grid, 256, 0, (cudaStream_t)stream>>>((const bf16*)x, (bf16*)y, n8);
  return (int)cudaGetLastError();
}
int gcow_gelu_bwd(const void* dy, const void* x, void* dx, uint64_t n, void* stream) {
  if (n % 8) return -1;
  if (!n) return 0;
  uint64_t n8 = n / 8; int grid = (int)((n8 + 255) / 256 < 148 * 16 ? (n8 + 255) / 256 : 148 * 16);
  gelu_bwd_kernel<<<grid, 256, 0, (cudaStream_t)stream>>>((const bf16*)dy, (const bf16*)x, (bf16*)dx, n8);
  return (int)cudaGetLastError();
}

int gcow_softmax_xent(void* logits, const int64_t* target, float* row_loss, const float* valid_count, int rows,
                      int V, int ld, int ignore_index, void* stream) {
  if (ld % 8 || V > ld || rows <= 0) return -1;
  softmax_xent_kernel<<<rows, 256, 0, (cudaStream_t)stream>>>((bf16*)logits, target, row_loss, valid_count, V, ld, ignore_index);
  return (int)cudaGetLastError();
}

// out[i] = sum_p part[p * n + i] in a fixed order (split-K partial products, bias partials).
int gcow_reduce_partials(const float* part, float* out, int parts, int64_t n, void* stream) {
  if (n <= 0 || parts <= 0 || n > 0x7fffffff) return -1;
  if (parts >= 64 && n <= 65536)
    gcow::launch_dependent(reduce_partials_tall_kernel, dim3((unsigned)((n + 31) / 32)), dim3(32, 32), 0, (cudaStream_t)stream, part, out,
                     parts, (int)n);
  // more partials than that are a longer chain per thread than fewer threads save: 16 of 1 M columns 6.2 us a column, 6.6 four
  else if (parts <= 8 && n >= 262144 && n % 4 == 0 && (((uintptr_t)part | (uintptr_t)out) & 15) == 0)
    gcow::launch_dependent(reduce_partials_wide_kernel, dim3((unsigned)((n / 4 + 255) / 256)), dim3(256), 0, (cudaStream_t)stream,
                           (const float4*)part, (float4*)out, parts, (int)(n / 4));
  else
    gcow::launch_dependent(reduce_partials_kernel, dim3((unsigned)((n + 255) / 256)), dim3(256), 0, (cudaStream_t)stream, part, out, parts,
                     (int)n);
  return (int)cudaGetLastError();
}

int gcow_softmax_fwd(const void* x, void* y, int64_t rows, int S, float scale, void* stream) {
  if (S % 8 || rows <= 0) return -1;
  int64_t g = (rows + 3) / 4; if (g > 148 * 16) g = 148 * 16;
  softmax_fwd_kernel<<<(int)g, 128, 0, (cudaStream_t)stream>>>((const bf16*)x, (bf16*)y, rows, S, scale);
  return (int)cudaGetLastError();
}
int gcow_softmax_bwd(const void* dp, const void* p, void* ds, int64_t rows, int S, float scale, void* stream) {
  if (S % 8 || rows <= 0) return -1;
  int64_t g = (rows + 3) / 4; if (g > 148 * 16) g = 148 * 16;
  softmax_bwd_kernel<<<(int)g, 128, 0, (cudaStream_t)stream>>>((const bf16*)dp, (const bf16*)p, (bf16*)ds, rows, S, scale);
  return (int)cudaGetLastError();
}

// Column sums of a bf16 [rows, cols] matrix (ld even, cols even) into fp32 out[cols];
// `part` must hold gcow_colsum_parts(rows) * cols floats.
int gcow_colsum_parts(int rows) { int p = (rows + 127) / 128; return p < 128 ? (p < 1 ? 1 : p) : 128; }
// Kernels that gcow_colsum launches: one (`part` is not used), or the partial sums and their reduction.
int gcow_colsum_launches(const void* g, int rows, int cols, int ld) {
  return rows <= kSumMostRows && cols <= kSumMostCols && cols % 8 == 0 && ld % 8 == 0 && ((uintptr_t)g & 15) == 0 ? 1 : 2;
}
int gcow_colsum(const void* g, float* part, float* out, int rows, int cols, int ld, void* stream) {
  if (cols % 2 || ld % 2 || rows <= 0) return -1;
  if (gcow_colsum_launches(g, rows, cols, ld) == 1) {
    gcow::launch_dependent(colsum_cluster_kernel, dim3((cols + kSumCols - 1) / kSumCols, kSumCtas), dim3(256), 0, (cudaStream_t)stream,
                           (const bf16*)g, out, rows, cols, ld);
    return (int)cudaGetLastError();
  }
  const int parts = gcow_colsum_parts(rows);
  const int rows_per = (rows + parts - 1) / parts;
  if (cols % 8 == 0 && ld % 8 == 0 && ((uintptr_t)g & 15) == 0) {
    dim3 grid((cols + 255) / 256, parts);
    gcow::launch_dependent(colsum_partial8_kernel, grid, dim3(256), 0, (cudaStream_t)stream, (const bf16*)g, part, rows, cols, ld, rows_per);
  } else {
    dim3 grid((cols / 2 + 255) / 256, parts);
    gcow::launch_dependent(colsum_partial_kernel, grid, dim3(256), 0, (cudaStream_t)stream, (const bf16*)g, part, rows, cols, ld, rows_per);
  }
  if (parts >= 64)
    gcow::launch_dependent(reduce_partials_tall_kernel, dim3((cols + 31) / 32), dim3(32, 32), 0, (cudaStream_t)stream, (const float*)part,
                     out, parts, cols);
  else
    gcow::launch_dependent(reduce_partials_kernel, dim3((cols + 255) / 256), dim3(256), 0, (cudaStream_t)stream, (const float*)part, out,
                     parts, cols);
  return (int)cudaGetLastError();
}
// Both sums of partial results of a linear layer: a weight gradient of n elements (parts 0: there is none to add up, and n, part and out are not
// looked at) and a bias gradient of bias_n. n a multiple of 4, part and out at multiples of 16 bytes.
int gcow_reduce_weight_bias(const float* part, float* out, int parts, int64_t n, const float* bias_part, float* bias_out, int bias_parts,
                            int bias_n, void* stream) {
  if (parts < 0 || bias_parts <= 0 || bias_n <= 0) return -1;
  if (!parts) n = 0;
  else if (n < 0 || n % 4 || n / 4 > 0x7fffffff - 255 || (((uintptr_t)part | (uintptr_t)out) & 15)) return -1;
  const unsigned first = (unsigned)((n / 4 + 255) / 256);
  gcow::launch_dependent(reduce_weight_bias_kernel, dim3(first + (unsigned)((bias_n + 31) / 32)), dim3(256), 0, (cudaStream_t)stream,
                         (const float4*)part, (float4*)out, parts, (int)(n / 4), bias_part, bias_out, bias_parts, bias_n, first);
  return (int)cudaGetLastError();
}

int gcow_cast_bf16(const float* x, void* y, uint64_t n, void* stream) {
  if (!n) return 0;
  const uint64_t ctas = (n + 2047) / 2048;
  if (ctas > 0x7fffffff) return -1;
  const int wide = (((uintptr_t)x | (uintptr_t)y) & 15) == 0;
  gcow::launch_dependent(cast_bf16_kernel, dim3((unsigned)ctas), dim3(256), 0, (cudaStream_t)stream, x, (bf16*)y, (size_t)n, wide);
  return (int)cudaGetLastError();
}

int gcow_u8_to_bf16_norm(const void* x, void* y, uint64_t pixels, int cpad, const float* mean3, const float* std3,
                         void* stream) {
  if (!pixels) return 0;
  int grid = (int)((pixels + 255) / 256 < 148 * 16 ? (pixels + 255) / 256 : 148 * 16);
  u8_to_bf16_norm_kernel<<<grid, 256, 0, (cudaStream_t)stream>>>((const uint8_t*)x, (bf16*)y, pixels, cpad, mean3[0], mean3[1],
                                                                 mean3[2], 1.0f / std3[0], 1.0f / std3[1], 1.0f / std3[2]);
  return (int)cudaGetLastError();
}

}  // extern "C"
