// Fused BatchNorm2d (+ residual add) (+ ReLU) for channels-last bf16 activations
// (sm_100a), forward and backward, training and inference statistics.
//
// x is viewed as R = N*H*W rows of C channels. A thread owns 8 consecutive
// channels (one 16-byte access) of every (256*8/C)-th row, keeps its partial
// sums in fp32 registers and the CTA folds them per channel; per-CTA partials
// are summed in a fixed order by a second small kernel, which also derives the
// per-channel scale/shift and updates the running statistics. The normalise
// pass then applies y = x*scale + shift (+ residual), optional ReLU, in one
// read-modify-write sweep, so the add and the activation never touch memory on
// their own, and records the ReLU outcome as one bit per element (one byte per
// thread and row). Backward mirrors it: one sweep for dgamma/dbeta (reading that
// bit mask instead of the activations, and writing the masked gradient out when a
// residual branch needs it), one sweep for dx.
//
// The reference's ResNet uses nn.BatchNorm2d + ReLU + add as separate ATen /
// cuDNN operators (hw/models/resenet.py:12-22,28-40,80-89).
#include <cooperative_groups.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <atomic>
#include <type_traits>

#include "pdl.cuh"
#include <stdlib.h>
#include <stdint.h>

namespace gcow {
namespace bn {



typedef __nv_bfloat16 bf16;
constexpr int kThreads = 256;
// Every sweep over the tensor is launched with at most this many CTAs per SM, and compiled for exactly as many: the sweeps are bound by how
// many loads are in flight, so each thread gets the registers (80) that keep several rows' loads outstanding. Which operands a sweep has (a
// residual, a second gradient, a ReLU and its mask) is a template argument: as run-time conditions inside the unrolled loop they kept each
// row's loads behind the row before. 256 x 512 x 28 x 28, without the template and the bound -> with both: forward 114 -> 110 us, with ReLU
// 126 -> 113, with residual and ReLU 165 -> 138; backward 192 -> 187, 250 -> 193 and 260 -> 221 us, with a second gradient 315 -> 253.
// The bound at 4 CTAs or the grid at 6 made the backward slower (55 -> 61..64 us for 256 x 128 x 28 x 28). Rows unrolled: as many as the 80
// registers hold, measured at 2, 3, 4, 6 and 8.
constexpr int kSweepCtas = 3;

__device__ __forceinline__ void load8(const bf16* p, float (&v)[8]) {
  uint4 u = *reinterpret_cast<const uint4*>(p);
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

// Fold per-thread sums a[8], b[8] over the threads that share a channel group and
// write them to part[blockIdx.x][0][C] / [1][C].
__device__ __forceinline__ void cta_fold(const float (&a)[8], const float (&b)[8], int C, float* __restrict__ part) {
  __shared__ float sm[kThreads * 17];          // 16 values per thread, padded against bank conflicts
  const int groups = C / 8, tid = threadIdx.x;
  float* mine = sm + tid * 17;
#pragma unroll
  for (int i = 0; i < 8; i++) { mine[i] = a[i]; mine[8 + i] = b[i]; }
  __syncthreads();
  const int lanes = kThreads / groups;          // threads per channel group (>= 1)
  for (int idx = tid; idx < groups * 16; idx += kThreads) {
    const int g = idx / 16, k = idx % 16;
    float s = 0;
    for (int j = 0; j < lanes; j++) s += sm[(j * groups + g) * 17 + k];
    const int c = g * 8 + (k & 7);
    part[(size_t)blockIdx.x * 2 * C + (k < 8 ? 0 : C) + c] = s;
  }
}

// ---- forward statistics: partial sum(x), sum(x^2)
__global__ void __launch_bounds__(kThreads, kSweepCtas)
stats_kernel(const bf16* __restrict__ x, float* __restrict__ part, int64_t R, int C) {
  pdl_trigger();
  pdl_wait();       // launched under the tail of the kernel that writes x
  const int groups = C / 8, g = threadIdx.x % groups, r0 = threadIdx.x / groups, rstep = kThreads / groups;
  float s[8] = {0, 0, 0, 0, 0, 0, 0, 0}, q[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll 8
  for (int64_t r = (int64_t)blockIdx.x * rstep + r0; r < R; r += (int64_t)gridDim.x * rstep) {
    float v[8];
    load8(x + r * C + g * 8, v);
#pragma unroll
    for (int i = 0; i < 8; i++) { s[i] += v[i]; q[i] += v[i] * v[i]; }
  }
  cta_fold(s, q, C, part);
}

// The sums of the CTAs' partials for 8 channels (a sector of each partial), in double precision: a variance is a difference of two large sums.
// Thread (channel, row) adds partials row, row + 128, ... with the loads of a turn all on their way before the first addition (partials past
// the end count as zeros). Then a warp's four rows are added by shuffles and the warps' sums by the first warp, each in an order of its
// own, so the result does not depend on scheduling. Returns true in the 8 threads that hold the channels' sums.
// Bound by latency: the launch, one trip to the L2 (three sweep CTAs an SM leave at most 444 partials) and the fold. With 32 channels a CTA, four
// trips and every thread repeating the last fold in double precision, forward of 256 x 128 x 28 x 28 31.2 us, now 29.5, x 64 x 56 x 56 55.8, 54.7,
// 16 x 64 x 56 x 56 10.8, 9.2; backward 52.6, 51.9, the same, 12.3, 11.6. Fewer threads and more trips are slower: 512 threads in turns of 7 30.3, 256
// 32.7, 128 35.4. Two CTAs of 32 registers fit on an SM: at 50 registers 256 x 2048 x 7 x 7, which has 256 CTAs here, takes 37.8 us instead of 33.3.
constexpr int kFinX = 8, kFinY = 128, kFinThreads = kFinX * kFinY, kFinWarps = kFinThreads / 32;
__device__ __forceinline__ bool fold_partials(const float* __restrict__ part, int parts, int C, int c, double& s, double& q) {
  constexpr int TURN = 4;
  __shared__ double sm[2][kFinWarps][kFinX];
  const int row = threadIdx.x / kFinX, lane = threadIdx.x % 32, warp = threadIdx.x / 32;
  s = 0; q = 0;
#pragma unroll 1
  for (int p0 = row; p0 < parts; p0 += TURN * kFinY) {
    float a[TURN], b[TURN];
#pragma unroll
    for (int j = 0; j < TURN; j++) {
      const float* from = part + (size_t)(p0 + j * kFinY) * 2 * C + c;
      const bool there = p0 + j * kFinY < parts;
      a[j] = there ? from[0] : 0.0f; b[j] = there ? from[C] : 0.0f;
    }
#pragma unroll
    for (int j = 0; j < TURN; j++) { s += a[j]; q += b[j]; }
  }
  auto rows = [](double v) {      // the four rows of a warp, to all of its lanes
#pragma unroll
    for (int m = kFinX; m < 32; m *= 2) v += __shfl_xor_sync(~0u, v, m);
    return v;
  };
  s = rows(s); q = rows(q);
  if (lane < kFinX) { sm[0][warp][lane] = s; sm[1][warp][lane] = q; }
  __syncthreads();
  if (warp != 0) return false;
  s = 0; q = 0;
#pragma unroll
  for (int j = lane / kFinX; j < kFinWarps; j += 32 / kFinX) { s += sm[0][j][lane % kFinX]; q += sm[1][j][lane % kFinX]; }
  s = rows(s); q = rows(q);
  return lane < kFinX;
}

// ---- finalize forward: mean/rstd, scale/shift, running statistics
__global__ void __launch_bounds__(kFinThreads, 2048 / kFinThreads)
finalize_fwd_kernel(const float* __restrict__ part, int parts, int C, int64_t R, float eps, float momentum,
                    const float* __restrict__ gamma, const float* __restrict__ beta,
                    float* __restrict__ mean, float* __restrict__ rstd, float* __restrict__ scale,
                    float* __restrict__ shift, float* __restrict__ run_mean, float* __restrict__ run_var) {
  pdl_wait();
  pdl_trigger();
  const int c = blockIdx.x * kFinX + threadIdx.x % kFinX;      // C is a multiple of kFinX
  double s, q;
  if (!fold_partials(part, parts, C, c, s, q)) return;
  const double mu = s / (double)R;
  double var = q / (double)R - mu * mu;
  if (var < 0) var = 0;
  const float rs = rsqrtf((float)var + eps);
  mean[c] = (float)mu; rstd[c] = rs;
  const float sc = gamma[c] * rs;
  scale[c] = sc; shift[c] = beta[c] - (float)mu * sc;
  if (run_mean) {
    const double unbiased = R > 1 ? var * (double)R / (double)(R - 1) : var;
    run_mean[c] = (1.0f - momentum) * run_mean[c] + momentum * (float)mu;
    run_var[c] = (1.0f - momentum) * run_var[c] + momentum * (float)unbiased;
  }
}

// scale/shift from given (running) statistics, for inference
__global__ void affine_from_stats_kernel(const float* __restrict__ gamma, const float* __restrict__ beta,
                                         const float* __restrict__ mean_in, const float* __restrict__ var_in, float eps,
                                         int C, float* __restrict__ scale, float* __restrict__ shift) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= C) return;
  const float sc = gamma[c] * rsqrtf(var_in[c] + eps);
  scale[c] = sc; shift[c] = beta[c] - mean_in[c] * sc;
}

// ---- normalise: y = x*scale + shift (+ residual when ADD) (ReLU when RELU, its outcome to the mask when RELU is 2)
// ROWS: how many are unrolled. Behind the statistics, whose last rows the L2 still holds, eight without other operands; where x comes from
// memory (inference) four: 256 x 64 x 56 x 56 38.0 -> 36.5 us, 32 x 1024 x 14 x 14 7.9 -> 7.3; training with four 256 x 128 x 28 x 28 31.3 -> 32.9.
template <bool ADD, int RELU, int ROWS = ADD ? 3 : RELU ? 4 : 8>
__global__ void __launch_bounds__(kThreads, kSweepCtas)
apply_kernel(const bf16* __restrict__ x, const bf16* __restrict__ residual, bf16* __restrict__ y,
             uint8_t* __restrict__ mask, const float* __restrict__ scale, const float* __restrict__ shift, int64_t R,
             int C) {
  pdl_wait();
  pdl_trigger();    // the consumer of y may set itself up meanwhile
  const int groups = C / 8, g = threadIdx.x % groups, r0 = threadIdx.x / groups, rstep = kThreads / groups;
  float sc[8], sh[8];
#pragma unroll
  for (int i = 0; i < 8; i++) { sc[i] = scale[g * 8 + i]; sh[i] = shift[g * 8 + i]; }
#pragma unroll ROWS
  for (int64_t r = (int64_t)blockIdx.x * rstep + r0; r < R; r += (int64_t)gridDim.x * rstep) {
    const int64_t off = r * C + g * 8;
    float v[8];
    load8(x + off, v);
#pragma unroll
    for (int i = 0; i < 8; i++) v[i] = v[i] * sc[i] + sh[i];
    if (ADD) {
      float w[8];
      load8(residual + off, w);
#pragma unroll
      for (int i = 0; i < 8; i++) v[i] += w[i];
    }
    if (RELU) {
      uint32_t bits = 0;
#pragma unroll
      for (int i = 0; i < 8; i++) { bits |= (v[i] > 0.0f ? 1u : 0u) << i; v[i] = fmaxf(v[i], 0.0f); }
      if (RELU == 2) mask[r * groups + g] = (uint8_t)bits;      // bit i: channel g*8+i passed the ReLU
    }
    store8(y + off, v);
  }
}

// ---- backward sweep 1: partial sum(g), sum(g*xhat); g = dy (+ dy2) masked by (y > 0) when RELU.
// dy2 is a second gradient of the same output (the output feeds two consumers): adding it here saves
// the separate addition kernel and its three passes over the tensor.
// The masked gradient is written to gmask_out when OUT (the residual branch's gradient). TWO: there is a dy2, RELU: there is a mask.
template <bool TWO, bool RELU, bool OUT>
__global__ void __launch_bounds__(kThreads, kSweepCtas)
bwd_reduce_kernel(const bf16* __restrict__ dy, const bf16* __restrict__ dy2, const uint8_t* __restrict__ mask,
                  const bf16* __restrict__ x,
                  const float* __restrict__ mean, const float* __restrict__ rstd, bf16* __restrict__ gmask_out,
                  float* __restrict__ part, int64_t R, int C) {
  pdl_trigger();
  pdl_wait();
  const int groups = C / 8, g = threadIdx.x % groups, r0 = threadIdx.x / groups, rstep = kThreads / groups;
  float mu[8], rs[8], s[8] = {0, 0, 0, 0, 0, 0, 0, 0}, q[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll
  for (int i = 0; i < 8; i++) { mu[i] = mean[g * 8 + i]; rs[i] = rstd[g * 8 + i]; }
#pragma unroll (OUT && !TWO ? 3 : 4)
  for (int64_t r = (int64_t)blockIdx.x * rstep + r0; r < R; r += (int64_t)gridDim.x * rstep) {
    const int64_t off = r * C + g * 8;
    float gv[8], xv[8];
    load8(dy + off, gv);
    load8(x + off, xv);
    if (TWO) {
      float w[8];
      load8(dy2 + off, w);
#pragma unroll
      for (int i = 0; i < 8; i++) gv[i] += w[i];
    }
    if (RELU) {
      const uint32_t bits = mask[r * groups + g];
#pragma unroll
      for (int i = 0; i < 8; i++) gv[i] = (bits >> i) & 1u ? gv[i] : 0.0f;
    }
    if (OUT) store8(gmask_out + off, gv);
#pragma unroll
    for (int i = 0; i < 8; i++) { s[i] += gv[i]; q[i] += gv[i] * (xv[i] - mu[i]) * rs[i]; }
  }
  cta_fold(s, q, C, part);
}

// ---- finalize backward: dbeta = sum g, dgamma = sum g*xhat (fixed order)
__global__ void __launch_bounds__(kFinThreads, 2048 / kFinThreads)
finalize_bwd_kernel(const float* __restrict__ part, int parts, int C, float* __restrict__ dgamma,
                    float* __restrict__ dbeta) {
  pdl_wait();
  pdl_trigger();
  const int c = blockIdx.x * kFinX + threadIdx.x % kFinX;      // C is a multiple of kFinX
  double s, q;
  if (!fold_partials(part, parts, C, c, s, q)) return;
  dbeta[c] = (float)s; dgamma[c] = (float)q;
}

// ---- backward sweep 2: dx = gamma*rstd * (g - dbeta/R - xhat*dgamma/R). From the last row to the first: sweep 1 has just read the last
// ones, which the L2 still holds, and what reads dx next finds its first rows there. Backward of 256 x 128 x 28 x 28: 57.8 -> 55.4 us, x 2048 x
// 7 x 7 62.8 -> 60.7, x 64 x 56 x 56 102.3 -> 100.7, x 256 x 56 x 56 as before, all before the
// registers that kSweepCtas gives. (The forward's second sweep backwards: 33.5 -> 38.2 us.)
template <bool RELU>
__global__ void __launch_bounds__(kThreads, kSweepCtas)
bwd_dx_kernel(const bf16* __restrict__ dy, const uint8_t* __restrict__ mask, const bf16* __restrict__ x,
              const float* __restrict__ gamma, const float* __restrict__ mean, const float* __restrict__ rstd,
              const float* __restrict__ dgamma, const float* __restrict__ dbeta, bf16* __restrict__ dx, int64_t R, int C) {
  pdl_wait();
  pdl_trigger();
  const int groups = C / 8, g = threadIdx.x % groups, r0 = threadIdx.x / groups, rstep = kThreads / groups;
  float mu[8], rs[8], k0[8], k1[8], k2[8];
  const float invR = 1.0f / (float)R;
#pragma unroll
  for (int i = 0; i < 8; i++) {
    const int c = g * 8 + i;
    mu[i] = mean[c]; rs[i] = rstd[c];
    k0[i] = gamma[c] * rs[i];
    k1[i] = dbeta[c] * invR;
    k2[i] = dgamma[c] * invR;
  }
#pragma unroll 4
  for (int64_t r = R - 1 - (int64_t)blockIdx.x * rstep - r0; r >= 0; r -= (int64_t)gridDim.x * rstep) {
    const int64_t off = r * C + g * 8;
    float gv[8], xv[8];
    load8(dy + off, gv);
    load8(x + off, xv);
    if (RELU) {
      const uint32_t bits = mask[r * groups + g];
#pragma unroll
      for (int i = 0; i < 8; i++) gv[i] = (bits >> i) & 1u ? gv[i] : 0.0f;
    }
#pragma unroll
    for (int i = 0; i < 8; i++) gv[i] = k0[i] * (gv[i] - k1[i] - (xv[i] - mu[i]) * rs[i] * k2[i]);
    store8(dx + off, gv);
  }
}

// ------------------------------------------------------------------ one launch: a cluster takes CH channels
// Tensors that the shared memory of the clusters holds: a CTA reads its share of the rows of its cluster's channels once, keeps them, and
// the cluster adds up its sums through distributed shared memory, so the second sweep reads shared memory and there is nothing between the sweeps
// but a cluster barrier. The three launches spend most of a small tensor's time on their starts and ends and read it twice. Bound by latency up to a
// few MB, then by a row's 32 or 64 bytes per CTA and by the waves' phases, which load, wait and store alike. The rule is at held_plan.
constexpr int kHeldThreads = 512, kHeldWarps = kHeldThreads / 32, kHeldBytes = 104 * 1024;

__device__ __forceinline__ void unpack8(const uint4& u, float (&v)[8]) {
  const __nv_bfloat162* b = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
  for (int i = 0; i < 4; i++) { const float2 f = __bfloat1622float2(b[i]); v[2 * i] = f.x; v[2 * i + 1] = f.y; }
}
__device__ __forceinline__ uint4 pack8(const float (&v)[8]) {
  uint4 u;
  __nv_bfloat162* b = reinterpret_cast<__nv_bfloat162*>(&u);
#pragma unroll
  for (int i = 0; i < 4; i++) b[i] = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
  return u;
}
// The sums of a cluster's channels: a thread's of its 8, over the warp, the CTA and the cluster's CTAs, always in the same order. A thread's 13
// rows at most are added in fp32, everything behind them in double, as a variance is a difference of two large sums: with fp32 up to the CTA's 784 to 1568 rows its
// relative error at a mean of 10 (100) and a deviation of 1 was 5e-6 (6e-4). In the warp the lanes of a channel chunk halve the 16 sums between them, so
// that each exchanges 14 of them instead of 48. Thread c < CH has channel c's. The other CTAs' `mine` is read until the barrier that this
// arrives at completes.
template <int CH>
__device__ __forceinline__ void cluster_fold(cooperative_groups::cluster_group& cluster, const float (&s)[8], const float (&q)[8],
                                             double (&fold)[kHeldWarps][2 * CH], double (&mine)[2 * CH], double& s_out, double& q_out) {
  constexpr int CHUNKS = CH / 8;
  const int tid = threadIdx.x, lane = tid & 31;
  double v[16];
#pragma unroll
  for (int i = 0; i < 8; i++) { v[i] = s[i]; v[8 + i] = q[i]; }
  int first = 0;                                            // of the sums that the lane is left with
#pragma unroll
  for (int step = 0; step < (CHUNKS == 4 ? 3 : 4); step++) {
    const int d = CHUNKS << step, left = 8 >> step;
    const bool upper = lane & d;
#pragma unroll
    for (int i = 0; i < 8; i++) {
      if (i >= left) continue;
      const double other = __shfl_xor_sync(0xffffffffu, upper ? v[i] : v[i + left], d);
      v[i] = (upper ? v[i + left] : v[i]) + other;
    }
    if (upper) first += left;
  }
#pragma unroll
  for (int i = 0; i < CHUNKS / 2; i++) {
    const int k = first + i;
    fold[tid >> 5][(k >> 3) * CH + (lane % CHUNKS) * 8 + (k & 7)] = v[i];
  }
  __syncthreads();
  if (tid < 2 * CH) {
    double a[4] = {0, 0, 0, 0};
#pragma unroll
    for (int w = 0; w < kHeldWarps; w++) a[w & 3] += fold[w][tid];
    mine[tid] = (a[0] + a[1]) + (a[2] + a[3]);
  }
  cluster.sync();
  s_out = q_out = 0;
  if (tid < CH) {
    const int size = (int)cluster.num_blocks();
    for (int j = 0; j < size; j++) {
      const double* const other = cluster.map_shared_rank(&mine[0], j);
      s_out += other[tid];
      q_out += other[CH + tid];
    }
  }
}

template <int CH, bool ADD, int RELU>
__global__ void __launch_bounds__(kHeldThreads, 2)
held_fwd_kernel(const bf16* x, const bf16* residual, bf16* __restrict__ y, uint8_t* __restrict__ mask, const float* gamma, const float* beta,
                float* __restrict__ stats, float* run_mean, float* run_var, int R, int C, float eps, float momentum) {
  constexpr int CHUNKS = CH / 8, LANES = kHeldThreads / CHUNKS;
  extern __shared__ uint4 held[];                           // [rows][CHUNKS]
  __shared__ double fold[kHeldWarps][2 * CH], mine[2 * CH];
  __shared__ float affine[2][CH];
  cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
  const int size = (int)cluster.num_blocks(), rank = (int)cluster.block_rank(), tid = threadIdx.x, chunk = tid % CHUNKS, row = tid / CHUNKS;
  const int c0 = (int)(blockIdx.x / size) * CH, rows = (int)((int64_t)R * (rank + 1) / size - (int64_t)R * rank / size);
  const size_t at = ((int64_t)R * rank / size) * C + c0 + chunk * 8;
  float s[8] = {0, 0, 0, 0, 0, 0, 0, 0}, q[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  pdl_wait();
#pragma unroll 4
  for (int r = row; r < rows; r += LANES) {
    const uint4 u = *reinterpret_cast<const uint4*>(x + at + (size_t)r * C);
    held[r * CHUNKS + chunk] = u;
    float v[8];
    unpack8(u, v);
#pragma unroll
    for (int i = 0; i < 8; i++) { s[i] += v[i]; q[i] += v[i] * v[i]; }
  }
  double sum, sq;
  cluster_fold<CH>(cluster, s, q, fold, mine, sum, sq);
  if (tid < CH) {
    const int c = c0 + tid;
    const double mu = sum / (double)R;
    double var = sq / (double)R - mu * mu;
    if (var < 0) var = 0;
    const float rs = rsqrtf((float)var + eps), sc = gamma[c] * rs, sh = beta[c] - (float)mu * sc;
    affine[0][tid] = sc; affine[1][tid] = sh;
    if (rank == 0) {
      stats[c] = (float)mu; stats[C + c] = rs; stats[2 * C + c] = sc; stats[3 * C + c] = sh;
      if (run_mean) {
        const double unbiased = R > 1 ? var * (double)R / (double)(R - 1) : var;
        run_mean[c] = (1.0f - momentum) * run_mean[c] + momentum * (float)mu;
        run_var[c] = (1.0f - momentum) * run_var[c] + momentum * (float)unbiased;
      }
    }
  }
  cluster.barrier_arrive();
  __syncthreads();
  pdl_trigger();
  float sc[8], sh[8];
#pragma unroll
  for (int i = 0; i < 8; i++) { sc[i] = affine[0][chunk * 8 + i]; sh[i] = affine[1][chunk * 8 + i]; }
#pragma unroll 4
  for (int r = row; r - row < rows; r += LANES) {
    const bool there = r < rows;
    float v[8];
    if (there) {
      unpack8(held[r * CHUNKS + chunk], v);
#pragma unroll
      for (int i = 0; i < 8; i++) v[i] = v[i] * sc[i] + sh[i];
      if (ADD) {
        float w[8];
        load8(residual + at + (size_t)r * C, w);
#pragma unroll
        for (int i = 0; i < 8; i++) v[i] += w[i];
      }
    }
    if (RELU) {
      uint32_t bits = 0;
      if (there) {
#pragma unroll
        for (int i = 0; i < 8; i++) { bits |= (v[i] > 0.0f ? 1u : 0u) << i; v[i] = fmaxf(v[i], 0.0f); }
      }
      if (RELU == 2) {                                      // a row's bytes together
        bits <<= 8 * chunk;
#pragma unroll
        for (int d = 1; d < CHUNKS; d *= 2) bits |= __shfl_xor_sync(0xffffffffu, bits, d);
        if (there && chunk == 0) {
          uint8_t* const m = mask + (at + (size_t)r * C) / 8;
          if (CHUNKS == 4) *reinterpret_cast<uint32_t*>(m) = bits; else *reinterpret_cast<uint16_t*>(m) = (uint16_t)bits;
        }
      }
    }
    if (there) *reinterpret_cast<uint4*>(y + at + (size_t)r * C) = pack8(v);
  }
  cluster.barrier_wait();
}

template <int CH, bool TWO, bool RELU, bool OUT>
__global__ void __launch_bounds__(kHeldThreads, 2)
held_bwd_kernel(const bf16* dy, const bf16* dy2, const uint8_t* mask, const bf16* x, const float* gamma, const float* stats, bf16* __restrict__ dx,
                bf16* __restrict__ gmask_out, float* __restrict__ dgamma, float* __restrict__ dbeta, int R, int C, int most) {
  constexpr int CHUNKS = CH / 8, LANES = kHeldThreads / CHUNKS;
  extern __shared__ uint4 held[];                           // the masked gradient and x: [most][CHUNKS] each
  __shared__ double fold[kHeldWarps][2 * CH], mine[2 * CH];
  __shared__ float affine[2][CH];
  uint4* const held_x = held + most * CHUNKS;
  cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
  const int size = (int)cluster.num_blocks(), rank = (int)cluster.block_rank(), tid = threadIdx.x, chunk = tid % CHUNKS, row = tid / CHUNKS;
  const int c0 = (int)(blockIdx.x / size) * CH, rows = (int)((int64_t)R * (rank + 1) / size - (int64_t)R * rank / size);
  const size_t at = ((int64_t)R * rank / size) * C + c0 + chunk * 8;
  float mu[8], rs[8], s[8] = {0, 0, 0, 0, 0, 0, 0, 0}, q[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  pdl_wait();
#pragma unroll
  for (int i = 0; i < 8; i++) { mu[i] = stats[c0 + chunk * 8 + i]; rs[i] = stats[C + c0 + chunk * 8 + i]; }
#pragma unroll (TWO ? 2 : 4)
  for (int r = row; r < rows; r += LANES) {
    const size_t off = at + (size_t)r * C;
    uint4 gu = *reinterpret_cast<const uint4*>(dy + off);
    const uint4 xu = *reinterpret_cast<const uint4*>(x + off);
    held_x[r * CHUNKS + chunk] = xu;
    float gv[8], xv[8];
    unpack8(gu, gv);
    unpack8(xu, xv);
    if (TWO) {
      float w[8];
      load8(dy2 + off, w);
#pragma unroll
      for (int i = 0; i < 8; i++) gv[i] += w[i];
    }
    if (RELU) {
      const uint32_t bits = mask[off / 8];
#pragma unroll
      for (int i = 0; i < 8; i++) gv[i] = (bits >> i) & 1u ? gv[i] : 0.0f;
    }
    if (TWO || RELU) gu = pack8(gv);
    if (OUT) *reinterpret_cast<uint4*>(gmask_out + off) = gu;
    held[r * CHUNKS + chunk] = gu;
#pragma unroll
    for (int i = 0; i < 8; i++) { s[i] += gv[i]; q[i] += gv[i] * (xv[i] - mu[i]) * rs[i]; }
  }
  double sum, dot;
  cluster_fold<CH>(cluster, s, q, fold, mine, sum, dot);
  if (tid < CH) {
    affine[0][tid] = (float)sum; affine[1][tid] = (float)dot;
    if (rank == 0) { dbeta[c0 + tid] = (float)sum; dgamma[c0 + tid] = (float)dot; }
  }
  cluster.barrier_arrive();
  __syncthreads();
  pdl_trigger();
  float k0[8], k1[8], k2[8];
  const float invR = 1.0f / (float)R;
#pragma unroll
  for (int i = 0; i < 8; i++) {
    k0[i] = gamma[c0 + chunk * 8 + i] * rs[i];
    k1[i] = affine[0][chunk * 8 + i] * invR;
    k2[i] = affine[1][chunk * 8 + i] * invR;
  }
#pragma unroll 4
  for (int r = row; r < rows; r += LANES) {
    float gv[8], xv[8];
    unpack8(held[r * CHUNKS + chunk], gv);
    unpack8(held_x[r * CHUNKS + chunk], xv);
#pragma unroll
    for (int i = 0; i < 8; i++) gv[i] = k0[i] * (gv[i] - k1[i] - (xv[i] - mu[i]) * rs[i] * k2[i]);
    *reinterpret_cast<uint4*>(dx + at + (size_t)r * C) = pack8(gv);
  }
  cluster.barrier_wait();
}

// the form of a sweep for the operands that a call has
inline auto apply_for(const void* residual, const void* mask, int relu) {
  const int form = relu ? (mask ? 2 : 1) : 0;
  if (residual) return form == 2 ? apply_kernel<true, 2> : form == 1 ? apply_kernel<true, 1> : apply_kernel<true, 0>;
  return form == 2 ? apply_kernel<false, 2> : form == 1 ? apply_kernel<false, 1> : apply_kernel<false, 0>;
}
inline auto bwd_reduce_for(const void* dy2, const void* dres, int relu) {
  if (dy2) return relu ? bwd_reduce_kernel<true, true, true> : bwd_reduce_kernel<true, false, true>;
  if (dres) return relu ? bwd_reduce_kernel<false, true, true> : bwd_reduce_kernel<false, false, true>;
  return relu ? bwd_reduce_kernel<false, true, false> : bwd_reduce_kernel<false, false, false>;
}

inline int grid_for(int64_t R, int C) {
  const int rstep = kThreads / (C / 8);
  int64_t g = (R + rstep - 1) / rstep;
  if (g > 148 * kSweepCtas) g = 148 * kSweepCtas;
  return (int)(g < 1 ? 1 : g);
}
// Whether clusters of sixteen CTAs can be scheduled on the device (more than a program may count on).
inline bool wide_clusters() {
  static std::atomic<int> held[64];                         // by device: 0 not asked yet, 1 no, 2 yes
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev >= 64) return false;
  int v = held[dev].load(std::memory_order_relaxed);
  if (!v) {
    const auto kernel = held_bwd_kernel<32, true, true, true>;
    int n = 0;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(16); cfg.blockDim = dim3(kHeldThreads); cfg.dynamicSmemBytes = kHeldBytes;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = 16; attr.val.clusterDim.y = 1; attr.val.clusterDim.z = 1;
    cfg.attrs = &attr; cfg.numAttrs = 1;
    const bool ok = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kHeldBytes) == cudaSuccess &&
                    cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
                    cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) == cudaSuccess && n > 0;
    if (!ok) cudaGetLastError();
    held[dev].store(v = ok ? 2 : 1, std::memory_order_relaxed);
  }
  return v == 2;
}

// How a call that holds `tensors` tensors of R x C is laid out: `ch` channels to a cluster (0: it takes the three launches), `cluster` CTAs, bytes
// per CTA. extra: it reads or writes another tensor besides (a residual, a second gradient, the residual's gradient); relu: it has one.
// All clusters are resident at once, with 64 CTAs at least to fetch for, and small clusters before large ones: sixteen CTAs have to find room in
// one part of the GPU, so of those no more than 128. Shares of 52 KB leave two CTAs on an SM room to work while the other one waits; a forward call
// that writes a mask or reads a residual has less to win, the less the fewer bytes its rows have in a CTA. us, three launches, one;
// inside: forward of 784 x 2048 11.4, 5.9, 3328 x 2048 19.0, 10.3, 13312 x 1024 22.9, 21.7, with ReLU 23.7, 22.9, 26624 x 64 with ReLU 8.2, 7.3, 20480 x 128 9.6, 9.4, with residual
// and ReLU 10976 x 128 8.4, 8.0, 10240 x 256 10.7, 10.0, 9408 x 512 15.3, 14.7, 18000 x 64 7.7, 7.6; backward of 3328 x 2048 24.1, 17.9, with ReLU 25.1, 22.0, 13312 x 256 17.0,
// 15.4, with ReLU 17.4, 17.3, with all operands 10240 x 128 10.8, 10.8, 5120 x 512 17.1, 11.3.
// Outside: forward of 26624 x 128 with ReLU 10.9, 11.4, with residual and ReLU 12544 x 128 8.3, 8.6, x 256 11.9, 12.1, 10240 x 512 15.6, 16.8, 20480 x 64 7.6, 7.9, by clusters of 16
// channels 14000 x 128 8.6, 9.8, 20480 x 128 9.6, 12.0; by more CTAs or larger shares 25088 x 256 16.9, 17.8, x 512 21.4, 27.4, 13312 x 512 backward 22.6, 26.5, with all operands 13312 x 128
// 11.8, 12.7, 9408 x 512 21.6, 22.3. Some calls there would gain: backward of 2205 x 2048 with all operands 22.3, 13.2 with shares of 104 KB, of 8192 x 512 18.9,
// 15.9 with 256 CTAs in clusters of sixteen, of 12544 x 64 with residual 9.0, 7.8, forward of 18816 x 256 14.5, 13.8.
// The backward instances spill up to 156 bytes of their 64 registers, which two CTAs on an SM leave them.
struct HeldPlan { int ch, cluster; size_t bytes; };
inline HeldPlan held_plan(int64_t R, int C, int tensors, bool extra, bool relu) {
  constexpr int KB = 1024;
  if (R > 0x7fffffff) return {0, 0, 0};
  for (const int most : {52 * KB, kHeldBytes}) {
    if (most == kHeldBytes && extra) break;
    for (const int ch : {32, 16}) {
      if (C % ch || (ch == 16 && most == kHeldBytes)) continue;
      for (int cluster = 1; cluster <= (most == kHeldBytes && tensors == 1 ? 8 : 16); cluster *= 2) {
        const int64_t ctas = (int64_t)C / ch * cluster, bytes = (R + cluster - 1) / cluster * ch * 2 * tensors;
        const bool wide_forward = cluster == 16 && tensors == 1;
        const int many = cluster < 16 ? 296 : wide_forward && ch == 16 && extra ? 64 : 128;
        const int limit = ch == 16 && extra ? (tensors == 1 ? 37 * KB : 40 * KB) : wide_forward && extra ? 44 * KB : wide_forward && ch == 16 && relu && ctas > 64 ? 40 * KB : most;
        if (ctas >= 64 && ctas <= many && bytes <= limit && (cluster < 16 || wide_clusters())) return {ch, cluster, (size_t)bytes};
      }
    }
  }
  return {0, 0, 0};
}
template <class... K, class... A> cudaError_t launch_ex(const cudaLaunchConfig_t& cfg, void (*kernel)(K...), A... args) {
  return cudaLaunchKernelEx(&cfg, kernel, static_cast<K>(args)...);
}
template <auto kKernel, class... A>
int launch_held(const HeldPlan& p, int C, cudaStream_t s, A... args) {
  static std::atomic<bool> done[64];                        // by device
  int dev = 0, e = (int)cudaGetDevice(&dev);
  if (!e && (dev >= 64 || !done[dev].load(std::memory_order_relaxed))) {
    e = (int)cudaFuncSetAttribute(kKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kHeldBytes);
    if (!e) e = (int)cudaFuncSetAttribute(kKernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (!e && dev < 64) done[dev].store(true, std::memory_order_relaxed);
  }
  if (e) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(C / p.ch * p.cluster); cfg.blockDim = dim3(kHeldThreads); cfg.dynamicSmemBytes = p.bytes; cfg.stream = s;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = p.cluster; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  static const bool pdl = [] { const char* v = getenv("GCOW_PDL"); return !(v && v[0] == '0'); }();
  cfg.attrs = attr; cfg.numAttrs = pdl ? 2 : 1;
  return (int)launch_ex(cfg, kKernel, args...);
}
template <int CH, class... A> int held_fwd(bool add, int form, const HeldPlan& p, int C, cudaStream_t s, A... args) {   // form: as RELU
  if (add) return form == 2 ? launch_held<held_fwd_kernel<CH, true, 2>>(p, C, s, args...) : form == 1 ? launch_held<held_fwd_kernel<CH, true, 1>>(p, C, s, args...)
                                                                                                  : launch_held<held_fwd_kernel<CH, true, 0>>(p, C, s, args...);
  return form == 2 ? launch_held<held_fwd_kernel<CH, false, 2>>(p, C, s, args...) : form == 1 ? launch_held<held_fwd_kernel<CH, false, 1>>(p, C, s, args...)
                                                                                              : launch_held<held_fwd_kernel<CH, false, 0>>(p, C, s, args...);
}
template <int CH, class... A> int held_bwd(bool two, bool out, bool relu, const HeldPlan& p, int C, cudaStream_t s, A... args) {
  if (two) return relu ? launch_held<held_bwd_kernel<CH, true, true, true>>(p, C, s, args...) : launch_held<held_bwd_kernel<CH, true, false, true>>(p, C, s, args...);
  if (out) return relu ? launch_held<held_bwd_kernel<CH, false, true, true>>(p, C, s, args...) : launch_held<held_bwd_kernel<CH, false, false, true>>(p, C, s, args...);
  return relu ? launch_held<held_bwd_kernel<CH, false, true, false>>(p, C, s, args...) : launch_held<held_bwd_kernel<CH, false, false, false>>(p, C, s, args...);
}
inline bool shape_ok(int C) { return C % 8 == 0 && C >= 8 && C <= 2048 && kThreads % (C / 8) == 0; }

}  // namespace bn
}  // namespace gcow

using namespace gcow::bn;

extern "C" {

int gcow_bn_supported(int C) { return shape_ok(C) ? 1 : 0; }
// Kernels that a training call launches: one (`part` is not used), or two sweeps with the sums' second half between them.
// extra: 1 a residual forward, the residual's gradient backward; 2 a ReLU.
int gcow_bn_launches(int64_t R, int C, int backward, int extra) {
  return shape_ok(C) && held_plan(R, C, backward ? 2 : 1, extra & 1, extra & 2).ch ? 1 : 3;
}
int gcow_bn_parts(int64_t R, int C) { return shape_ok(C) ? grid_for(R, C) : 0; }

// Training forward. part: gcow_bn_parts * 2 * C floats of scratch, or null where gcow_bn_launches says 1 (and mask is at a multiple of 4 bytes). stats: 4*C floats out
// (mean, rstd, scale, shift). run_mean/run_var may be null. mask: R*C/8 bytes out (ReLU
// outcome, one bit per element), required when relu != 0 and a backward pass will follow.
int gcow_bn_fwd_train(const void* x, const void* residual, void* y, void* mask, const float* gamma, const float* beta,
                      float* run_mean, float* run_var, float* stats, float* part, int64_t R, int C, float eps,
                      float momentum, int relu, void* stream) {
  if (!shape_ok(C) || R <= 0) return -1;
  cudaStream_t s = (cudaStream_t)stream;
  const HeldPlan plan = held_plan(R, C, 1, residual != nullptr, relu != 0);
  if (plan.ch && ((uintptr_t)mask & 3) == 0) {
    const int form = relu ? (mask ? 2 : 1) : 0;
    auto run = [&](auto ch) {
      return held_fwd<ch.value>(residual != nullptr, form, plan, C, s, (const bf16*)x, (const bf16*)residual, (bf16*)y, (uint8_t*)mask, gamma, beta, stats,
                                run_mean, run_var, (int)R, C, eps, momentum);
    };
    return plan.ch == 32 ? run(std::integral_constant<int, 32>()) : run(std::integral_constant<int, 16>());
  }
  if (!part) return -1;
  const int g = grid_for(R, C);
  float *mean = stats, *rstd = stats + C, *scale = stats + 2 * C, *shift = stats + 3 * C;
  gcow::launch_dependent(stats_kernel, dim3(g), dim3(kThreads), 0, s, (const bf16*)x, part, R, C);
  gcow::launch_dependent(finalize_fwd_kernel, dim3(C / kFinX), dim3(kFinThreads), 0, s, part, g, C, R, eps, momentum, gamma,
                   beta, mean, rstd, scale, shift, run_mean, run_var);
  gcow::launch_dependent(apply_for(residual, mask, relu), dim3(g), dim3(kThreads), 0, s, (const bf16*)x, (const bf16*)residual, (bf16*)y, (uint8_t*)mask,
                   (const float*)scale, (const float*)shift, R, C);
  return (int)cudaGetLastError();
}

// Inference forward with given statistics; scratch: 2*C floats.
int gcow_bn_fwd_eval(const void* x, const void* residual, void* y, const float* gamma, const float* beta,
                     const float* run_mean, const float* run_var, float* scratch, int64_t R, int C, float eps, int relu,
                     void* stream) {
  if (!shape_ok(C) || R <= 0) return -1;
  cudaStream_t s = (cudaStream_t)stream;
  affine_from_stats_kernel<<<(C + 127) / 128, 128, 0, s>>>(gamma, beta, run_mean, run_var, eps, C, scratch, scratch + C);
  const auto kernel = residual || relu ? apply_for(residual, nullptr, relu) : apply_kernel<false, 0, 4>;
  kernel<<<grid_for(R, C), kThreads, 0, s>>>((const bf16*)x, (const bf16*)residual, (bf16*)y, nullptr, scratch, scratch + C, R, C);
  return (int)cudaGetLastError();
}

// Backward. stats and mask as written by the forward. dres (nullable) receives the gradient
// of the residual input (the ReLU-masked dy). dgb: 2*C floats out (dgamma, dbeta).
// dy2 (nullable): a second gradient of the same output, added to dy on the fly; it needs dres (any buffer of the
// tensor's size) to carry the masked sum to the second sweep.
// dgamma and dbeta (C floats each) may lie anywhere, e.g. in the two parameters' gradient tensors.
int gcow_bn_bwd3(const void* dy, const void* dy2, const void* mask, const void* x, const float* gamma, const float* stats,
                 void* dx, void* dres, float* dgamma, float* dbeta, float* part, int64_t R, int C, int relu, void* stream) {
  if (!shape_ok(C) || R <= 0 || (dy2 && !dres)) return -1;
  cudaStream_t s = (cudaStream_t)stream;
  const HeldPlan plan = held_plan(R, C, 2, dres != nullptr, relu != 0);
  if (plan.ch) {
    auto run = [&](auto ch) {
      return held_bwd<ch.value>(dy2 != nullptr, dres != nullptr, relu != 0, plan, C, s, (const bf16*)dy, (const bf16*)dy2, (const uint8_t*)mask, (const bf16*)x,
                                gamma, stats, (bf16*)dx, (bf16*)dres, dgamma, dbeta, (int)R, C, (int)((R + plan.cluster - 1) / plan.cluster));
    };
    return plan.ch == 32 ? run(std::integral_constant<int, 32>()) : run(std::integral_constant<int, 16>());
  }
  if (!part) return -1;
  const int g = grid_for(R, C);
  const float *mean = stats, *rstd = stats + C;
  gcow::launch_dependent(bwd_reduce_for(dy2, dres, relu), dim3(g), dim3(kThreads), 0, s, (const bf16*)dy, (const bf16*)dy2, (const uint8_t*)mask,
                         (const bf16*)x, mean, rstd, (bf16*)dres, part, R, C);
  gcow::launch_dependent(finalize_bwd_kernel, dim3(C / kFinX), dim3(kFinThreads), 0, s, (const float*)part, g, C, dgamma, dbeta);
  // the second sweep applies the mask again, or reads the masked gradient if it was written
  gcow::launch_dependent(!dres && relu ? bwd_dx_kernel<true> : bwd_dx_kernel<false>, dim3(g), dim3(kThreads), 0, s, (const bf16*)(dres ? dres : dy), (const uint8_t*)mask, (const bf16*)x,
                   gamma, mean, rstd, (const float*)dgamma, (const float*)dbeta, (bf16*)dx, R, C);
  return (int)cudaGetLastError();
}

int gcow_bn_bwd2(const void* dy, const void* dy2, const void* mask, const void* x, const float* gamma, const float* stats,
                 void* dx, void* dres, float* dgb, float* part, int64_t R, int C, int relu, void* stream) {
  return gcow_bn_bwd3(dy, dy2, mask, x, gamma, stats, dx, dres, dgb, dgb + C, part, R, C, relu, stream);
}

int gcow_bn_bwd(const void* dy, const void* mask, const void* x, const float* gamma, const float* stats, void* dx,
                void* dres, float* dgb, float* part, int64_t R, int C, int relu, void* stream) {
  return gcow_bn_bwd2(dy, nullptr, mask, x, gamma, stats, dx, dres, dgb, part, R, C, relu, stream);
}

}  // extern "C"
