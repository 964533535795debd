// Fused multi-head self-attention on the 5th-generation tensor cores (sm_100a), head dimension 64,
// sequence length a multiple of 128 up to 512, no mask, no dropout: forward and backward.
//
// All three kernels read the packed projection qkv [B][S][3][H][64] (bf16) in place through 4-D
// tensor maps {d, h, s, b} - a box is 128 sequence positions of one head, 128-byte rows with the
// 128-byte swizzle - and write the context / gradients in the layouts the neighbouring GEMMs use
// ([B][S][H][64] and [B][S][3][H][64]), so no transposed copy of Q, K or V exists.
//
//  forward   one CTA per (128 queries, head): S = Q K^T for ALL keys lands in tensor memory (up to
//            512 fp32 columns, one row per thread), the row maximum and the exponentials are taken
//            straight from there, P goes to shared memory as bf16 in the MMA's K-major layout and
//            O = P V accumulates in the tensor-memory columns that S has vacated. exp(S - max)
//            needs no running rescale because the whole row is present. Also stores the row's
//            log2-sum-exp for the backward pass.
//  backward  recomputes P from Q, K and the stored log-sum-exp, a 128 x 64 tile at a time (128 x 128 where the grid leaves
//            each CTA an SM to itself).
//     dK/dV  one CTA per (128 keys, head), loop over blocks of 64 queries: S^T = K Q^T and dP^T = V dO^T in
//            tensor memory (one key per row, so lse and delta are per column, read from shared memory), P^T and
//            dS^T = P^T (dP^T - delta) to shared memory as K-major operands, dV and dK accumulate in tensor memory.
//     dQ     one CTA per (128 queries, head), loop over blocks of 64 keys: S, dP, dS, then dQ += dS K.
//            Recomputing S and dP here instead of adding dQ with atomics keeps the gradients deterministic.
//            The steps of one tile (products, exponentials, operands, products) follow one another, so what hides them
//            is a second CTA on the SM: tiles of 64 keep a CTA within 256 tensor-memory columns and 113 KB of shared
//            memory, where 128 x 128 tiles took 320 to 384 columns and 128 to 160 KB, one CTA per SM.
//            512 x 32 sequences of 16 heads, both kernels and delta: 398 -> 337 us (dK/dV 206 -> 192, dQ 169 -> 133).
//  delta = rowsum(dO * O) comes from a small elementwise kernel.
//
// 512 threads per CTA: four threads share an accumulator row (the four warps that may read a
// tensor-memory lane quarter each take a quarter of the columns), which is what hides the latency
// of the exponentials; thread 0 issues the TMA loads and the MMAs. Every mbarrier wait is bounded: after a fixed number of polls the CTA records an error
// code, leaves its loops, waits (bounded) for outstanding MMAs, frees its tensor memory and
// returns. No load uses cluster multicast. The reference's models are CNNs
// (hw/models/train_imagenet.py:199-202); this kernel serves the BERT configuration.
#include <stdio.h>
#include <mutex>

#include "tc_common.cuh"

namespace gcow {
namespace attn {

using namespace gcow::tc;

constexpr int D = 64;                 // head dimension: one 128-byte row
constexpr int TILE = 128;             // rows of a query / key tile
constexpr int TILE_BYTES = TILE * D * 2;   // 16 KB
constexpr int MAX_S = 512;
constexpr int NT = 512;               // threads per CTA: 4 column groups x 128 rows
// Backward, by the queries / keys per loop step (64 or 128): bytes of a block of them, tensor-memory columns (S and dP of a
// step, two accumulators), CTAs per SM.
template <int STEP> struct Step {
  static constexpr int BYTES = STEP * D * 2, COLS = STEP == 64 ? 256 : 512, CTAS = STEP == 64 ? 2 : 1;
  static constexpr int PANELS = STEP / 64;   // of P and dS: [128 rows][64 columns], 16 KB each
};

struct Params {
  __nv_bfloat16* out;      // forward: context [B][S][H][64]
  float* lse;              // [B][H][S] log2-sum-exp of the scaled scores
  const float* delta;      // backward: [B][H][S] rowsum(dO * O)
  __nv_bfloat16* dqkv;     // backward: [B][S][3][H][64]
  int B, S, H;
  float scale_log2;        // softmax scale * log2(e)
  float scale;             // softmax scale
  uint32_t* error;
};

struct Bars {
  uint64_t a, b, c, d, e[2], f[2], drain;
  uint32_t tmem_base;
  volatile uint32_t abort;
  float red[4][TILE];      // per-row partial maxima / sums of the four column groups
};

__device__ __forceinline__ uint32_t idesc_f16(int n, bool a_mn, bool b_mn) {
  // fp32 accumulate, bf16 x bf16, operand major-ness, N, M = 128
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)a_mn << 15) | ((uint32_t)b_mn << 16) |
         ((uint32_t)(n >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
}
__device__ __forceinline__ void proxy_fence() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ bool wait(Bars* bs, uint64_t* bar, uint32_t parity, uint32_t* error, uint32_t code) {
  return mbar_wait_abortable(&bs->abort, bar, parity, error, code);
}
__device__ __forceinline__ uint32_t pack2(float a, float b) {
  __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&v);
}
// Byte offset of the 16-byte chunk holding elements 8j..8j+7 of row r in a [rows][64] bf16 tile with
// 128-byte rows and the 128-byte swizzle (the layout TMA writes and the K-major descriptor reads).
__device__ __forceinline__ uint32_t sw128(int r, int j) { return (uint32_t)(r * 128 + ((j ^ (r & 7)) << 4)); }

// Store 32 consecutive fp32 values of this thread's row as bf16 into a K-major operand: the row has `64`
// elements per 16 KB block, the 32 values are elements e0..e0+31 of the row (e0 a multiple of 32).
__device__ __forceinline__ void store_kmajor32(uint8_t* tile, int row, int e0, const float (&v)[32]) {
  uint8_t* blk = tile + (e0 >> 6) * TILE_BYTES;
  const int j0 = (e0 & 63) >> 3;
#pragma unroll
  for (int j = 0; j < 4; j++) {
    uint4 o = make_uint4(pack2(v[8 * j], v[8 * j + 1]), pack2(v[8 * j + 2], v[8 * j + 3]),
                         pack2(v[8 * j + 4], v[8 * j + 5]), pack2(v[8 * j + 6], v[8 * j + 7]));
    *reinterpret_cast<uint4*>(blk + sw128(row, j0 + j)) = o;
  }
}
// 16 values, elements e0..e0+15 of the row, of an operand with 64 elements per row.
__device__ __forceinline__ void store_kmajor16(uint8_t* tile, int row, int e0, const float (&v)[16]) {
#pragma unroll
  for (int j = 0; j < 2; j++) {
    uint4 o = make_uint4(pack2(v[8 * j], v[8 * j + 1]), pack2(v[8 * j + 2], v[8 * j + 3]),
                         pack2(v[8 * j + 4], v[8 * j + 5]), pack2(v[8 * j + 6], v[8 * j + 7]));
    *reinterpret_cast<uint4*>(tile + sw128(row, (e0 >> 3) + j)) = o;
  }
}

template <uint32_t COLS>
__device__ __forceinline__ void tmem_alloc(Bars* bs, int warp) {
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&bs->tmem_base)), "r"(COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
}
template <uint32_t COLS>
__device__ __forceinline__ void tmem_free(uint32_t base, int warp) {
  if (warp == 0) {
    __syncwarp();
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(base), "r"(COLS) : "memory");
  }
}
// All MMAs issued by this thread have completed (bounded), so tensor memory and the operands may go.
__device__ __forceinline__ void drain(Bars* bs) {
  tc_commit(&bs->drain);
  for (uint32_t it = 0; it < kSpinLimit; it++) if (mbar_try_wait(&bs->drain, 0)) break;
}

// A [128 x 64k] K-major (rows x reduction) times B: 4 k-steps per 64 reduction elements.
__device__ __forceinline__ void mma_kk(uint32_t d_tmem, uint32_t a_smem, uint32_t b_smem, int n, bool acc) {
  const uint32_t id = idesc_f16(n, false, false);
  const uint64_t da = smem_desc_sw128(a_smem), db = smem_desc_sw128(b_smem);
#pragma unroll
  for (int k = 0; k < 4; k++) tc_mma(d_tmem, da + 2 * k, db + 2 * k, id, acc || k);
}

// ------------------------------------------------------------------------------ forward
__global__ void __launch_bounds__(NT, 1)
attn_fwd_kernel(const __grid_constant__ CUtensorMap tq, const __grid_constant__ CUtensorMap tk,
                const __grid_constant__ CUtensorMap tv, const Params p) {
  extern __shared__ uint8_t raw[];
  uint8_t* base = reinterpret_cast<uint8_t*>(((uintptr_t)raw + 1023) & ~(uintptr_t)1023);
  uint8_t* sQ = base;                       // 16 KB
  uint8_t* sK = sQ + TILE_BYTES;            // S/128 tiles; P of the first 256 keys overwrites it
  uint8_t* sV = sK + 4 * TILE_BYTES;
  uint8_t* sP1 = sV + 4 * TILE_BYTES;       // P of keys 256..511
  Bars* bs = reinterpret_cast<Bars*>(sP1 + 4 * TILE_BYTES);
  const int tid = threadIdx.x, warp = tid >> 5;
  const int row = (warp & 3) * 32 + (tid & 31), cg = warp >> 2;      // accumulator row, column group 0..3
  const int q0 = blockIdx.x * TILE, h = blockIdx.y, b = blockIdx.z;
  const int nk = p.S, ntile = nk / TILE;
  const int half0 = nk < 256 ? nk : 256, half1 = nk - half0;

  if (tid == 0) {
    mbar_init(&bs->a, 1); mbar_init(&bs->b, 1); mbar_init(&bs->c, 1); mbar_init(&bs->d, 1); mbar_init(&bs->drain, 1);
    bs->abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  tmem_alloc<512>(bs, warp);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = bs->tmem_base;
  const uint32_t lane_addr = tmem + ((uint32_t)((warp & 3) * 32) << 16);
  bool ok = true;

  if (tid == 0) {
    mbar_expect_tx(&bs->a, TILE_BYTES + nk * 128);
    tma_load_4d(smem_u32(sQ), &tq, smem_u32(&bs->a), 0, h, q0, b);
    for (int t = 0; t < ntile; t++) tma_load_4d(smem_u32(sK + t * TILE_BYTES), &tk, smem_u32(&bs->a), 0, h, t * TILE, b);
    mbar_expect_tx(&bs->b, nk * 128);
    for (int t = 0; t < ntile; t++) tma_load_4d(smem_u32(sV + t * TILE_BYTES), &tv, smem_u32(&bs->b), 0, h, t * TILE, b);
    ok = wait(bs, &bs->a, 0, p.error, 21);
    if (ok) {
      tc_fence_after();
      mma_kk(tmem, smem_u32(sQ), smem_u32(sK), half0, false);                       // S[:, 0:half0]
      if (half1) mma_kk(tmem + 256, smem_u32(sQ), smem_u32(sK + 2 * TILE_BYTES), half1, false);
      tc_commit(&bs->c);
    }
  }
  ok = wait(bs, &bs->c, 0, p.error, 22);
  ok = __syncthreads_and(ok);
  if (ok) {
    tc_fence_after();
    // pass 1: row maximum over every key; this thread scans its quarter of the columns
    float m = -INFINITY;
    {
      // tensor-memory loads two chunks ahead of the arithmetic
      const int c0 = cg * (nk / 128), c1 = (cg + 1) * (nk / 128);
      uint32_t ra[32], rb[32];
      tc_ld32(lane_addr + c0 * 32, ra);
      for (int c = c0; c < c1; c += 2) {
        tc_wait_ld();
        if (c + 1 < c1) tc_ld32(lane_addr + (c + 1) * 32, rb);
#pragma unroll
        for (int j = 0; j < 32; j++) m = fmaxf(m, __uint_as_float(ra[j]));
        if (c + 1 < c1) {
          tc_wait_ld();
          if (c + 2 < c1) tc_ld32(lane_addr + (c + 2) * 32, ra);
#pragma unroll
          for (int j = 0; j < 32; j++) m = fmaxf(m, __uint_as_float(rb[j]));
        }
      }
    }
    bs->red[cg][row] = m;
    __syncthreads();
    m = fmaxf(fmaxf(bs->red[0][row], bs->red[1][row]), fmaxf(bs->red[2][row], bs->red[3][row]));
    __syncthreads();                        // red is reused for the row sums below
    const float ms = m * p.scale_log2;
    float l = 0.0f;
    // pass 2: exponentials, row sum, P as bf16 in the A-operand layout; then O += P V for that half
    for (int hf = 0; hf < 2; hf++) {      // same trip count for every thread: the loop body holds barriers
      const int keys = hf ? half1 : half0;
      if (!keys) break;
      uint8_t* sP = hf ? sP1 : sK;
      {
        // this thread's one or two chunks of the half: both loads are issued before the first is used
        const int c0 = cg * (keys / 128), two = keys / 128 == 2;
        uint32_t ra[32], rb[32];
        tc_ld32(lane_addr + hf * 256 + c0 * 32, ra);
        if (two) tc_ld32(lane_addr + hf * 256 + (c0 + 1) * 32, rb);
        tc_wait_ld();
        float v[32];
#pragma unroll
        for (int j = 0; j < 32; j++) {
          v[j] = ex2_ftz(fmaf(__uint_as_float(ra[j]), p.scale_log2, -ms));
          l += v[j];
        }
        store_kmajor32(sP, row, c0 * 32, v);
        if (two) {
#pragma unroll
          for (int j = 0; j < 32; j++) {
            v[j] = ex2_ftz(fmaf(__uint_as_float(rb[j]), p.scale_log2, -ms));
            l += v[j];
          }
          store_kmajor32(sP, row, (c0 + 1) * 32, v);
        }
      }
      proxy_fence();
      tc_fence_before();
      __syncthreads();
      if (tid == 0) {
        if (hf == 0 && ok) ok = wait(bs, &bs->b, 0, p.error, 23);
        if (ok) {
          tc_fence_after();
          const uint32_t id = idesc_f16(D, false, true);
          for (int blk = 0; blk < keys / 64; blk++) {
            const uint64_t da = smem_desc_sw128(smem_u32(sP + blk * TILE_BYTES));
            const uint64_t db = smem_desc_mn_sw128(smem_u32(sV + (hf * 256 + blk * 64) * 128));
#pragma unroll
            for (int k = 0; k < 4; k++) tc_mma(tmem, da + 2 * k, db + (2048 >> 4) * k, id, (hf | blk | k) != 0);
          }
          if (hf == 1 || !half1) tc_commit(&bs->d);
        }
      }
    }
    bs->red[cg][row] = l;
    ok = ok && wait(bs, &bs->d, 0, p.error, 24);
    ok = __syncthreads_and(ok);
    if (ok) {
      tc_fence_after();
      l = (bs->red[0][row] + bs->red[1][row]) + (bs->red[2][row] + bs->red[3][row]);
      const float inv = 1.0f / l;
      const size_t orow = (((size_t)b * p.S + q0 + row) * p.H + h) * D;
      if (cg < 2) {                          // 64 output columns: column groups 0 and 1 take 32 each
        const int c = cg;
        uint32_t r[32];
        tc_ld32(lane_addr + c * 32, r);
        tc_wait_ld();
#pragma unroll
        for (int j = 0; j < 4; j++) {
          uint4 o = make_uint4(pack2(__uint_as_float(r[8 * j]) * inv, __uint_as_float(r[8 * j + 1]) * inv),
                               pack2(__uint_as_float(r[8 * j + 2]) * inv, __uint_as_float(r[8 * j + 3]) * inv),
                               pack2(__uint_as_float(r[8 * j + 4]) * inv, __uint_as_float(r[8 * j + 5]) * inv),
                               pack2(__uint_as_float(r[8 * j + 6]) * inv, __uint_as_float(r[8 * j + 7]) * inv));
          *reinterpret_cast<uint4*>(p.out + orow + c * 32 + j * 8) = o;
        }
      }
      if (cg == 0) p.lse[((size_t)b * p.H + h) * p.S + q0 + row] = ms + log2f(l);
    }
  }
  if (tid == 0) drain(bs);
  tc_fence_before();
  __syncthreads();
  tmem_free<512>(tmem, warp);
}

// delta[b][h][s] = sum_d dO[b][s][h][d] * O[b][s][h][d]; eight lanes per row, so that a warp reads whole lines (262 144
// rows: 15 us, one thread per row took 24).
__global__ void attn_delta_kernel(const __nv_bfloat16* __restrict__ o, const __nv_bfloat16* __restrict__ go,
                                  float* __restrict__ delta, int B, int S, int H) {
  const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  const size_t i = t >> 3, rows = (size_t)B * S * H;                   // over b, s, h
  const int part = (int)(t & 7);
  float acc = 0.0f;
  if (i < rows) {
    const uint4 x = reinterpret_cast<const uint4*>(o + i * D)[part], y = reinterpret_cast<const uint4*>(go + i * D)[part];
    const __nv_bfloat162* xb = reinterpret_cast<const __nv_bfloat162*>(&x);
    const __nv_bfloat162* yb = reinterpret_cast<const __nv_bfloat162*>(&y);
#pragma unroll
    for (int e = 0; e < 4; e++) {
      const float2 a = __bfloat1622float2(xb[e]), c = __bfloat1622float2(yb[e]);
      acc = fmaf(a.x, c.x, fmaf(a.y, c.y, acc));
    }
  }
#pragma unroll
  for (int d = 1; d < 8; d <<= 1) acc += __shfl_xor_sync(0xffffffffu, acc, d);
  if (i < rows && part == 0) {
    const int h = (int)(i % H);
    const size_t bs = i / H;
    delta[((bs / S) * H + h) * S + bs % S] = acc;
  }
}

__device__ __forceinline__ void tc_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr) : "memory");
}

// P and dS of one 128 x STEP tile from S (tensor-memory columns 0..STEP-1) and dP (the STEP columns behind), this thread's row
// and 16-column group c of each 64-column panel, as K-major operands. COLS: lse and delta belong to the columns (nlse / ndelta: their negatives for
// this tile's columns in shared memory) and P is written too; else they are the row's (nlse[0], ndelta[0]).
template <bool COLS, int STEP>
__device__ __forceinline__ void softmax_grad_tile(uint32_t lane_addr, int row, int c, const float* nlse, const float* ndelta,
                                                  const Params& p, uint8_t* sP, uint8_t* sdS) {
  const uint64_t sl = tc::pack2(p.scale_log2, p.scale_log2), sc = tc::pack2(p.scale, p.scale), one = tc::pack2(1.0f, 1.0f);
#pragma unroll
  for (int h = 0; h < Step<STEP>::PANELS; h++) {
    const int col = h * 64 + c * 16;
    uint32_t rs[16], rd[16];
    tc_ld16(lane_addr + col, rs);
    tc_ld16(lane_addr + STEP + col, rd);
    tc_wait_ld();
    float pv[16], ds[16];
#pragma unroll
    for (int j = 0; j < 16; j += 2) {
      const uint64_t nl = COLS ? *reinterpret_cast<const uint64_t*>(nlse + col + j) : tc::pack2(nlse[0], nlse[0]);
      const uint64_t nd = COLS ? *reinterpret_cast<const uint64_t*>(ndelta + col + j) : tc::pack2(ndelta[0], ndelta[0]);
      float a, b;
      unpack2(fma2(tc::pack2(__uint_as_float(rs[j]), __uint_as_float(rs[j + 1])), sl, nl), a, b);
      pv[j] = ex2_ftz(a);
      pv[j + 1] = ex2_ftz(b);
      const uint64_t d = fma2(tc::pack2(__uint_as_float(rd[j]), __uint_as_float(rd[j + 1])), one, nd);
      unpack2(mul2(mul2(tc::pack2(pv[j], pv[j + 1]), d), sc), ds[j], ds[j + 1]);
    }
    if (COLS) store_kmajor16(sP + h * TILE_BYTES, row, c * 16, pv);
    store_kmajor16(sdS + h * TILE_BYTES, row, c * 16, ds);
  }
}

// Write this thread's row of a 64-column fp32 accumulator (tensor-memory column `col`) as bf16 to `dst`.
__device__ __forceinline__ void store_acc_row(uint32_t lane_addr, int col, int c, __nv_bfloat16* dst) {
  {                                          // chunk c (0 or 1) of the 64 columns
    uint32_t r[32];
    tc_ld32(lane_addr + col + c * 32, r);
    tc_wait_ld();
#pragma unroll
    for (int j = 0; j < 4; j++) {
      uint4 o = make_uint4(pack2(__uint_as_float(r[8 * j]), __uint_as_float(r[8 * j + 1])),
                           pack2(__uint_as_float(r[8 * j + 2]), __uint_as_float(r[8 * j + 3])),
                           pack2(__uint_as_float(r[8 * j + 4]), __uint_as_float(r[8 * j + 5])),
                           pack2(__uint_as_float(r[8 * j + 6]), __uint_as_float(r[8 * j + 7])));
      *reinterpret_cast<uint4*>(dst + c * 32 + j * 8) = o;
    }
  }
}

// ------------------------------------------------------------------- backward: dK and dV
template <int STEP>
__global__ void __launch_bounds__(NT, Step<STEP>::CTAS)
attn_bwd_dkdv_kernel(const __grid_constant__ CUtensorMap tq, const __grid_constant__ CUtensorMap tk,
                     const __grid_constant__ CUtensorMap tv, const __grid_constant__ CUtensorMap tdo, const Params p) {
  constexpr int STEP_BYTES = Step<STEP>::BYTES, PANELS = Step<STEP>::PANELS;
  extern __shared__ uint8_t raw[];
  uint8_t* base = reinterpret_cast<uint8_t*>(((uintptr_t)raw + 1023) & ~(uintptr_t)1023);
  uint8_t* sK = base;                        // 16 KB each
  uint8_t* sV = sK + TILE_BYTES;
  uint8_t* sP = sV + TILE_BYTES;             // P^T, dS^T: panels of [128 keys][64 queries]
  uint8_t* sdS = sP + PANELS * TILE_BYTES;
  uint8_t* sQ = sdS + PANELS * TILE_BYTES;   // two buffers each
  uint8_t* sdO = sQ + 2 * STEP_BYTES;
  float* nlse = reinterpret_cast<float*>(sdO + 2 * STEP_BYTES);      // -lse and -delta of every query
  float* ndelta = nlse + MAX_S;
  Bars* bs = reinterpret_cast<Bars*>(ndelta + MAX_S);
  const int tid = threadIdx.x, warp = tid >> 5;
  const int row = (warp & 3) * 32 + (tid & 31), cg = warp >> 2;
  const int k0 = blockIdx.x * TILE, h = blockIdx.y, b = blockIdx.z;
  const int nq = p.S / STEP;

  if (tid == 0) {
    mbar_init(&bs->a, 1); mbar_init(&bs->c, 1); mbar_init(&bs->d, 1); mbar_init(&bs->drain, 1);
    mbar_init(&bs->e[0], 1); mbar_init(&bs->e[1], 1);
    bs->abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  static_assert(MAX_S <= NT, "one query's statistics per thread");
  if (tid < p.S) {
    const size_t stat = ((size_t)b * p.H + h) * p.S + tid;
    nlse[tid] = -p.lse[stat];
    ndelta[tid] = -p.delta[stat];
  }
  tmem_alloc<Step<STEP>::COLS>(bs, warp);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = bs->tmem_base;
  const uint32_t lane_addr = tmem + ((uint32_t)((warp & 3) * 32) << 16);
  constexpr uint32_t COL_S = 0, COL_DV = 2 * STEP, COL_DK = COL_DV + D;      // dP^T sits at COL_S + STEP
  bool ok = true;

  if (tid == 0) {
    mbar_expect_tx(&bs->a, 2 * TILE_BYTES);
    tma_load_4d(smem_u32(sK), &tk, smem_u32(&bs->a), 0, h, k0, b);
    tma_load_4d(smem_u32(sV), &tv, smem_u32(&bs->a), 0, h, k0, b);
    mbar_expect_tx(&bs->e[0], 2 * STEP_BYTES);
    tma_load_4d(smem_u32(sQ), &tq, smem_u32(&bs->e[0]), 0, h, 0, b);
    tma_load_4d(smem_u32(sdO), &tdo, smem_u32(&bs->e[0]), 0, h, 0, b);
    ok = wait(bs, &bs->a, 0, p.error, 31);
  }
  for (int i = 0; i < nq; i++) {
    const int buf = i & 1;
    uint8_t* q = sQ + buf * STEP_BYTES;
    uint8_t* go = sdO + buf * STEP_BYTES;
    if (tid == 0 && ok) {
      // S and dP of this step right behind the products of the last one, whose end nothing here waits for
      ok = wait(bs, &bs->e[buf], (i >> 1) & 1, p.error, 33);
      if (ok) {
        tc_fence_after();
        mma_kk(tmem + COL_S, smem_u32(sK), smem_u32(q), STEP, false);            // S^T  = K_j Q_i^T
        mma_kk(tmem + COL_S + STEP, smem_u32(sV), smem_u32(go), STEP, false);    // dP^T = V_j dO_i^T
        tc_commit(&bs->c);
      }
      // the other buffer was last read by the MMAs of step i-1; once they are done, block i+1 is fetched into it
      if (ok && i + 1 < nq) {
        if (i >= 1) ok = wait(bs, &bs->d, (i - 1) & 1, p.error, 32);
        if (ok) {
          mbar_expect_tx(&bs->e[buf ^ 1], 2 * STEP_BYTES);
          tma_load_4d(smem_u32(sQ + (buf ^ 1) * STEP_BYTES), &tq, smem_u32(&bs->e[buf ^ 1]), 0, h, (i + 1) * STEP, b);
          tma_load_4d(smem_u32(sdO + (buf ^ 1) * STEP_BYTES), &tdo, smem_u32(&bs->e[buf ^ 1]), 0, h, (i + 1) * STEP, b);
        }
      }
    }
    ok = ok && wait(bs, &bs->c, i & 1, p.error, 34);
    // P / dS of iteration i-1 must have been consumed by its MMAs before they are overwritten
    if (i >= 1) ok = ok && wait(bs, &bs->d, (i - 1) & 1, p.error, 35);
    ok = __syncthreads_and(ok);
    if (!ok) break;
    tc_fence_after();
    softmax_grad_tile<true, STEP>(lane_addr + COL_S, row, cg, nlse + i * STEP, ndelta + i * STEP, p, sP, sdS);
    proxy_fence();
    tc_fence_before();
    __syncthreads();
    if (tid == 0) {
      tc_fence_after();
      const uint32_t id = idesc_f16(D, false, true);                // A = P^T / dS^T (K-major), B = dO / Q as [q][d]
#pragma unroll
      for (int h = 0; h < PANELS; h++) {
        const uint64_t dap = smem_desc_sw128(smem_u32(sP + h * TILE_BYTES)), dad = smem_desc_sw128(smem_u32(sdS + h * TILE_BYTES));
        const uint64_t dbo = smem_desc_mn_sw128(smem_u32(go + h * 8192)), dbq = smem_desc_mn_sw128(smem_u32(q + h * 8192));
#pragma unroll
        for (int k = 0; k < 4; k++) {
          tc_mma(tmem + COL_DV, dap + 2 * k, dbo + (2048 >> 4) * k, id, (i | h | k) != 0);
          tc_mma(tmem + COL_DK, dad + 2 * k, dbq + (2048 >> 4) * k, id, (i | h | k) != 0);
        }
      }
      tc_commit(&bs->d);
    }
  }
  ok = ok && wait(bs, &bs->d, (nq - 1) & 1, p.error, 36);
  ok = __syncthreads_and(ok);
  if (ok) {
    tc_fence_after();
    const size_t orow = ((((size_t)b * p.S + k0 + row) * 3) * p.H + h) * D;     // [b][s][which][h][d], which = 0
    // column groups 0, 1: the two halves of dK's row; 2, 3: of dV's row
    store_acc_row(lane_addr, cg < 2 ? COL_DK : COL_DV, cg & 1, p.dqkv + orow + (size_t)(cg < 2 ? 1 : 2) * p.H * D);
  }
  if (tid == 0) drain(bs);
  tc_fence_before();
  __syncthreads();
  tmem_free<Step<STEP>::COLS>(tmem, warp);
}

// ------------------------------------------------------------------------ backward: dQ
template <int STEP>
__global__ void __launch_bounds__(NT, Step<STEP>::CTAS)
attn_bwd_dq_kernel(const __grid_constant__ CUtensorMap tq, const __grid_constant__ CUtensorMap tk,
                   const __grid_constant__ CUtensorMap tv, const __grid_constant__ CUtensorMap tdo, const Params p) {
  constexpr int STEP_BYTES = Step<STEP>::BYTES, PANELS = Step<STEP>::PANELS;
  extern __shared__ uint8_t raw[];
  uint8_t* base = reinterpret_cast<uint8_t*>(((uintptr_t)raw + 1023) & ~(uintptr_t)1023);
  uint8_t* sQ = base;
  uint8_t* sdO = sQ + TILE_BYTES;
  uint8_t* sdS = sdO + TILE_BYTES;           // panels of [128 queries][64 keys]
  uint8_t* sK = sdS + PANELS * TILE_BYTES;   // two buffers each
  uint8_t* sV = sK + 2 * STEP_BYTES;
  Bars* bs = reinterpret_cast<Bars*>(sV + 2 * STEP_BYTES);
  const int tid = threadIdx.x, warp = tid >> 5;
  const int row = (warp & 3) * 32 + (tid & 31), cg = warp >> 2;
  const int q0 = blockIdx.x * TILE, h = blockIdx.y, b = blockIdx.z;
  const int nkv = p.S / STEP;

  if (tid == 0) {
    mbar_init(&bs->a, 1); mbar_init(&bs->c, 1); mbar_init(&bs->d, 1); mbar_init(&bs->drain, 1);
    mbar_init(&bs->e[0], 1); mbar_init(&bs->e[1], 1);
    bs->abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  tmem_alloc<Step<STEP>::COLS>(bs, warp);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = bs->tmem_base;
  const uint32_t lane_addr = tmem + ((uint32_t)((warp & 3) * 32) << 16);
  constexpr uint32_t COL_S = 0, COL_DQ = 2 * STEP;
  bool ok = true;
  const size_t stat = ((size_t)b * p.H + h) * p.S + q0 + row;
  const float nlse = -p.lse[stat], ndelta = -p.delta[stat];

  if (tid == 0) {
    mbar_expect_tx(&bs->a, 2 * TILE_BYTES);
    tma_load_4d(smem_u32(sQ), &tq, smem_u32(&bs->a), 0, h, q0, b);
    tma_load_4d(smem_u32(sdO), &tdo, smem_u32(&bs->a), 0, h, q0, b);
    mbar_expect_tx(&bs->e[0], 2 * STEP_BYTES);
    tma_load_4d(smem_u32(sK), &tk, smem_u32(&bs->e[0]), 0, h, 0, b);
    tma_load_4d(smem_u32(sV), &tv, smem_u32(&bs->e[0]), 0, h, 0, b);
    ok = wait(bs, &bs->a, 0, p.error, 41);
  }
  for (int j = 0; j < nkv; j++) {
    const int buf = j & 1;
    uint8_t* kt = sK + buf * STEP_BYTES;
    uint8_t* vt = sV + buf * STEP_BYTES;
    if (tid == 0 && ok) {
      ok = wait(bs, &bs->e[buf], (j >> 1) & 1, p.error, 43);                     // the order of the steps: as above
      if (ok) {
        tc_fence_after();
        mma_kk(tmem + COL_S, smem_u32(sQ), smem_u32(kt), STEP, false);           // S  = Q_i K_j^T
        mma_kk(tmem + COL_S + STEP, smem_u32(sdO), smem_u32(vt), STEP, false);   // dP = dO_i V_j^T
        tc_commit(&bs->c);
      }
      if (ok && j + 1 < nkv) {
        if (j >= 1) ok = wait(bs, &bs->d, (j - 1) & 1, p.error, 42);             // K of block j-1 is still read by its dQ MMAs
        if (ok) {
          mbar_expect_tx(&bs->e[buf ^ 1], 2 * STEP_BYTES);
          tma_load_4d(smem_u32(sK + (buf ^ 1) * STEP_BYTES), &tk, smem_u32(&bs->e[buf ^ 1]), 0, h, (j + 1) * STEP, b);
          tma_load_4d(smem_u32(sV + (buf ^ 1) * STEP_BYTES), &tv, smem_u32(&bs->e[buf ^ 1]), 0, h, (j + 1) * STEP, b);
        }
      }
    }
    ok = ok && wait(bs, &bs->c, j & 1, p.error, 44);
    if (j >= 1) ok = ok && wait(bs, &bs->d, (j - 1) & 1, p.error, 45);           // dS of tile j-1 consumed
    ok = __syncthreads_and(ok);
    if (!ok) break;
    tc_fence_after();
    softmax_grad_tile<false, STEP>(lane_addr + COL_S, row, cg, &nlse, &ndelta, p, nullptr, sdS);
    proxy_fence();
    tc_fence_before();
    __syncthreads();
    if (tid == 0) {
      tc_fence_after();
      const uint32_t id = idesc_f16(D, false, true);                // A = dS (K-major), B = K_j as [key][d] (MN-major)
#pragma unroll
      for (int h = 0; h < PANELS; h++) {
        const uint64_t da = smem_desc_sw128(smem_u32(sdS + h * TILE_BYTES)), db = smem_desc_mn_sw128(smem_u32(kt + h * 8192));
#pragma unroll
        for (int k = 0; k < 4; k++) tc_mma(tmem + COL_DQ, da + 2 * k, db + (2048 >> 4) * k, id, (j | h | k) != 0);
      }
      tc_commit(&bs->d);
    }
  }
  ok = ok && wait(bs, &bs->d, (nkv - 1) & 1, p.error, 46);
  ok = __syncthreads_and(ok);
  if (ok) {
    tc_fence_after();
    const size_t orow = ((((size_t)b * p.S + q0 + row) * 3) * p.H + h) * D;
    if (cg < 2) store_acc_row(lane_addr, COL_DQ, cg, p.dqkv + orow);
  }
  if (tid == 0) drain(bs);
  tc_fence_before();
  __syncthreads();
  tmem_free<Step<STEP>::COLS>(tmem, warp);
}

// ------------------------------------------------------------------------------ host side
// One of Q / K / V inside qkv [B][S][3][H][64] (which = 0, 1, 2), or a plain [B][S][H][64] tensor (which = -1):
// dims {d, h, s, b}, box = 64 x 1 x rows x 1 (that many rows of one head).
static int make_map(CUtensorMap* map, const void* ptr, int B, int S, int H, int which, int rows) {
  EncodeTiledFn fn = encode_tiled_fn();
  if (!fn) return -10;
  const uint64_t row = (which >= 0 ? 3ull : 1ull) * H * D;          // elements between consecutive sequence positions
  const char* basep = (const char*)ptr + (which > 0 ? (size_t)which * H * D * 2 : 0);
  if ((uintptr_t)basep & 15) return -11;
  cuuint64_t dims[4] = {(cuuint64_t)D, (cuuint64_t)H, (cuuint64_t)S, (cuuint64_t)B};
  cuuint64_t strides[3] = {(cuuint64_t)D * 2, row * 2, row * 2 * (cuuint64_t)S};
  cuuint32_t box[4] = {(cuuint32_t)D, 1, (cuuint32_t)rows, 1};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<char*>(basep), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    fprintf(stderr, "gcow attention: cuTensorMapEncodeTiled failed with CUresult %d (B %d S %d H %d which %d)\n", (int)r, B, S, H, which);
    return -12;
  }
  return 0;
}

constexpr size_t kFwdSmem = TILE_BYTES * 13 + sizeof(Bars) + 1024;      // Q + 4 K + 4 V + 4 P
template <int STEP> constexpr size_t kBwdSmem =                            // K, V, P, dS, 2 Q, 2 dO, statistics
    TILE_BYTES * (2 + 2 * Step<STEP>::PANELS) + Step<STEP>::BYTES * 4 + MAX_S * 8 + sizeof(Bars) + 1024;
template <int STEP> constexpr size_t kDqSmem =                             // Q, dO, dS, 2 K, 2 V
    TILE_BYTES * (2 + Step<STEP>::PANELS) + Step<STEP>::BYTES * 4 + sizeof(Bars) + 1024;
static_assert(kBwdSmem<64> <= 112 * 1024 && kDqSmem<64> <= 112 * 1024, "two CTAs per SM");
static_assert(kBwdSmem<128> <= 227 * 1024 && kDqSmem<128> <= 227 * 1024, "one CTA per SM");

static int check_shape(int B, int S, int H, int d) {
  if (d != D || S % TILE || S <= 0 || S > MAX_S || B <= 0 || H <= 0 || H > 65535 || B > 65535) return -1;
  return 0;
}

static void set_attrs() {
  static std::once_flag once;
  std::call_once(once, [] {
    cudaFuncSetAttribute(attn_fwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFwdSmem);
    cudaFuncSetAttribute(attn_bwd_dkdv_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kBwdSmem<64>);
    cudaFuncSetAttribute(attn_bwd_dkdv_kernel<128>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kBwdSmem<128>);
    cudaFuncSetAttribute(attn_bwd_dq_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kDqSmem<64>);
    cudaFuncSetAttribute(attn_bwd_dq_kernel<128>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kDqSmem<128>);
  });
}

// The backward kernels; STEP as in Step.
template <int STEP>
static int launch_bwd(const void* qkv, const void* out, const void* dout, float* delta, const Params& p, cudaStream_t st) {
  CUtensorMap tile[4], step[4];                              // Q, K, V, dO in boxes of TILE and of STEP rows
  for (int i = 0; i < 4; i++) {
    const void* const m = i < 3 ? qkv : dout;
    int rc;
    if ((rc = make_map(&tile[i], m, p.B, p.S, p.H, i < 3 ? i : -1, TILE))) return rc;
    if (STEP == TILE) step[i] = tile[i];
    else if ((rc = make_map(&step[i], m, p.B, p.S, p.H, i < 3 ? i : -1, STEP))) return rc;
  }
  const size_t rows = (size_t)p.B * p.S * p.H;
  attn_delta_kernel<<<(unsigned)((rows * 8 + 255) / 256), 256, 0, st>>>((const __nv_bfloat16*)out, (const __nv_bfloat16*)dout, delta, p.B, p.S, p.H);
  const dim3 grid(p.S / TILE, p.H, p.B);
  attn_bwd_dkdv_kernel<STEP><<<grid, NT, kBwdSmem<STEP>, st>>>(step[0], tile[1], tile[2], step[3], p);
  attn_bwd_dq_kernel<STEP><<<grid, NT, kDqSmem<STEP>, st>>>(tile[0], step[1], step[2], tile[3], p);
  return (int)cudaGetLastError();
}

}  // namespace attn
}  // namespace gcow

using namespace gcow::attn;

extern "C" {

// 1 if the fused kernels cover this problem (head dimension 64, S a multiple of 128 up to 512).
int gcow_attention_supported(int B, int S, int H, int d) { return check_shape(B, S, H, d) == 0; }

// out[B][S][H][64] = softmax(scale * Q K^T) V per head, qkv [B][S][3][H][64] bf16; lse [B][H][S] fp32 receives the
// log2-sum-exp of the scaled scores (kept for the backward pass). `error`: device word, set if a wait gave up.
int gcow_attention_fwd(const void* qkv, void* out, float* lse, int B, int S, int H, int d, float scale,
                       uint32_t* error, void* stream) {
  if (check_shape(B, S, H, d)) return -1;
  set_attrs();
  CUtensorMap tq, tk, tv;
  int rc;
  if ((rc = make_map(&tq, qkv, B, S, H, 0, TILE)) || (rc = make_map(&tk, qkv, B, S, H, 1, TILE)) || (rc = make_map(&tv, qkv, B, S, H, 2, TILE)))
    return rc;
  Params p = {};
  p.out = (__nv_bfloat16*)out; p.lse = lse; p.B = B; p.S = S; p.H = H;
  p.scale = scale; p.scale_log2 = scale * 1.4426950408889634f; p.error = error;
  attn_fwd_kernel<<<dim3(S / TILE, H, B), NT, kFwdSmem, (cudaStream_t)stream>>>(tq, tk, tv, p);
  return (int)cudaGetLastError();
}

// dqkv[B][S][3][H][64] from qkv, the forward's out and lse, and dout [B][S][H][64]; delta [B][H][S] fp32 is scratch.
int gcow_attention_bwd(const void* qkv, const void* out, const void* dout, const float* lse, float* delta, void* dqkv,
                       int B, int S, int H, int d, float scale, uint32_t* error, void* stream) {
  if (check_shape(B, S, H, d)) return -1;
  set_attrs();
  cudaStream_t st = (cudaStream_t)stream;
  Params p = {};
  p.lse = const_cast<float*>(lse); p.delta = delta; p.dqkv = (__nv_bfloat16*)dqkv; p.B = B; p.S = S; p.H = H;
  p.scale = scale; p.scale_log2 = scale * 1.4426950408889634f; p.error = error;
  // Two CTAs per SM hide one another's chain of steps, but only where there are more CTAs than SMs; with fewer, each has an SM
  // to itself and half as many steps are the shorter chain. 512 positions, 128 CTAs: 38.6 us with steps of 64, 29.9 with 128;
  // 192 CTAs: 48.4 and 55.4 (128 positions, 148 CTAs or fewer: 18.1 and 16.3).
  return (long long)(S / TILE) * H * B <= 148 ? launch_bwd<128>(qkv, out, dout, delta, p, st) : launch_bwd<64>(qkv, out, dout, delta, p, st);
}

}  // extern "C"
