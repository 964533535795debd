// Fused multi-head self-attention on the 5th-generation tensor cores (sm_100a), head dimension 64, 72 to 512 positions (a
// multiple of 8), no mask, no dropout: forward and backward.
//
// The kernels read the packed projection qkv [B][S][3][H][64] (bf16) in place through 4-D tensor maps {d, h, s, b} - a
// box is 128 sequence positions of one head, 128-byte rows with the 128-byte swizzle - and write the context / gradients in
// the layouts the neighbouring GEMMs use ([B][S][H][64] and [B][S][3][H][64]), so no transposed copy of Q, K or V exists.
//
//  forward   a tile is 128 queries of a head; S = Q K^T comes in blocks of 128 keys. One thread per query takes the block's
//            128 scores into registers (which frees their tensor-memory columns for the next block's product), their maximum
//            and their exponentials, and puts P as bf16 into tensor memory, from where it is the A operand of O += P V. O is
//            read back and rescaled where a row's running maximum has moved. Also stores the row's
//            log2-sum-exp for the backward pass.
//  backward  recomputes P from Q, K and the stored log-sum-exp, in blocks of 128 x 64, one row per thread as above.
//     dK/dV  a tile is 128 keys, the loop runs over the queries: S^T = K Q^T and dP^T = V dO^T, so lse and delta belong to the
//            columns; P^T and dS^T = P^T (dP^T - delta) are A operands in tensor memory of dV += P^T dO and dK += dS^T Q.
//     dQ     a tile is 128 queries, the loop runs over the keys: S, dP, dS, then dQ += dS K. Recomputing S and dP here
//            instead of adding dQ with atomics keeps the gradients deterministic.
//  delta = rowsum(dO * O) comes from a small elementwise kernel.
//
// One persistent CTA per SM with two tiles in flight, A and B, 128 threads each: while one waits for its product the other
// one's exponentials run. A warp per tile issues its products (two in the backward pass), another one the TMA loads; whole
// sequences of the streamed operands (64 KB each) are held, and refilled for the next unit of work block by block as the
// last product that reads a block completes.
//
// Every mbarrier wait is bounded: after a fixed number of polls the CTA records an error code, all roles leave their loops,
// wait (bounded) for outstanding copies and MMAs, free the tensor memory and return. No load uses cluster multicast. The
// reference's models are CNNs (hw/models/train_imagenet.py:199-202); these kernels serve the BERT configuration.
#include <stdio.h>
#include <mutex>

#include "pdl.cuh"
#include "tc_common.cuh"

namespace gcow {
namespace attn {

using namespace gcow::tc;

constexpr int D = 64;                 // head dimension: one 128-byte row
constexpr int TILE = 128;             // rows of a query / key tile
constexpr int TILE_BYTES = TILE * D * 2;   // 16 KB
constexpr int MAX_S = 512;

struct Params {
  float* lse;              // [B][H][S] log2-sum-exp of the scaled scores
  const float* delta;      // backward: [B][H][S] rowsum(dO * O)
  int B, S, H;
  float scale_log2;        // softmax scale * log2(e)
  float scale;             // softmax scale
  uint32_t* error;
};

__device__ __forceinline__ uint32_t idesc_f16(int n, bool a_mn, bool b_mn) {
  // fp32 accumulate, bf16 x bf16, operand major-ness, N, M = 128
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)a_mn << 15) | ((uint32_t)b_mn << 16) |
         ((uint32_t)(n >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
}
__device__ __forceinline__ void proxy_fence() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ uint32_t pack2(float a, float b) {
  __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&v);
}
__device__ __forceinline__ float max3(float a, float b, float c) {
  float r; asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c)); return r;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t r; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r;
}
// 32 fp32 values of a row as bf16 at elements e0.. of a 64-element row in the 128-byte swizzle that the TMA reads.
__device__ __forceinline__ void store_row32(uint8_t* tile, int row, int e0, const float (&v)[32]) {
#pragma unroll
  for (int j = 0; j < 4; j++) {
    const uint4 o = make_uint4(pack2(v[8 * j], v[8 * j + 1]), pack2(v[8 * j + 2], v[8 * j + 3]),
                               pack2(v[8 * j + 4], v[8 * j + 5]), pack2(v[8 * j + 6], v[8 * j + 7]));
    *reinterpret_cast<uint4*>(tile + row * 128 + ((((e0 >> 3) + j) ^ (row & 7)) << 4)) = o;
  }
}
__device__ __forceinline__ void tc_st32(uint32_t taddr, const uint32_t* r) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
      "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
      "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
      ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
        "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]),
        "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]), "r"(r[23]),
        "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
      : "memory");
}
__device__ __forceinline__ void tc_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// D += A B with A [128 x 16] in tensor memory: row r in lane r, two bf16 per column
__device__ __forceinline__ void tc_mma_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(acc) : "memory");
}
__device__ __forceinline__ void tma_store_4d(const CUtensorMap* map, uint32_t src, int x, int y, int z, int w) {
  asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.bulk_group [%0, {%2, %3, %4, %5}], [%1];"
               ::"l"((uint64_t)map), "r"(src), "r"(x), "r"(y), "r"(z), "r"(w) : "memory");
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}

// Work of a CTA: units of one or two tiles of 128 rows, A and B. kSingle: one tile each; kPair: two of one head (the last one
// of an odd number stands alone); kHeads (up to 128 positions): one tile of each of two heads.
enum UnitMode { kSingle, kPair, kHeads };
struct Unit { int bh[2], q[2]; bool both; };
__device__ __forceinline__ Unit unit_at(int u, int mode, int tiles, int heads) {
  Unit r;
  if (mode == kHeads) {
    r.bh[0] = 2 * u; r.bh[1] = 2 * u + 1; r.q[0] = r.q[1] = 0; r.both = 2 * u + 1 < heads;
  } else {
    const int per = mode == kSingle ? tiles : (tiles + 1) / 2;
    r.bh[0] = r.bh[1] = u / per;
    r.q[0] = (u % per) * (mode == kSingle ? 1 : 2); r.q[1] = r.q[0] + 1;
    r.both = mode == kPair && r.q[1] < tiles;
  }
  return r;
}

// The barriers of a CTA are numbered, and a role keeps the parities it waits for next in one word.
//
// B 32, S 512, 16 heads: forward 123 us with one tile in flight and the probabilities through shared memory, now 67 (0.51
// PFLOP/s; the 134 M exponentials take 29 at 16 a clock and SM); backward 327, now 211 (delta 12; 233 with the queries' statistics fetched one
// row a lane and one lane of a diverged warp issuing; before that 251 with one issuing warp per tile in the backward pass, 242 with dQ behind
// dK/dV, 231 as a launch of its own beside it). One head of 512: backward 24.8, now 16.5 us.
// Bound by the row warps' chains of load, exponentials and stores, two warps a scheduler (four backward): a block of the forward pass takes one 3900
// cycles, of which exponentials 1640, epilogue and stores 780, waits for the scores 460, where the exponential unit needs 1024. A quarter of the
// exponentials as polynomials on the multiply-add pipe: forward 64.7, 65.8, backward 210, 205 but short sequences 2 to 5 % longer.
//
// What the issuing warps do per product decides the pace. As code of one thread alone, with the descriptors worked out where
// they are used, a step of four to eight MMAs took it 1500 cycles (forward, B 32, S 512, 16 heads: 131 us). So the whole warp
// runs the loop, all its values are uniform, and one elected lane executes the MMAs, commits and copies alone (95 us). A wait that has nothing to wait for
// still takes 110 cycles and an MMA with its descriptors 70, so each tile has a warp of its own.
struct Phases {
  uint32_t bits = 0;
  __device__ __forceinline__ uint32_t next(int i) {
    const uint32_t p = (bits >> i) & 1u;
    bits ^= 1u << i;
    return p;
  }
};
// Waits (bounded) until the last copy that was issued on a barrier has landed: `next` has the parity of the one after it.
__device__ __forceinline__ void landed(uint64_t* bar, uint32_t next) {
  for (uint32_t it = 0; it < kSpinLimit; it++) if (mbar_try_wait(bar, next ^ 1u)) break;
}
__device__ __forceinline__ void drain(uint64_t* bar) {      // everything this thread has issued to the tensor core is done
  tc_commit(bar);
  for (uint32_t it = 0; it < kSpinLimit; it++) if (mbar_try_wait(bar, 0)) break;
}
__device__ __forceinline__ void tmem_alloc_all(uint32_t* slot) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)), "r"(512u) : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_free_all(uint32_t base) {
  __syncwarp();
  tc_fence_after();
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(base), "r"(512u) : "memory");
}

// Two groups of 128 threads that work on a row each, and one whose warps issue the products and the loads. A row's
// thread holds 128 scores and their 64 packed probabilities (backward: 64 scores, probabilities and gradients each), more than
// a third of an SM's registers allows (168 a thread): it takes what the third group gives up.
// The backward pass has two groups of the latter, 512 threads of 128 registers.
template <bool FWD> struct Shape {
  static constexpr int THREADS = FWD ? 384 : 512, REGS = FWD ? 168 : 128, ROW = FWD ? 208 : 184, ISSUE = FWD ? 88 : 72;
  static_assert(2 * ROW + (THREADS / 128 - 2) * ISSUE == THREADS / 128 * REGS && THREADS * REGS <= 65536, "setmaxnreg.inc waits for registers that must exist");
};
template <bool FWD> __device__ __forceinline__ void regs_issue() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(Shape<FWD>::ISSUE)); }
template <bool FWD> __device__ __forceinline__ void regs_row() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(Shape<FWD>::ROW)); }

// ------------------------------------------------------------------------------ forward
// Barriers, each for tile A and B or for the four blocks of keys. K and V blocks: full[2][4], free[2][4].
enum FwdBar { kQFull = 0, kQFree = 2, kKvFull = 4, kKvFree = 12, kSFull = 20, kSFree = 22, kPFull = 24, kPv = 26, kFwdDrain = 28, kFwdBars = 30 };
struct FwdBars {
  uint64_t bar[kFwdBars];
  uint32_t tmem_base;
  volatile uint32_t abort;
};

__global__ void __launch_bounds__(Shape<true>::THREADS, 1)
attn_fwd_kernel(const __grid_constant__ CUtensorMap tq, const __grid_constant__ CUtensorMap tk, const __grid_constant__ CUtensorMap tv,
                const __grid_constant__ CUtensorMap to, const Params p, int units, int mode) {
  extern __shared__ uint8_t raw[];
  uint8_t* base = reinterpret_cast<uint8_t*>(((uintptr_t)raw + 1023) & ~(uintptr_t)1023);
  uint8_t* const sQ = base;                  // A, B
  uint8_t* const sO = sQ + 2 * TILE_BYTES;   // 4 KB per softmax warp
  uint8_t* const sK = sO + 2 * TILE_BYTES;   // blocks of 128 keys
  uint8_t* const sV = sK + 4 * TILE_BYTES;
  FwdBars* const bs = reinterpret_cast<FwdBars*>(sV + 4 * TILE_BYTES);
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;   // warp: uniform
  const int tiles = (p.S + TILE - 1) / TILE, heads = p.B * p.H;
  const int blocks = tiles;                  // blocks of 128 keys; the last one may be partial: its copy fills up with zeros
  const int u0 = (int)((long long)units * blockIdx.x / gridDim.x), u1 = (int)((long long)units * (blockIdx.x + 1) / gridDim.x);

  if (tid == 0) {
    // 4: the warps of a tile; keys and values that two tiles share are free when both have used them
    for (int i = 0; i < kFwdBars; i++) mbar_init(&bs->bar[i], i >= kSFree && i < kPv ? 4 : i >= kKvFree && i < kSFull && mode == kPair ? 2 : 1);
    bs->abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) tmem_alloc_all(&bs->tmem_base);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = bs->tmem_base;
  pdl_trigger();
  pdl_wait();
  // columns: S of A, B (128 each), P of A, B (64 each), O of A, B (64 each)
  auto col_s = [&](int x) { return tmem + x * 128; };
  auto col_p = [&](int x) { return tmem + 256 + x * 64; };
  auto col_o = [&](int x) { return tmem + 384 + x * 64; };

  if (warp >= 8) {
    regs_issue<true>();
    const bool one = elect_one();
    Phases ph;
    bool ok = true;
    auto wait = [&](int i, uint32_t code) {
      ok = __all_sync(0xffffffffu, mbar_wait_abortable(&bs->abort, &bs->bar[i], ph.next(i), p.error, code)) && ok;
    };
    if (warp == 10) {                                        // ---- loads
      uint32_t issued = 0, landing = 0;                      // by barrier: a copy has been issued; the parity after it
      for (int u = u0; u < u1 && ok; u++) {
        const Unit un = unit_at(u, mode, tiles, heads);
        const int nx = un.both ? 2 : 1, nk = mode == kHeads ? nx : blocks;   // key blocks held: those of the head, or one of each
        // Q of A, the first keys, Q of B, the other keys, the values
#pragma unroll 1
        for (int n = 0; n < nx + 2 * nk && ok; n++) {
          const bool is_q = n == 0 || (n == 2 && nx == 2);
          const int kv = n - 1 - (n > 2 && nx == 2), x = n >> 1, is_v = kv >= nk, i = is_v ? kv - nk : kv;
          const int full = is_q ? kQFull + x : kKvFull + 4 * is_v + i, empty = is_q ? kQFree + x : kKvFree + 4 * is_v + i;
          const int bh = is_q ? un.bh[x] : mode == kHeads ? un.bh[i] : un.bh[0];
          const int row = is_q ? un.q[x] * TILE : mode == kHeads ? 0 : i * TILE;
          uint8_t* const dst = is_q ? sQ + x * TILE_BYTES : (is_v ? sV : sK) + i * TILE_BYTES;
          if ((issued >> full) & 1u) wait(empty, 21);
          if (!ok) break;
          const int b = bh / p.H, h = bh - b * p.H;
          if (one) {
            mbar_expect_tx(&bs->bar[full], TILE_BYTES);
            tma_load_4d(smem_u32(dst), is_q ? &tq : is_v ? &tv : &tk, smem_u32(&bs->bar[full]), 0, h, row, b);
          }
          issued |= 1u << full;
          landing ^= 1u << full;
        }
      }
      // nothing may be in flight when the CTA ends (there is something to wait for only after a wait gave up)
#pragma unroll 1
      for (int i = 0; i < kKvFree; i++) if ((issued >> i) & 1u) landed(&bs->bar[i], (landing >> i) & 1u);
    } else if (warp < 10) {                                  // ---- products, warp 8: of tile A, 9: of tile B
      const int x = warp - 8;
      bool held = false, ahead = false;                      // S has been written before; this unit's first S has been issued
      const uint32_t id_qk = idesc_f16(TILE, false, false), id_pv = idesc_f16(D, false, true);
      const uint64_t dq = smem_desc_sw128(smem_u32(sQ + x * TILE_BYTES)), dk = smem_desc_sw128(smem_u32(sK)), dv = smem_desc_mn_sw128(smem_u32(sV));
      const bool apart = mode == kHeads;                     // each tile has its own keys
      for (int u = u0; u < u1 && ok; u++) {
        const Unit un = unit_at(u, mode, tiles, heads);
        if (x && !un.both) {                                 // nothing to do but to let go of what the other tile is given
          if (mode == kPair)
#pragma unroll 1
            for (int i = 0; i < 2 * blocks && ok; i++) {
              const int op = i < blocks ? i : 4 + i - blocks;
              wait(kKvFull + op, 22);
              if (ok && one) mbar_arrive(&bs->bar[kKvFree + op]);
              __syncwarp();
            }
          continue;
        }
        auto qk = [&](int j) {
          const int i = apart ? x : j;
          if (j == 0) wait(kQFull + x, 23);
          wait(kKvFull + i, 24);
          if (held) wait(kSFree + x, 25);
          held = true;
          if (!ok) return;
          tc_fence_after();
          const uint64_t db = dk + i * (uint64_t)(TILE_BYTES >> 4);
          if (one) {
#pragma unroll
            for (int k = 0; k < 4; k++) tc_mma(col_s(x), dq + 2 * k, db + 2 * k, id_qk, k != 0);
            tc_commit(&bs->bar[kSFull + x]);
            tc_commit(&bs->bar[kKvFree + i]);
            if (j == blocks - 1) tc_commit(&bs->bar[kQFree + x]);
          }
          __syncwarp();
        };
        // step j: S of block j, then O of block j - 1; the next unit's first S comes before this one's last O
        if (!ahead) qk(0);
        ahead = u + 1 < u1 && (!x || unit_at(u + 1, mode, tiles, heads).both);
#pragma unroll 1
        for (int j = 1; j <= blocks && ok; j++) {
          if (j < blocks || ahead) qk(j < blocks ? j : 0);
          const int i = apart ? x : j - 1;
          wait(kKvFull + 4 + i, 26);
          wait(kPFull + x, 27);
          if (!ok) break;
          tc_fence_after();
          const uint64_t db = dv + i * (uint64_t)(TILE_BYTES >> 4);
          if (one) {
#pragma unroll
            for (int k = 0; k < 8; k++) tc_mma_ts(col_o(x), col_p(x) + 8 * k, db + (2048 >> 4) * k, id_pv, k != 0 || j != 1);
            tc_commit(&bs->bar[kPv + x]);
            tc_commit(&bs->bar[kKvFree + 4 + i]);
          }
          __syncwarp();
        }
      }
      if (one) drain(&bs->bar[kFwdDrain + x]);
    }
  } else {
    // ---- softmax and output: one query per thread
    regs_row<true>();
    const int x = warp >> 2, row = tid & 127;
    // the whole warp goes on or gives up: what follows is collective
    Phases ph;
    auto wait_all = [&](int i, uint32_t code) {
      return __all_sync(0xffffffffu, mbar_wait_abortable(&bs->abort, &bs->bar[i], ph.next(i), p.error, code)) != 0;
    };
    const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
    uint8_t* const stage = sO + warp * (32 * 128);           // the warp's 32 rows
    bool ok = true;
    for (int u = u0; u < u1 && ok; u++) {
      const Unit un = unit_at(u, mode, tiles, heads);
      if (x == 1 && !un.both) continue;
      float m = 0.0f;
      uint64_t l2 = 0, l2b = 0;
      for (int j = 0; j < blocks; j++) {
        if (!(ok = ok && wait_all(kSFull + x, 28))) break;
        tc_fence_after();
        uint32_t s[4][32];
#pragma unroll
        for (int c = 0; c < 4; c++) tc_ld32(col_s(x) + lanes + c * 32, s[c]);
        tc_wait_ld();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bs->bar[kSFree + x]);
        if (j == blocks - 1 && p.S < blocks * TILE) {        // keys that do not exist
          const int valid = p.S - j * TILE;
#pragma unroll
          for (int c = 0; c < 4; c++)
#pragma unroll
            for (int i = 0; i < 32; i++) if (c * 32 + i >= valid) s[c][i] = 0xff800000u;   // -inf
        }
        float bm[4];
#pragma unroll
        for (int c = 0; c < 4; c++) {
          bm[c] = fmaxf(__uint_as_float(s[c][0]), __uint_as_float(s[c][1]));
#pragma unroll
          for (int i = 2; i < 32; i += 2) bm[c] = max3(bm[c], __uint_as_float(s[c][i]), __uint_as_float(s[c][i + 1]));
        }
        const float top = max3(fmaxf(bm[0], bm[1]), bm[2], bm[3]);
        // The running maximum is followed at once: a row's largest probability is then exactly 1, also as bf16. Following it only
        // where it has fallen 8 powers of two behind saves 3 of 67 us and costs concentrated rows a sixth more error (scores of
        // deviation 9 over 512 keys: 1.65e-3 -> 1.91e-3).
        float keep = 1.0f;
        if (j == 0) m = fmaxf(top, -1e30f);                  // finite: a block of -inf does not decide the row
        else if (top > m) {
          keep = ex2_ftz((m - top) * p.scale_log2);
          m = top;
        }
        const float ms = m * p.scale_log2;
        const uint64_t sl = tc::pack2(p.scale_log2, p.scale_log2), nm = tc::pack2(-ms, -ms);
        if (j) {
          const uint64_t k2 = tc::pack2(keep, keep);
          l2 = mul2(l2, k2);
          l2b = mul2(l2b, k2);
        }
        uint32_t pk[64];
#pragma unroll
        for (int c = 0; c < 4; c++)
#pragma unroll
          for (int i = 0; i < 32; i += 2) {
            float a, b;
            unpack2(fma2(tc::pack2(__uint_as_float(s[c][i]), __uint_as_float(s[c][i + 1])), sl, nm), a, b);
            a = ex2_ftz(a);
            b = ex2_ftz(b);
            if (i & 2) l2 = add2(l2, tc::pack2(a, b)); else l2b = add2(l2b, tc::pack2(a, b));
            pk[c * 16 + i / 2] = pack2(a, b);
          }
        if (j) {
          if (!(ok = ok && wait_all(kPv + x, 29))) break;   // P of the last block has been read, O holds it
          tc_fence_after();
          if (__any_sync(0xffffffffu, keep != 1.0f)) {
            uint32_t o[32];
#pragma unroll
            for (int c = 0; c < 2; c++) {
              tc_ld32(col_o(x) + lanes + c * 32, o);
              tc_wait_ld();
#pragma unroll
              for (int i = 0; i < 32; i++) o[i] = __float_as_uint(__uint_as_float(o[i]) * keep);
              tc_st32(col_o(x) + lanes + c * 32, o);
            }
          }
        }
        tc_st32(col_p(x) + lanes, pk);
        tc_st32(col_p(x) + lanes + 32, pk + 32);
        tc_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&bs->bar[kPFull + x]);
      }
      ok = ok && wait_all(kPv + x, 30);
      if (!ok) break;
      tc_fence_after();
      float la, lb, lc, ld;
      unpack2(l2, la, lb);
      unpack2(l2b, lc, ld);
      const float l = (la + lb) + (lc + ld), inv = 1.0f / l;
      uint32_t o[2][32];
      tc_ld32(col_o(x) + lanes, o[0]);
      tc_ld32(col_o(x) + lanes + 32, o[1]);
      tc_wait_ld();
      if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");   // the last store has read the staging rows
      __syncwarp();
#pragma unroll
      for (int c = 0; c < 2; c++) {
        float v[32];
#pragma unroll
        for (int i = 0; i < 32; i++) v[i] = __uint_as_float(o[c][i]) * inv;
        store_row32(stage, lane, c * 32, v);
      }
      if (un.q[x] * TILE + row < p.S) p.lse[(size_t)un.bh[x] * p.S + un.q[x] * TILE + row] = m * p.scale_log2 + log2f(l);
      proxy_fence();
      __syncwarp();
      const int r0 = un.q[x] * TILE + (warp & 3) * 32;       // the map clips a partial block's rows
      if (lane == 0 && r0 < p.S) tma_store_4d(&to, smem_u32(stage), 0, un.bh[x] % p.H, r0, un.bh[x] / p.H);
    }
    if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_free_all(tmem);
}

// delta[b][h][s] = sum_d dO[b][s][h][d] * O[b][s][h][d]; eight lanes per row, so that a warp reads whole lines, and kDeltaRows rows to a
// lane, all of whose loads are under way before the first sum. Bound by memory. With one row and 64-bit divisions for its place, two rows, four
// rows to a lane, the whole backward takes: 32 x 512 x 16 heads 240.4, 238.2, 238.4 us; 8 x 512 x 16 74.0, 73.3, 75.5; 2 x 512 x 16 30.0, 30.3, 31.0;
// 1 x 128 x 2 9.8, 9.6, 10.0: with four, few rows are too few CTAs.
constexpr int kDeltaRows = 2;
__global__ void __launch_bounds__(256)
attn_delta_kernel(const __nv_bfloat16* o, const __nv_bfloat16* go, float* __restrict__ delta, uint32_t rows, uint32_t S, uint32_t H) {
  pdl_trigger();
  pdl_wait();
  const uint32_t first = blockIdx.x * (32 * kDeltaRows) + (threadIdx.x >> 3), part = threadIdx.x & 7;      // rows over b, s, h
  uint4 x[kDeltaRows], y[kDeltaRows];
#pragma unroll
  for (int k = 0; k < kDeltaRows; k++) {
    const uint32_t i = first + 32 * k;
    x[k] = y[k] = make_uint4(0, 0, 0, 0);
    if (i < rows) {
      x[k] = reinterpret_cast<const uint4*>(o + (size_t)i * D)[part];
      y[k] = reinterpret_cast<const uint4*>(go + (size_t)i * D)[part];
    }
  }
  float mine = 0.0f;                                   // lane `part` < kDeltaRows stores row `part`
#pragma unroll
  for (int k = 0; k < kDeltaRows; k++) {
    const __nv_bfloat162* xb = reinterpret_cast<const __nv_bfloat162*>(&x[k]);
    const __nv_bfloat162* yb = reinterpret_cast<const __nv_bfloat162*>(&y[k]);
    float acc = 0.0f;
#pragma unroll
    for (int e = 0; e < 4; e++) {
      const float2 a = __bfloat1622float2(xb[e]), c = __bfloat1622float2(yb[e]);
      acc = fmaf(a.x, c.x, fmaf(a.y, c.y, acc));
    }
#pragma unroll
    for (int d = 1; d < 8; d <<= 1) acc += __shfl_xor_sync(0xffffffffu, acc, d);
    if ((int)part == k) mine = acc;
  }
  const uint32_t i = first + 32 * part;
  if (part < kDeltaRows && i < rows) {
    const uint32_t bs = i / H, h = i - bs * H, b = bs / S, at = bs - b * S;
    delta[((size_t)b * H + h) * S + at] = mine;
  }
}

// ------------------------------------------------------------------------------ backward
// Barriers, each for tile A and B, for the two operands of the sequence's four blocks, or for two units' statistics.
enum BwdBar { kAFull = 0, kAFree = 2, kBFull = 4, kBFree = 12, kStatFull = 16, kStatFree = 18, kSAt = 20, kSGone = 22, kDpAt = 24,
              kReady = 26, kAcc = 28, kBwdBars = 30 };
struct BwdBars {
  uint64_t bar[kBwdBars], drain[4];
  uint32_t tmem_base;
  volatile uint32_t abort;
};

// KV = true: a tile is 128 keys, the loop runs over blocks of 64 queries: S^T = K Q^T, dP^T = V dO^T, dV += P^T dO, dK += dS^T Q.
// KV = false: a tile is 128 queries, the loop runs over blocks of 64 keys: S = Q K^T, dP = dO V^T, dQ += dS K.
// a1, a2: the tile's operands (K, V or Q, dO); b1, b2: those of the whole sequence (Q, dO or K, V); to1, to2: dV, dK or -, dQ.
template <bool KV>
__device__ __forceinline__ void attn_bwd_body(const CUtensorMap& ta1, const CUtensorMap& ta2, const CUtensorMap& tb1, const CUtensorMap& tb2,
                                              const CUtensorMap& to1, const CUtensorMap& to2, const Params& p, int units, int mode, int cta, int ctas) {
  constexpr int STEP = 64, STEP_BYTES = STEP * D * 2;
  extern __shared__ uint8_t raw[];
  uint8_t* base = reinterpret_cast<uint8_t*>(((uintptr_t)raw + 1023) & ~(uintptr_t)1023);
  uint8_t* const sA = base;                  // [tile A, B][a1, a2]
  uint8_t* const sB1 = sA + 4 * TILE_BYTES;  // the sequence, 128 rows per slot
  uint8_t* const sB2 = sB1 + 4 * TILE_BYTES;
  uint8_t* const sO = sB2 + 4 * TILE_BYTES;  // 2 KB per row warp
  float* const stats = reinterpret_cast<float*>(sO + TILE_BYTES);      // KV: [2][-lse, -delta][MAX_S], the units in turn
  BwdBars* const bs = reinterpret_cast<BwdBars*>(stats + 4 * MAX_S);
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;   // warp: uniform
  const int tiles = (p.S + TILE - 1) / TILE, heads = p.B * p.H;
  const int u0 = (int)((long long)units * cta / ctas), u1 = (int)((long long)units * (cta + 1) / ctas);
  const int nb = (p.S + STEP - 1) / STEP;

  if (tid == 0) {
    // 4: the warps of a tile, 8: all row warps, 32: the warp that fetches statistics; a sequence that two tiles share is free
    // when both have used it, a tile's operands when each warp that reads them has. For dK/dV tile B's score warp counts beside
    // its accumulator warp: where there is no tile B neither waits for the other, and a block refilled before one of
    // them has looked would be a phase that it misses.
    for (int i = 0; i < kBwdBars; i++) {
      const int pair = i & ~1;
      mbar_init(&bs->bar[i], pair == kSGone || pair == kReady ? 4 : pair == kStatFree ? 8 : pair == kStatFull ? 32
                             : i >= kBFree && i < kStatFull && mode == kPair ? (KV ? 3 : 2) : KV && pair == kAFree ? 2 : 1);
    }
    for (int i = 0; i < 4; i++) mbar_init(&bs->drain[i], 1);
    bs->abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) tmem_alloc_all(&bs->tmem_base);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = bs->tmem_base;
  pdl_wait();
  pdl_trigger();
  // Columns of a tile: S 64, dP 64, two accumulators of 64. P and dS (32 each, bf16) take dP's place once it has been read; with
  // one accumulator dS has a place of its own, and dP can be refilled at once.
  auto col = [&](int x) { return tmem + x * 256; };
  constexpr uint32_t DP = 64, P_AT = 64, DS_AT = KV ? 96 : 128, ACC1 = 128, ACC2 = 192;

  if (warp >= 8) {
    regs_issue<false>();
    const bool one = elect_one();
    Phases ph;
    bool ok = true;
    auto wait = [&](int i, uint32_t code) {
      ok = __all_sync(0xffffffffu, mbar_wait_abortable(&bs->abort, &bs->bar[i], ph.next(i), p.error, code)) && ok;
    };
    if (warp == 12) {                                        // ---- loads
      uint32_t issued = 0, landing = 0;                      // by barrier: a copy has been issued; the parity after it
      for (int u = u0; u < u1 && ok; u++) {
        const Unit un = unit_at(u, mode, tiles, heads);
        const int nx = un.both ? 2 : 1, slots = mode == kHeads ? nx : tiles;
        // the operands of A, the first block of the sequence, the operands of B, the other blocks; two copies each
#pragma unroll 1
        for (int n = 0; n < 2 * (nx + slots) && ok; n++) {
          const int which = n & 1, m = n >> 1;
          const bool is_a = m == 0 || (m == 2 && nx == 2);
          const int x = m >> 1, i = m - 1 - (m > 2 && nx == 2);
          const int full = is_a ? kAFull + x : kBFull + 4 * which + i;
          const int bh = is_a ? un.bh[x] : mode == kHeads ? un.bh[i] : un.bh[0];
          const int row = is_a ? un.q[x] * TILE : mode == kHeads ? 0 : i * TILE;
          uint8_t* const dst = is_a ? sA + (2 * x + which) * TILE_BYTES : (which ? sB2 : sB1) + i * TILE_BYTES;
          if (!which && ((issued >> full) & 1u)) wait(is_a ? kAFree + x : kBFree + i, 31);
          if (!ok) break;
          const int b = bh / p.H, h = bh - b * p.H;
          const bool arms = !is_a || !which;                 // one barrier for both operands of a tile
          if (one) {
            if (arms) mbar_expect_tx(&bs->bar[full], is_a ? 2 * TILE_BYTES : TILE_BYTES);
            tma_load_4d(smem_u32(dst), is_a ? (which ? &ta2 : &ta1) : (which ? &tb2 : &tb1), smem_u32(&bs->bar[full]), 0, h, row, b);
          }
          if (arms) landing ^= 1u << full;
          issued |= 1u << full;
        }
      }
      // nothing may be in flight when the CTA ends (there is something to wait for only after a wait gave up)
#pragma unroll 1
      for (int i = 0; i < kBFree; i++) if ((i < kAFree || i >= kBFull) && ((issued >> i) & 1u)) landed(&bs->bar[i], (landing >> i) & 1u);
    } else if (warp < 12) {
      // ---- products: warps 8, 9 issue S (with dP, where that has a place of its own) of tiles A, B, warps 10, 11 the accumulators
      // (and dP, where it takes the place of what they have read)
      const int x = warp & 1;
      const bool scores = warp < 10, apart = mode == kHeads; // apart: each tile has its own sequence
      const uint32_t id_s = idesc_f16(STEP, false, false), id_acc = idesc_f16(D, false, true), tm = col(x);
      const uint64_t da1 = smem_desc_sw128(smem_u32(sA + 2 * x * TILE_BYTES)), da2 = smem_desc_sw128(smem_u32(sA + (2 * x + 1) * TILE_BYTES));
      const int first = apart ? x * TILE_BYTES : 0;
      const uint64_t db1 = smem_desc_sw128(smem_u32(sB1 + first)), db2 = smem_desc_sw128(smem_u32(sB2 + first));
      const uint64_t dm1 = smem_desc_mn_sw128(smem_u32(sB1 + first)), dm2 = smem_desc_mn_sw128(smem_u32(sB2 + first));
      constexpr uint64_t kStep = STEP_BYTES >> 4;
      bool held = false;                                     // S has been written before
      for (int u = u0; u < u1 && ok; u++) {
        const Unit un = unit_at(u, mode, tiles, heads);
        if (x && !un.both) {                                 // nothing to do but to let go of what the other tile is given
          if (mode == kPair && (scores || KV))
#pragma unroll 1
            for (int i = 0; i < tiles && ok; i++) {          // each warp waits for what it waits for in the other units
              if (scores) wait(kBFull + i, 32);
              if (scores != KV) wait(kBFull + 4 + i, 32);
              if (ok && one) mbar_arrive(&bs->bar[kBFree + i]);
              __syncwarp();
            }
          continue;
        }
        if (scores) {
#pragma unroll 1
          for (int i = 0; i < nb && ok; i++) {
            const int sl = apart ? x : i >> 1;
            if (i == 0) wait(kAFull + x, 33);
            if (!(i & 1)) {
              wait(kBFull + sl, 34);
              if (!KV) wait(kBFull + 4 + sl, 34);
              if (KV && x && mode == kPair && ok && one) mbar_arrive(&bs->bar[kBFree + sl]);   // it is in use until the accumulators' products
            }
            if (held) wait(kSGone + x, 35);
            held = true;
            if (!ok) break;
            tc_fence_after();
            const uint64_t b1 = db1 + i * kStep, b2 = db2 + i * kStep;
            if (one) {
#pragma unroll
              for (int k = 0; k < 4; k++) {
                tc_mma(tm, da1 + 2 * k, b1 + 2 * k, id_s, k != 0);
                if (!KV) tc_mma(tm + DP, da2 + 2 * k, b2 + 2 * k, id_s, k != 0);
              }
              tc_commit(&bs->bar[kSAt + x]);
              if (i == nb - 1) tc_commit(&bs->bar[kAFree + x]);
            }
            __syncwarp();
          }
        } else {
          if (KV) wait(kAFull + x, 36);
#pragma unroll 1
          for (int i = 0; i <= nb && ok; i++) {
            const int sl = apart ? x : i >> 1;
            if (i > 0) {
              const uint64_t b1 = dm1 + (i - 1) * kStep, b2 = dm2 + (i - 1) * kStep;
              wait(kReady + x, 37);
              if (!ok) break;
              tc_fence_after();
              if (one) {
#pragma unroll
                for (int k = 0; k < 4; k++) {
                  if (KV) tc_mma_ts(tm + ACC1, tm + P_AT + 8 * k, b2 + (2048 >> 4) * k, id_acc, k != 0 || i != 1);
                  tc_mma_ts(tm + ACC2, tm + DS_AT + 8 * k, b1 + (2048 >> 4) * k, id_acc, k != 0 || i != 1);
                }
                tc_commit(&bs->bar[kAcc + x]);
                if (!(i & 1) || i == nb) tc_commit(&bs->bar[kBFree + (apart ? x : (i - 1) >> 1)]);
              }
              __syncwarp();
            }
            if (KV && i < nb) {
              if (!(i & 1)) wait(kBFull + 4 + sl, 38);
              if (!ok) break;
              tc_fence_after();
              const uint64_t b2 = db2 + i * kStep;
              if (one) {
#pragma unroll
                for (int k = 0; k < 4; k++) tc_mma(tm + DP, da2 + 2 * k, b2 + 2 * k, id_s, k != 0);
                tc_commit(&bs->bar[kDpAt + x]);
                if (i == nb - 1) tc_commit(&bs->bar[kAFree + x]);
              }
              __syncwarp();
            }
          }
        }
      }
      if (one) drain(&bs->drain[warp - 8]);
    } else if (KV && warp == 13) {                           // ---- statistics of the queries
      for (int u = u0, n = 0; u < u1 && ok; u++, n++) {
        const Unit un = unit_at(u, mode, tiles, heads);
        if (n >= 2) wait(kStatFree + (n & 1), 39);
        if (!ok) break;
        float* const st = stats + (n & 1) * 2 * MAX_S;
        // kHeads: one head's rows per 128. A query that does not exist has no probabilities (its rows of Q and dO are zeros).
        const int rows = mode == kHeads ? (un.both ? 2 * TILE : TILE) : tiles * TILE;
        // Eight rows a lane under way at a time: one after the other they took longer than a unit, which waited for them.
#pragma unroll 1
        for (int r0 = lane; r0 < rows; r0 += 8 * 32) {
          float l[8], d[8];
#pragma unroll
          for (int j = 0; j < 8; j++) {
            const int r = r0 + 32 * j, q = mode == kHeads ? r & (TILE - 1) : r;
            const size_t at = (size_t)(mode == kHeads && r >= TILE ? un.bh[1] : un.bh[0]) * p.S + q;
            l[j] = INFINITY;
            d[j] = 0.0f;
            if (r < rows && q < p.S) { l[j] = p.lse[at]; d[j] = p.delta[at]; }
          }
#pragma unroll
          for (int j = 0; j < 8; j++) {
            if (r0 + 32 * j < rows) { st[r0 + 32 * j] = -l[j]; st[MAX_S + r0 + 32 * j] = -d[j]; }
          }
        }
        mbar_arrive(&bs->bar[kStatFull + (n & 1)]);
      }
    }
  } else {
    // ---- gradients of the scores, results: one row of the tile per thread
    regs_row<false>();
    const int x = warp >> 2, row = tid & 127;
    // the whole warp goes on or gives up: what follows is collective
    Phases ph;
    auto wait_all = [&](int i, uint32_t code) {
      return __all_sync(0xffffffffu, mbar_wait_abortable(&bs->abort, &bs->bar[i], ph.next(i), p.error, code)) != 0;
    };
    const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
    uint8_t* const stage = sO + warp * kStageWarpBytes;
    bool ok = true;
    const uint64_t sl = tc::pack2(p.scale_log2, p.scale_log2), sc = tc::pack2(p.scale, p.scale);
    for (int u = u0, n = 0; u < u1 && ok; u++, n++) {
      const Unit un = unit_at(u, mode, tiles, heads);
      const float* st = stats + (n & 1) * 2 * MAX_S + (mode == kHeads && x ? TILE : 0);
      uint64_t nl = 0, nd = 0;
      if (KV) {
        if (!(ok = wait_all(kStatFull + (n & 1), 40))) break;
      } else if ((x == 0 || un.both) && un.q[x] * TILE + row < p.S) {   // rows past the end give values that nothing stores
        const size_t at = (size_t)un.bh[x] * p.S + un.q[x] * TILE + row;
        const float l = -p.lse[at], d = -p.delta[at];
        nl = tc::pack2(l, l);
        nd = tc::pack2(d, d);
      }
      if (x == 0 || un.both) {
        for (int i = 0; i < nb; i++) {
          if (!(ok = wait_all(kSAt + x, 41))) break;
          tc_fence_after();
          uint32_t s[2][32], dp[2][32];
          tc_ld32(col(x) + lanes, s[0]);
          tc_ld32(col(x) + lanes + 32, s[1]);
          if (!KV) {                                         // dP comes with S
            tc_ld32(col(x) + DP + lanes, dp[0]);
            tc_ld32(col(x) + DP + lanes + 32, dp[1]);
          }
          tc_wait_ld();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&bs->bar[kSGone + x]);
          uint32_t pk[32], dk[32];
          float pv[64];
#pragma unroll
          for (int c = 0; c < 2; c++)
#pragma unroll
            for (int e = 0; e < 32; e += 4) {
              uint64_t l0 = nl, l1 = nl;
              if (KV) {
                const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(st + i * STEP + c * 32 + e);
                l0 = v.x; l1 = v.y;
              }
              float* const o = pv + c * 32 + e;
              unpack2(fma2(tc::pack2(__uint_as_float(s[c][e]), __uint_as_float(s[c][e + 1])), sl, l0), o[0], o[1]);
              unpack2(fma2(tc::pack2(__uint_as_float(s[c][e + 2]), __uint_as_float(s[c][e + 3])), sl, l1), o[2], o[3]);
#pragma unroll
              for (int k = 0; k < 4; k++) o[k] = ex2_ftz(o[k]);
              if (KV) {
                pk[c * 16 + e / 2] = pack2(o[0], o[1]);
                pk[c * 16 + e / 2 + 1] = pack2(o[2], o[3]);
              }
            }
          if (KV) {
            if (!(ok = wait_all(kDpAt + x, 42))) break;
            tc_fence_after();
            tc_ld32(col(x) + DP + lanes, dp[0]);
            tc_ld32(col(x) + DP + lanes + 32, dp[1]);
            tc_wait_ld();
          }
#pragma unroll
          for (int c = 0; c < 2; c++)
#pragma unroll
            for (int e = 0; e < 32; e += 4) {
              uint64_t d0 = nd, d1 = nd;
              if (KV) {
                const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(st + MAX_S + i * STEP + c * 32 + e);
                d0 = v.x; d1 = v.y;
              }
              const float* const o = pv + c * 32 + e;
              float a, b;
              unpack2(mul2(mul2(tc::pack2(o[0], o[1]), add2(tc::pack2(__uint_as_float(dp[c][e]), __uint_as_float(dp[c][e + 1])), d0)), sc), a, b);
              dk[c * 16 + e / 2] = pack2(a, b);
              unpack2(mul2(mul2(tc::pack2(o[2], o[3]), add2(tc::pack2(__uint_as_float(dp[c][e + 2]), __uint_as_float(dp[c][e + 3])), d1)), sc), a, b);
              dk[c * 16 + e / 2 + 1] = pack2(a, b);
            }
          if (!KV && i == nb - 1 && p.S < nb * STEP) {       // keys that do not exist: their score of 0 may be far above the row's
            const int valid = (p.S - i * STEP) >> 1;         // others, their P beyond fp32
#pragma unroll
            for (int e = 0; e < 32; e++) if (e >= valid) dk[e] = 0;
          }
          if (i) {                                           // the last block's P and dS have been read
            if (!(ok = wait_all(kAcc + x, 43))) break;
            tc_fence_after();
          }
          if (KV) tc_st32(col(x) + P_AT + lanes, pk);
          tc_st32(col(x) + DS_AT + lanes, dk);
          tc_wait_st();
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&bs->bar[kReady + x]);
        }
        ok = ok && wait_all(kAcc + x, 44);
        if (!ok) break;
        tc_fence_after();
        const int h = un.bh[x] % p.H, b = un.bh[x] / p.H, r0 = un.q[x] * TILE + (warp & 3) * 32;
#pragma unroll
        for (int c = KV ? 0 : 2; c < 4; c++) {               // dV, then dK or dQ; 32 columns at a time
          uint32_t a[32];
          tc_ld32(col(x) + ACC1 + lanes + c * 32, a);
          tc_wait_ld();
          if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
          __syncwarp();
#pragma unroll
          for (int k = 0; k < 4; k++)
            *reinterpret_cast<uint4*>(stage + stage_offset(lane, k)) =
                make_uint4(pack2(__uint_as_float(a[8 * k]), __uint_as_float(a[8 * k + 1])), pack2(__uint_as_float(a[8 * k + 2]), __uint_as_float(a[8 * k + 3])),
                           pack2(__uint_as_float(a[8 * k + 4]), __uint_as_float(a[8 * k + 5])), pack2(__uint_as_float(a[8 * k + 6]), __uint_as_float(a[8 * k + 7])));
          proxy_fence();
          __syncwarp();
          if (lane == 0 && r0 < p.S) tma_store_4d(c < 2 ? &to1 : &to2, smem_u32(stage), (c & 1) * 32, h, r0, b);
        }
      }
      if (KV) {
        __syncwarp();
        if (lane == 0) mbar_arrive(&bs->bar[kStatFree + (n & 1)]);
      }
    }
    if (lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_free_all(tmem);
}

// Both in one launch, dK/dV on the first half of the CTAs, dQ on the other: they read the same and write apart, so neither waits
// for the other. A grid that leaves SMs idle, and the end of dK/dV, is filled with dQ's CTAs.
__global__ void __launch_bounds__(Shape<false>::THREADS, 1)
attn_bwd_kernel(const __grid_constant__ CUtensorMap tq, const __grid_constant__ CUtensorMap tk, const __grid_constant__ CUtensorMap tv,
                const __grid_constant__ CUtensorMap tdo, const __grid_constant__ CUtensorMap tdq, const __grid_constant__ CUtensorMap tdk,
                const __grid_constant__ CUtensorMap tdv, const Params p, int units, int mode) {
  const int ctas = (int)gridDim.x / 2, cta = (int)blockIdx.x;
  if (cta < ctas) attn_bwd_body<true>(tk, tv, tq, tdo, tdv, tdk, p, units, mode, cta, ctas);
  else attn_bwd_body<false>(tq, tdo, tk, tv, tdq, tdq, p, units, mode, cta - ctas, ctas);
}

// ------------------------------------------------------------------------------ host side
// One of Q / K / V inside qkv [B][S][3][H][64] (which = 0, 1, 2), or a plain [B][S][H][64] tensor (which = -1):
// dims {d, h, s, b}, box = cols x 1 x rows x 1 (that many rows of one head); 32 columns in the 64-byte swizzle.
static int make_map(CUtensorMap* map, const void* ptr, int B, int S, int H, int which, int rows, int cols = D) {
  EncodeTiledFn fn = encode_tiled_fn();
  if (!fn) return -10;
  const uint64_t row = (which >= 0 ? 3ull : 1ull) * H * D;          // elements between consecutive sequence positions
  const char* basep = (const char*)ptr + (which > 0 ? (size_t)which * H * D * 2 : 0);
  if ((uintptr_t)basep & 15) return -11;
  cuuint64_t dims[4] = {(cuuint64_t)D, (cuuint64_t)H, (cuuint64_t)S, (cuuint64_t)B};
  cuuint64_t strides[3] = {(cuuint64_t)D * 2, row * 2, row * 2 * (cuuint64_t)S};
  cuuint32_t box[4] = {(cuuint32_t)cols, 1, (cuuint32_t)rows, 1};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<char*>(basep), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, cols == D ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) {
    fprintf(stderr, "gcow attention: cuTensorMapEncodeTiled failed with CUresult %d (B %d S %d H %d which %d)\n", (int)r, B, S, H, which);
    return -12;
  }
  return 0;
}

constexpr size_t kFwdSmem = TILE_BYTES * 12 + sizeof(FwdBars) + 1024;   // 2 Q, 2 O, 4 K, 4 V
constexpr size_t kBwdSmem = TILE_BYTES * 13 + MAX_S * 16 + sizeof(BwdBars) + 1024;   // a1, a2 of both tiles, b1, b2, staging, statistics
static_assert(kFwdSmem <= 227 * 1024 && kBwdSmem <= 227 * 1024, "one CTA per SM");

// Two tiles per CTA share the sequence's operands, and each keeps the arithmetic units busy while the other one waits for a
// product; where there are no more tiles than SMs (dK/dV and dQ share them in the backward pass) each has an SM to itself.
static int plan_units(int B, int S, int H, int sms, int* mode, int* units) {
  const long long heads = (long long)B * H, tiles = (S + TILE - 1) / TILE;
  *mode = heads * tiles <= sms ? kSingle : tiles == 1 ? kHeads : kPair;
  const long long n = *mode == kSingle ? heads * tiles : *mode == kHeads ? (heads + 1) / 2 : heads * ((tiles + 1) / 2);
  if (n > 0x7fffffff) return -1;
  *units = (int)n;
  return 0;
}

// Up to 64 positions the 128-row tiles are mostly empty.
static int check_shape(int B, int S, int H, int d) {
  if (d != D || S % 8 || S <= 64 || S > MAX_S || B <= 0 || H <= 0 || H > 65535 || B > 65535) return -1;
  return 0;
}

static void set_attrs() {
  static std::once_flag once;
  std::call_once(once, [] {
    cudaFuncSetAttribute(attn_fwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kFwdSmem);
    cudaFuncSetAttribute(attn_bwd_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kBwdSmem);
  });
}

}  // namespace attn
}  // namespace gcow

using namespace gcow::attn;

extern "C" {

// 1 if the fused kernels cover this problem (head dimension 64, S a multiple of 8 from 72 to 512).
int gcow_attention_supported(int B, int S, int H, int d) { return check_shape(B, S, H, d) == 0; }

// out[B][S][H][64] = softmax(scale * Q K^T) V per head, qkv [B][S][3][H][64] bf16; lse [B][H][S] fp32 receives the
// log2-sum-exp of the scaled scores (kept for the backward pass). `error`: device word, set if a wait gave up.
int gcow_attention_fwd(const void* qkv, void* out, float* lse, int B, int S, int H, int d, float scale,
                       uint32_t* error, void* stream) {
  if (check_shape(B, S, H, d)) return -1;
  set_attrs();
  int mode, units, rc;
  if (plan_units(B, S, H, 148, &mode, &units)) return -1;
  CUtensorMap tq, tk, tv, to;
  if ((rc = make_map(&tq, qkv, B, S, H, 0, TILE)) || (rc = make_map(&tk, qkv, B, S, H, 1, TILE)) || (rc = make_map(&tv, qkv, B, S, H, 2, TILE)) ||
      (rc = make_map(&to, out, B, S, H, -1, 32)))
    return rc;
  Params p = {};
  p.lse = lse; p.B = B; p.S = S; p.H = H;
  p.scale = scale; p.scale_log2 = scale * 1.4426950408889634f; p.error = error;
  gcow::launch_dependent(attn_fwd_kernel, dim3(units < 148 ? units : 148), dim3(Shape<true>::THREADS), kFwdSmem, (cudaStream_t)stream, tq, tk, tv, to, p, units, mode);
  return (int)cudaGetLastError();
}

// dqkv[B][S][3][H][64] from qkv, the forward's out and lse, and dout [B][S][H][64]; delta [B][H][S] fp32 is scratch.
int gcow_attention_bwd(const void* qkv, const void* out, const void* dout, const float* lse, float* delta, void* dqkv,
                       int B, int S, int H, int d, float scale, uint32_t* error, void* stream) {
  if (check_shape(B, S, H, d)) return -1;
  set_attrs();
  cudaStream_t st = (cudaStream_t)stream;
  int mode, units, rc;
  if (plan_units(B, S, H, 148 / 2, &mode, &units)) return -1;
  CUtensorMap in[4], dq, dk, dv;                             // Q, K, V, dO
  for (int i = 0; i < 4; i++)
    if ((rc = make_map(&in[i], i < 3 ? qkv : dout, B, S, H, i < 3 ? i : -1, TILE))) return rc;
  if ((rc = make_map(&dq, dqkv, B, S, H, 0, 32, 32)) || (rc = make_map(&dk, dqkv, B, S, H, 1, 32, 32)) || (rc = make_map(&dv, dqkv, B, S, H, 2, 32, 32)))
    return rc;
  Params p = {};
  p.lse = const_cast<float*>(lse); p.delta = delta; p.B = B; p.S = S; p.H = H;
  p.scale = scale; p.scale_log2 = scale * 1.4426950408889634f; p.error = error;
  const uint32_t rows = (uint32_t)B * S * H;                 // of 128 bytes each in every tensor: far below 2^32 in any memory
  gcow::launch_dependent(attn_delta_kernel, dim3((unsigned)(((size_t)rows + 32 * kDeltaRows - 1) / (32 * kDeltaRows))), dim3(256), 0, st,
                         (const __nv_bfloat16*)out, (const __nv_bfloat16*)dout, delta, rows, (uint32_t)S, (uint32_t)H);
  gcow::launch_dependent(attn_bwd_kernel, dim3(2 * (units < 148 ? units : 148)), dim3(Shape<false>::THREADS), kBwdSmem, st, in[0], in[1], in[2], in[3],
                         dq, dk, dv, p, units, mode);
  return (int)cudaGetLastError();
}

}  // extern "C"
