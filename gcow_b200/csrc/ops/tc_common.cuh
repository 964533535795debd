// Inline-PTX building blocks shared by the tcgen05 kernels (GEMM and implicit-GEMM
// convolution): mbarrier operations with bounded waits, TMA tile loads, tcgen05
// MMA / commit / tensor-memory loads and the shared-memory matrix descriptors of
// the 128-byte-swizzled tile layouts. No load here uses cluster multicast.
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../divisor.h"

namespace gcow {
namespace tc {

constexpr uint32_t kSpinLimit = 1u << 26;   // polls before a wait gives up

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// True in one lane of the warp, which has to be converged: for what a warp issues for all of its lanes - MMAs, commits, tensor copies. Four MMAs and
// the sums for their descriptors take a warp 447 cycles behind `lane == 0` and 281 behind this (M128 N64, whose MMAs take 128). Asked once per
// role: the same lane has to issue MMAs and the commits that track them.
__device__ __forceinline__ bool elect_one() {
  uint32_t one;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.b32 %0, 1, 0, p;\n\t}" : "=r"(one));
  return one != 0;
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ uint32_t mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
  return ok;
}
// Bounded wait. Returns false when the CTA is aborting (this or another role gave up):
// after kSpinLimit polls the abort word is raised and `code` is recorded in *error.
__device__ __forceinline__ bool mbar_wait_abortable(volatile uint32_t* abort, uint64_t* bar, uint32_t parity,
                                                    uint32_t* error, uint32_t code) {
  for (uint32_t it = 0; it < kSpinLimit; it++) {
    if (mbar_try_wait(bar, parity)) return true;
    if (*abort) return false;
  }
  *abort = 1;
  atomicCAS(error, 0u, code);
  return false;
}

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int x, int y) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
               ::"r"(dst), "l"((uint64_t)map), "r"(bar), "r"(x), "r"(y) : "memory");
}

__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int x, int y, int z) {
  asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
               ::"r"(dst), "l"((uint64_t)map), "r"(bar), "r"(x), "r"(y), "r"(z) : "memory");
}
__device__ __forceinline__ void tma_load_4d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int x, int y, int z, int w) {
  asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
               ::"r"(dst), "l"((uint64_t)map), "r"(bar), "r"(x), "r"(y), "r"(z), "r"(w) : "memory");
}
__device__ __forceinline__ void tma_load_5d(uint32_t dst, const CUtensorMap* map, uint32_t bar, int x, int y, int z, int w, int v) {
  asm volatile("cp.async.bulk.tensor.5d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6, %7}], [%2];"
               ::"r"(dst), "l"((uint64_t)map), "r"(bar), "r"(x), "r"(y), "r"(z), "r"(w), "r"(v) : "memory");
}
// x = innermost coordinate, y = row coordinate, z = batch index (used only by batched launches)
__device__ __forceinline__ void tma_load(uint32_t dst, const CUtensorMap* map, uint32_t bar, int x, int y, int z, bool batched) {
  if (batched) tma_load_3d(dst, map, bar, x, y, z);
  else tma_load_2d(dst, map, bar, x, y);
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void tc_mma(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(acc) : "memory");
}
__device__ __forceinline__ void tc_ld32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tc_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// Shared-memory matrix descriptor of a K-major tile stored as rows of 128 bytes
// with the 128-byte swizzle: 8-row groups are 1024 bytes apart.
__device__ __forceinline__ uint64_t smem_desc_sw128(uint32_t saddr) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr & 0x3ffffu) >> 4);        // start address
  d |= (uint64_t)(1024u >> 4) << 32;               // stride byte offset between 8-row groups
  d |= (uint64_t)1 << 46;                          // descriptor version of this architecture
  d |= (uint64_t)2 << 61;                          // layout: 128-byte swizzle
  return d;
}

// MN-major tile: boxes of [64 K-rows][64 elements = 128 bytes], 128-byte swizzle.
// Groups of 8 K-rows are 1024 bytes apart (stride offset); the next 64 elements
// along M/N start one box (8192 bytes) later (leading offset).
__device__ __forceinline__ uint64_t smem_desc_mn_sw128(uint32_t saddr) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr & 0x3ffffu) >> 4);
  d |= (uint64_t)(8192u >> 4) << 16;
  d |= (uint64_t)(1024u >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}

// GELU for GEMM epilogues, where eight warps do the elementwise math of a whole tile and libm's erff
// (a long dependent chain) would take longer than the tile's main loop. Phi(x) = 0.5 (1 + erf(x / sqrt 2)) from
// the rational approximation erf(z) = 1 - (a1 t + ... + a5 t^5) exp(-z^2), t = 1 / (1 + p z) (Abramowitz &
// Stegun 7.1.26, absolute error below 1.5e-7); exp(-z^2) = exp(-x^2 / 2) is also what the derivative needs.
// Two elements per instruction (f32x2), constant factors folded into the coefficients, and the flushing forms of the
// reciprocal (its argument is at least 1) and of the exponential (values below 2^-126 read as 0): the other forms
// wrap each in a range test. 16384 x 4096 x 1024 product with bias and GELU: 160 -> 128 us, of 97 us without GELU.
__device__ __forceinline__ uint64_t pack2(float a, float b) {
  uint64_t r; asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b)); return r;
}
__device__ __forceinline__ void unpack2(uint64_t v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
  uint64_t r; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b)); return r;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c)); return r;
}
__device__ __forceinline__ float rcp_ftz(float x) { float r; asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x)); return r; }
__device__ __forceinline__ float ex2_ftz(float x) { float r; asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x)); return r; }
// Phi and exp(-x^2 / 2) of two values
__device__ __forceinline__ void gelu_parts2(float x0, float x1, uint64_t x, uint64_t& cdf, uint64_t& gauss) {
  constexpr float kP = 0.3275911f * 0.70710678118654752f;
  float a, b;
  unpack2(fma2(pack2(fabsf(x0), fabsf(x1)), pack2(kP, kP), pack2(1.0f, 1.0f)), a, b);
  const uint64_t t = pack2(rcp_ftz(a), rcp_ftz(b));
  constexpr float kE = -0.72134752044448170f;               // -log2(e) / 2
  unpack2(mul2(mul2(x, x), pack2(kE, kE)), a, b);
  gauss = pack2(ex2_ftz(a), ex2_ftz(b));
  uint64_t q = fma2(t, pack2(0.5f * 1.061405429f, 0.5f * 1.061405429f), pack2(0.5f * -1.453152027f, 0.5f * -1.453152027f));
  q = fma2(q, t, pack2(0.5f * 1.421413741f, 0.5f * 1.421413741f));
  q = fma2(q, t, pack2(0.5f * -0.284496736f, 0.5f * -0.284496736f));
  q = fma2(q, t, pack2(0.5f * 0.254829592f, 0.5f * 0.254829592f));
  q = mul2(mul2(q, t), gauss);
  float q0, q1;
  unpack2(q, q0, q1);
  unpack2(fma2(q, pack2(-1.0f, -1.0f), pack2(1.0f, 1.0f)), a, b);
  cdf = pack2(x0 >= 0.0f ? a : q0, x1 >= 0.0f ? b : q1);
}
// v = GELU(v)
template <int N> __device__ __forceinline__ void gelu(float (&v)[N]) {
#pragma unroll
  for (int j = 0; j < N; j += 2) {
    const uint64_t x = pack2(v[j], v[j + 1]);
    uint64_t cdf, gauss;
    gelu_parts2(v[j], v[j + 1], x, cdf, gauss);
    unpack2(mul2(x, cdf), v[j], v[j + 1]);
  }
}
// v *= d/dx of x Phi(x) = Phi(x) + x phi(x)
__device__ __forceinline__ void gelu_grad8(float* v, const float* s) {
#pragma unroll
  for (int j = 0; j < 8; j += 2) {
    const uint64_t x = pack2(s[j], s[j + 1]);
    uint64_t cdf, gauss;
    gelu_parts2(s[j], s[j + 1], x, cdf, gauss);
    const uint64_t d = fma2(mul2(x, pack2(0.3989422804014327f, 0.3989422804014327f)), gauss, cdf);
    unpack2(mul2(pack2(v[j], v[j + 1]), d), v[j], v[j + 1]);
  }
}

// Coalesced bf16 rows for epilogues. After tcgen05.ld a lane owns one row of the tile (32 consecutive columns),
// so a direct 16-byte store per lane touches 32 different rows per instruction: 32 memory transactions of 16
// useful bytes. These helpers pass the warp's 32 x 32 block through a private shared-memory buffer of 32 rows
// x 64 bytes so that four lanes cover the 64 bytes of one row and an instruction touches 8 rows: a quarter of the
// transactions, all of them whole sectors. The 16-byte chunk k of row r sits at chunk k ^ ((r >> 1) & 3), which keeps
// both access patterns free of bank conflicts without padding (the 2 KB per warp matter: with eight of them a GEMM
// CTA still leaves room on its SM for one CTA of the all-reduce kernel).
// row_off: element offset of the lane's own row start (column 0 of the block), row_ok: whether that row exists.
constexpr int kStageRowBytes = 64, kStageWarpBytes = 32 * kStageRowBytes;
__device__ __forceinline__ int stage_offset(int row, int chunk) { return row * kStageRowBytes + ((chunk ^ ((row >> 1) & 3)) << 4); }

__device__ __forceinline__ void warp_store_rows_bf16(uint8_t* stg, int lane, const float (&v)[32], __nv_bfloat16* base,
                                                     size_t row_off, bool row_ok) {
#pragma unroll
  for (int k = 0; k < 4; k++) {
    uint4 o;
    __nv_bfloat162* ob = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
    for (int e = 0; e < 4; e++) ob[e] = __floats2bfloat162_rn(v[8 * k + 2 * e], v[8 * k + 2 * e + 1]);
    *reinterpret_cast<uint4*>(stg + stage_offset(lane, k)) = o;
  }
  __syncwarp();
#pragma unroll
  for (int it = 0; it < 4; it++) {
    const int row = it * 8 + (lane >> 2), ch = lane & 3;
    const unsigned long long off = __shfl_sync(0xffffffffu, (unsigned long long)row_off, row);
    const int ok = __shfl_sync(0xffffffffu, (int)row_ok, row);
    const uint4 x = *reinterpret_cast<const uint4*>(stg + stage_offset(row, ch));
    if (ok) *reinterpret_cast<uint4*>(base + off + ch * 8) = x;
  }
  __syncwarp();
}

// A warp's 32 x 32 fp32 block, a row per lane in r, to rows `ld` floats apart from `to` on, eight lanes a row, so that every store covers whole
// 128-byte rows; `rows` of them exist. stg: 4 KB of the warp's own. A row per lane stored by its own lane is 32 lines an instruction and half
// sectors.
__device__ __forceinline__ void warp_store_rows_f32(uint8_t* stg, int lane, const uint32_t (&r)[32], float* to, size_t ld, int rows) {
  __syncwarp();
#pragma unroll
  for (int k = 0; k < 8; k++)
    *reinterpret_cast<uint4*>(stg + lane * 128 + ((k ^ (lane & 7)) << 4)) = make_uint4(r[4 * k], r[4 * k + 1], r[4 * k + 2], r[4 * k + 3]);
  __syncwarp();
#pragma unroll
  for (int it = 0; it < 8; it++) {
    const int row = it * 4 + (lane >> 3);
    const uint4 x = *reinterpret_cast<const uint4*>(stg + row * 128 + (((lane & 7) ^ (row & 7)) << 4));
    if (row < rows) *reinterpret_cast<uint4*>(to + (size_t)row * ld + (lane & 7) * 4) = x;
  }
}

// The same with 2 KB, 16 columns and four lanes a row at a time.
__device__ __forceinline__ void warp_store_rows_f32_halves(uint8_t* stg, int lane, const uint32_t (&r)[32], float* to, size_t ld, int rows) {
#pragma unroll
  for (int h = 0; h < 2; h++) {
    __syncwarp();
#pragma unroll
    for (int k = 0; k < 4; k++)
      *reinterpret_cast<uint4*>(stg + stage_offset(lane, k)) = make_uint4(r[16 * h + 4 * k], r[16 * h + 4 * k + 1], r[16 * h + 4 * k + 2], r[16 * h + 4 * k + 3]);
    __syncwarp();
#pragma unroll
    for (int it = 0; it < 4; it++) {
      const int row = it * 8 + (lane >> 2);
      const uint4 x = *reinterpret_cast<const uint4*>(stg + stage_offset(row, lane & 3));
      if (row < rows) *reinterpret_cast<uint4*>(to + (size_t)row * ld + h * 16 + (lane & 3) * 4) = x;
    }
  }
}

// Eight columns of the lane's own row of a block in the staging buffer.
__device__ __forceinline__ void own_chunk(const uint8_t* stg, int lane, int k, float (&x)[8]) {
  const uint4 y = *reinterpret_cast<const uint4*>(stg + stage_offset(lane, k));
  const __nv_bfloat162* yb = reinterpret_cast<const __nv_bfloat162*>(&y);
#pragma unroll
  for (int e = 0; e < 4; e++) {
    const float2 f = __bfloat1622float2(yb[e]);
    x[2 * e] = f.x;
    x[2 * e + 1] = f.y;
  }
}

// out[j] (+)= the lane's own row of a bf16 tensor, fetched with the same coalesced pattern
template <bool ADD>
__device__ __forceinline__ void warp_load_rows_bf16(uint8_t* stg, int lane, const __nv_bfloat16* base, size_t row_off,
                                                    bool row_ok, float (&out)[32]) {
#pragma unroll
  for (int it = 0; it < 4; it++) {
    const int row = it * 8 + (lane >> 2), ch = lane & 3;
    const unsigned long long off = __shfl_sync(0xffffffffu, (unsigned long long)row_off, row);
    const int ok = __shfl_sync(0xffffffffu, (int)row_ok, row);
    uint4 x = make_uint4(0, 0, 0, 0);
    if (ok) x = *reinterpret_cast<const uint4*>(base + off + ch * 8);
    *reinterpret_cast<uint4*>(stg + stage_offset(row, ch)) = x;
  }
  __syncwarp();
#pragma unroll
  for (int k = 0; k < 4; k++) {
    const uint4 x = *reinterpret_cast<const uint4*>(stg + stage_offset(lane, k));
    const __nv_bfloat162* xb = reinterpret_cast<const __nv_bfloat162*>(&x);
#pragma unroll
    for (int e = 0; e < 4; e++) {
      const float2 f = __bfloat1622float2(xb[e]);
      if (ADD) { out[8 * k + 2 * e] += f.x; out[8 * k + 2 * e + 1] += f.y; }
      else { out[8 * k + 2 * e] = f.x; out[8 * k + 2 * e + 1] = f.y; }
    }
  }
  __syncwarp();
}

// The order in which a persistent GEMM takes its output tiles: `group` rows of tiles together, column by column. In groups of 4 the L2 has to
// hold B and the 1024 rows of the result that are being written, and A comes from memory once; column by column it has to hold A and a
// column of the result, and B comes once. Groups are taken where A has as many rows as B or more, unless only A's share fits: it is below
// 77 MB, B's above 64 MB and above 5/4 of it. Pair kernel by itself, single launches, column by column -> groups, us (the shares in MB):
//   groups: 16384 x 4096 x 1024 101.4 -> 98.3 (42, 17), x 8192 x 1024 192.5 -> 188.9 (42, 34), x 12288 x 1024 287.7 -> 289.8 (42, 50),
//   x 16384 x 2304 917 -> 878 (84, 109), 28672 x 16384 x 1024 737 -> 700 (73, 67), 32768 x 16384 x 512 460.8 -> 455.6 (50, 50),
//   x 12288 x 768 494.6 -> 459.8 (67, 44), x 30528 x 1024 1653 -> 1604 (84, 125), x 30528 x 2048 3347 -> 3070, 65536 x 16384 x 1024 1997 -> 1635,
//   30720 x 30528 x 1024 1487 -> 1485 and, back to back, 1768 -> 1722 (79, 125);
//   columns: 16384 x 16384 x 1024 384 -> 395 (42, 67), x 2048 781 -> 788 (75, 101), 20480 x 16384 x 1024 495.6 -> 497.8 (52, 67),
//   30720 x 30528 x 768 1142 -> 1174 (63, 109), 32768 x 30528 x 768 1256 -> 1258 (67, 109).
// Back to back, under the power limit, the differences are the same or larger (16384 x 1024 x 4096 119.7 -> 99.7, 32768 x 30528 x 2048 4310 -> 3546);
// launches of different kernels in turn show other ones, since each inherits what the one before it left of the power limit. Groups of 2, 8
// and 16 are within 2 % of 4. With fewer rows than B it is A that is kept (4096 x 16384 x 4096: 406 column by column, 449 in groups).
struct TileOrder {
  int tiles_m, group, group_tiles;
  __device__ __forceinline__ void at(int tile, int& m, int& n) const {
    if (group_tiles == group) {                          // one column of tiles: 802816 x 64 x 64 60.3 -> 55.9 us, x 256 x 64 95.1 -> 87.5
      m = tile;
      n = 0;
      return;
    }
    const int g = tile / group_tiles, in = tile - g * group_tiles, first = g * group, high = min(group, tiles_m - first);
    n = in / high;
    m = first + in - n * high;
  }
};
// The same with multiplications for the two divisions, some 30 dependent instructions less, which an epilogue of sixteen warps does not cover
// (gemm2_tcgen05.cu). Not for kernels whose registers are full: the one-CTA kernel takes 99 us with it instead of 85 (802816 x 256 x 64).
struct QuickTileOrder {
  TileOrder order;
  Divisor by_group_tiles, by_group, by_last;             // by_last: the last group's rows of tiles
  __device__ __forceinline__ void at(int tile, int& m, int& n) const {
    const int g = (int)by_group_tiles.under((uint32_t)tile), in = tile - g * order.group_tiles, first = g * order.group;
    const bool last = first + order.group > order.tiles_m;
    n = (int)(last ? by_last : by_group).under((uint32_t)in);
    m = first + in - n * (last ? order.tiles_m - first : order.group);
  }
};
inline TileOrder tile_order(int M, int N, int K, int tile_m, int tile_n) {
  const double mb = 1e-6, share_a = mb * M * (2.0 * K + 512), share_b = mb * N * (2.0 * K + 2048);
  const bool groups = M >= N && !(share_a < 77 && share_b > 64 && share_b > 1.25 * share_a);
  const int tiles_m = (M + tile_m - 1) / tile_m, group = groups && tiles_m > 4 ? 4 : tiles_m;
  return {tiles_m, group, group * ((N + tile_n - 1) / tile_n)};
}
inline QuickTileOrder quick(const TileOrder& o) {
  const int rest = o.tiles_m % o.group;
  return {o, divisor(o.group_tiles), divisor(o.group), divisor(rest ? rest : o.group)};
}

// Host side: the driver's tensor-map encoder, looked up once through the runtime.
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn encode_tiled_fn();

}  // namespace tc
}  // namespace gcow
