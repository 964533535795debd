// bf16 GEMM on CTA pairs (tcgen05 cta_group::2): C[M,N] = A[M,K] * B[N,K]^T, K-major operands, fp32 accumulation in
// tensor memory, fused epilogue (bias, GELU, residual, side tensor for the GELU gradient).
//
// Two CTAs on neighbouring SMs (a cluster of 2) compute one 256 x 256 tile. CTA r loads rows r*128.. of the A tile
// and rows r*128.. of the B tile (half of each), so per flop every SM fetches two thirds of what the one-CTA
// 128 x 256 tile needs; one thread of CTA 0 issues M256 x N256 x K16 MMAs that read both CTAs' shared memory, and
// each CTA ends up with its 128 rows x 256 columns in its own tensor memory - which leaves room for two
// accumulators, so the epilogue of a tile overlaps the main loop of the next.
// A stage holds 128 K-elements: the tensor maps describe an operand as {64, rows, K/64}, so ONE 32 KB box per
// operand brings both 64-wide K chunks (a copy costs its issue and its latency besides its bytes).
//
// Signalling inside the pair (no multicast qualifier anywhere; remote barriers are addressed with mapa):
//   full[s]       lives in CTA 0; armed by CTA 0's producer with the bytes of both CTAs' copies, which both
//                 complete on it (cp.async.bulk.tensor ... .cta_group::2 with CTA 0's barrier address);
//   empty[s]      one per CTA; the MMA thread commits to its own and to the peer's, and the warps of CTA 0 that add up columns arrive on its own;
//   tmem_full[a]  one per CTA, same; tmem_empty[a] lives in CTA 0, both CTAs' epilogue threads arrive on it.
// Every wait is bounded; a CTA that gives up raises the error word, and its peer's waits then run out too.
//
// Replaces the cuBLAS GEMMs behind nn.Linear in the forward pass of the transformer models trained by the
// benchmark (no counterpart in the reference, whose GEMMs are library calls: hw/models/resenet.py:90).
#include <stdlib.h>
#include <mutex>

#include "tc_common.cuh"

namespace gcow {
namespace gemm2 {

using namespace gcow::tc;

constexpr int BM = 256, BN = 256, UMMA_K = 16;
constexpr int BK = 128;                               // K elements per stage: two 64-wide chunks
constexpr int CHUNK_BYTES = 128 * 64 * 2;             // 128 rows x 128 bytes
constexpr int OPER_BYTES = 2 * CHUNK_BYTES;           // one CTA's half of an operand, one stage
constexpr int STAGE_BYTES = 2 * OPER_BYTES;           // 64 KB
constexpr int STAGES = 3;
// What an epilogue reads besides the accumulator.
enum Side : int { kNothing = 0, kSum = 1, kArgument = 2 };      // a residual; the argument of a GELU' factor (and perhaps a residual)
// Epilogue warps: eight, or sixteen where two per scheduler leave half of the issue slots to waiting: for a GELU (bias, GELU and its argument kept, eight,
// sixteen: 16384 x 4096 x 1024 142, 129 us, x 3072 110, 97, x 1024 44, 36) and for a side operand (a residual 115, 108, with a bias 160, 119; 4096 x
// 768 x 768 11.3, 10.4 and 13.3, 11.4).
template <int SIDE, bool WIDE> struct Epilogue { static constexpr int WARPS = WIDE || SIDE ? 16 : 8, THREADS = 64 + 32 * WARPS; };
// Warps of a weight gradient that add up the columns of A as they pass through shared memory (the bias gradient).
constexpr int SUM_WARPS = 4;
template <bool A_MN, int SIDE, bool WIDE> constexpr int kThreads = Epilogue<SIDE, WIDE>::THREADS + (A_MN ? 32 * SUM_WARPS : 0);
static_assert(Epilogue<kSum, false>::THREADS == Epilogue<kArgument, false>::THREADS && Epilogue<kSum, false>::THREADS == Epilogue<kNothing, true>::THREADS, "one launch shape");
constexpr uint32_t TMEM_COLS = 512;

enum Flags : int { kBias = 2, kGelu = 4, kResidual = 8, kAuxOut = 32, kGeluGrad = 64 };

struct Params {
  __nv_bfloat16* C;        // float* of a weight gradient
  const float* bias;
  const __nv_bfloat16* residual;
  __nv_bfloat16* aux;      // float* of a weight gradient: [slices * tile columns][M] partial column sums of A, or null. (A field of their own
                           // moves the others, and the epilogues spill: 16384 x 4096 x 1024 with a bias and a residual 133 -> 137 us.)
  int M, N, K, ldc, flags;
  int whole, items;        // items of work: `whole` 256 x 256 tiles (of every slice), then halves of 256 x 128
  int slice_blocks;        // stages per slice of the reduction
  int halves;              // weight gradient, an item per pair at most: a slice's two halves have an accumulator each
  size_t slice_stride;     // elements from one slice's result to the next
  QuickTileOrder order;
  uint32_t* error;
};

// An item of work: a tile, or the left or right half of one, over a slice of the reduction.
struct Item { int m0, n0, kb0, kb1, slice; bool half; };
// Which half of a tile's rows a CTA of the pair takes: its own, in a weight gradient's odd tile columns the other one (see the column sums).
template <bool A_MN> __device__ __forceinline__ int half_of(const Item& it, uint32_t rank) { return (int)rank ^ (A_MN ? it.n0 / BN & 1 : 0); }
template <bool SLICES> __device__ __forceinline__ Item item_at(const Params& p, int i, int tiles, int kblocks) {
  Item r;
  r.half = i >= p.whole;
  const int j = r.half ? (i - p.whole) >> 1 : i;
  r.slice = SLICES ? j / tiles : 0;
  const int tile = r.half ? p.whole + j : j - r.slice * tiles;
  p.order.at(tile, r.m0, r.n0);
  r.m0 *= BM;
  r.n0 = r.n0 * BN + (r.half ? ((i - p.whole) & 1) * (BN / 2) : 0);
  r.kb0 = SLICES ? r.slice * p.slice_blocks : 0;
  r.kb1 = SLICES && r.kb0 + p.slice_blocks < kblocks ? r.kb0 + p.slice_blocks : kblocks;
  return r;
}

__device__ __forceinline__ void tc_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tma_store_2d(const CUtensorMap* map, const uint8_t* from, int x, int y) {   // rows past the end are clipped
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];"
               ::"l"((uint64_t)map), "r"(smem_u32(from)), "r"(x), "r"(y) : "memory");
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}
__device__ __forceinline__ uint4 pack8(const float (&v)[8]) {
  uint4 o;
  __nv_bfloat162* const b = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
  for (int e = 0; e < 4; e++) b[e] = __floats2bfloat162_rn(v[2 * e], v[2 * e + 1]);
  return o;
}
__device__ __forceinline__ void add8(float (&v)[8], const uint4& x) {
  const __nv_bfloat162* const b = reinterpret_cast<const __nv_bfloat162*>(&x);
#pragma unroll
  for (int e = 0; e < 4; e++) { const float2 f = __bfloat1622float2(b[e]); v[2 * e] += f.x; v[2 * e + 1] += f.y; }
}

struct Smem {
  uint64_t full[STAGES], empty[STAGES], tmem_full[2], tmem_empty[2], drain, side[16];
  uint32_t tmem_base;
  volatile uint32_t abort;
};

__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t map_to_cta(uint32_t saddr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(saddr), "r"(rank));
  return r;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// the copy lands in this CTA's shared memory; its bytes complete on the barrier at cluster address `bar`
__device__ __forceinline__ void tma_load_3d_pair(uint32_t dst, const CUtensorMap* map, uint32_t bar, int x, int y, int z) {
  asm volatile("cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
               ::"r"(dst), "l"((uint64_t)map), "r"(bar), "r"(x), "r"(y), "r"(z) : "memory");
}
__device__ __forceinline__ void tc_commit_pair(uint32_t bar_cluster_addr) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar_cluster_addr) : "memory");
}
__device__ __forceinline__ void tc_mma_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(acc) : "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t bar_cluster_addr) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(bar_cluster_addr) : "memory");
}

// MN-major operand tile fetched as ONE box {64 columns, 128 K-rows, 2 column groups}: each 64-column group is
// 128 K-rows x 128 bytes = 16 KB, so groups are 16 KB apart (leading offset) and 8-row groups 1 KB (stride offset).
__device__ __forceinline__ uint64_t smem_desc_mn_sw128_16k(uint32_t saddr) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr & 0x3ffffu) >> 4);
  d |= (uint64_t)(16384u >> 4) << 16;
  d |= (uint64_t)(1024u >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}

// B_MN: B is stored [K][N] (the data-gradient product dX = dY * W reads the weight matrix in place); A_MN: A is stored [K][M]
// (with B_MN the weight gradient, which reads both in place). SIDE: what the epilogue reads.
template <bool A_MN, bool B_MN, int SIDE, bool WIDE>
__global__ void __launch_bounds__((kThreads<A_MN, SIDE, WIDE>), 1)
gemm2_bf16_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                  const __grid_constant__ CUtensorMap tmap_bh, const Params p, const __grid_constant__ CUtensorMap tmap_side,
                  const __grid_constant__ CUtensorMap tmap_c) {
  constexpr int EPI_WARPS = Epilogue<SIDE, WIDE>::WARPS;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* base = reinterpret_cast<uint8_t*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  Smem* sm = reinterpret_cast<Smem*>(base + STAGES * STAGE_BYTES);
  uint8_t* stage_base = reinterpret_cast<uint8_t*>(((uintptr_t)(sm + 1) + 511) & ~(uintptr_t)511);

  const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;   // warp: uniform
  const uint32_t rank = cluster_rank();               // 0: issues the MMAs and owns full / tmem_empty
  const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
  const int tiles_m = (p.M + BM - 1) / BM, tiles_n = (p.N + BN - 1) / BN;
  const int tiles = tiles_m * tiles_n;
  const int kblocks = (p.K + BK - 1) / BK;

  if (threadIdx.x == 0) {
    const uint32_t readers = A_MN && p.aux && rank == 0 ? 1 + SUM_WARPS : 1;
    for (int s = 0; s < STAGES; s++) { mbar_init(&sm->full[s], 1); mbar_init(&sm->empty[s], readers); }
    for (int a = 0; a < 2; a++) { mbar_init(&sm->tmem_full[a], 1); mbar_init(&sm->tmem_empty[a], 2 * EPI_WARPS * 32); }
    mbar_init(&sm->drain, 1);
    if (SIDE) for (int w = 0; w < EPI_WARPS; w++) mbar_init(&sm->side[w], 1);
    sm->abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sm->tmem_base)), "r"(TMEM_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync();            // both CTAs' barriers are initialised before either signals the other
  tc_fence_after();
  const uint32_t tmem_base = sm->tmem_base;
  // programmatic dependent launch: the next kernel of the stream may set itself up from here on, and this one, when
  // launched the same way, has set itself up under the tail of its predecessor; global memory only after that
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer (both CTAs)
    if (elect_one()) {
      uint32_t s = 0, phase = 0;
      bool ok = true;
      for (int i = pair; i < p.items && ok; i += pairs) {
        const Item it = item_at<A_MN>(p, i, tiles, kblocks);
        const int m0 = it.m0 + half_of<A_MN>(it, rank) * 128, n0 = it.n0 + (int)rank * (it.half ? 64 : 128);
        const CUtensorMap* const map_b = it.half ? &tmap_bh : &tmap_b;
        for (int kb = it.kb0; kb < it.kb1; kb++) {
          if (!(ok = mbar_wait_abortable(&sm->abort, &sm->empty[s], phase ^ 1, p.error, 1))) break;
          if (rank == 0) mbar_expect_tx(&sm->full[s], 2 * (it.half ? OPER_BYTES + OPER_BYTES / 2 : STAGE_BYTES));
          const uint32_t bar = map_to_cta(smem_u32(&sm->full[s]), 0);
          uint8_t* st = base + s * STAGE_BYTES;
          if (A_MN) tma_load_3d_pair(smem_u32(st), &tmap_a, bar, 0, kb * BK, m0 / 64);
          else tma_load_3d_pair(smem_u32(st), &tmap_a, bar, 0, m0, kb * 2);
          if (B_MN) tma_load_3d_pair(smem_u32(st + OPER_BYTES), map_b, bar, 0, kb * BK, n0 / 64);
          else tma_load_3d_pair(smem_u32(st + OPER_BYTES), map_b, bar, 0, n0, kb * 2);
          if (++s == STAGES) { s = 0; phase ^= 1; }
        }
      }
      if (!ok) {
        // giving up: let copies already in flight land before the CTA's shared memory is released
        for (int i = 0; i < 1000; i++) __nanosleep(1000);
      }
    }
  } else if (warp == 1) {
    // -------------------------------------------------------------- MMA issuer (CTA 0 only)
    if (rank == 0) {                                    // the warp keeps together, so that every operand is uniform; one lane issues
      const bool one = elect_one();
      // instruction descriptor: fp32 accumulate, bf16 x bf16, operand major-ness, M 256 (128 rows per CTA), N 256 or 128
      const uint32_t idesc0 = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)A_MN << 15) | ((uint32_t)B_MN << 16) | ((uint32_t)(BM >> 4) << 24);
      uint32_t s = 0, phase = 0, t = 0;
      bool ok = true;
      auto wait = [&](uint64_t* bar, uint32_t parity, uint32_t code) {
        return __all_sync(0xffffffffu, mbar_wait_abortable(&sm->abort, bar, parity, p.error, code)) != 0;
      };
      for (int i = pair; i < p.items && ok; i += pairs, t++) {
        const Item it = item_at<A_MN>(p, i, tiles, kblocks);
        const uint32_t idesc = idesc0 | ((uint32_t)((it.half ? BN / 2 : BN) >> 3) << 17), chunk_b = it.half ? CHUNK_BYTES / 2 : CHUNK_BYTES;
        const uint32_t acc = t & 1, aphase = (t >> 1) & 1;
        if (!(ok = wait(&sm->tmem_empty[acc], aphase ^ 1, 2))) break;
        tc_fence_after();
        const int second = A_MN && p.halves ? (it.kb0 + it.kb1 + 1) / 2 : it.kb1;    // from this stage on in the other accumulator
        for (int kb = it.kb0; kb < it.kb1; kb++) {
          if (!(ok = wait(&sm->full[s], phase, 3))) break;
          tc_fence_after();
          const uint32_t d_tmem = tmem_base + acc * BN + (A_MN && kb >= second ? BN : 0);
          const uint32_t sa = smem_u32(base + s * STAGE_BYTES), sb = sa + OPER_BYTES;
          const uint32_t eb0 = map_to_cta(smem_u32(&sm->empty[s]), 0), eb1 = map_to_cta(smem_u32(&sm->empty[s]), 1);
          if (one) {
#pragma unroll
            for (int k = 0; k < BK / UMMA_K; k++) {
              const uint32_t in = (k & 3) * 32;                               // 64-wide chunk, then 32 bytes per K step
              // MN-major: 16 K-rows of 128 bytes per step, 128 rows contiguous within a column group
              const uint64_t da = A_MN ? smem_desc_mn_sw128_16k(sa + k * 2048) : smem_desc_sw128(sa + (k >> 2) * CHUNK_BYTES + in);
              const uint64_t db = B_MN ? smem_desc_mn_sw128_16k(sb + k * 2048) : smem_desc_sw128(sb + (k >> 2) * chunk_b + in);
              tc_mma_pair(d_tmem, da, db, idesc, (kb != it.kb0 && (!A_MN || kb != second)) || k);
            }
            tc_commit_pair(eb0);
            tc_commit_pair(eb1);
          }
          __syncwarp();
          if (++s == STAGES) { s = 0; phase ^= 1; }
        }
        if (ok && one) {
          const uint32_t fb = smem_u32(&sm->tmem_full[acc]);
          tc_commit_pair(map_to_cta(fb, 0));
          tc_commit_pair(map_to_cta(fb, 1));
        }
        __syncwarp();
      }
      // drain: everything issued by this thread has finished before tensor memory is freed
      if (one) {
        tc_commit_pair(map_to_cta(smem_u32(&sm->drain), 0));
        for (uint32_t it = 0; it < kSpinLimit; it++) if (mbar_try_wait(&sm->drain, 0)) break;
      }
    }
  } else if (A_MN && warp >= 2 + EPI_WARPS) {
    // ------------------------------------------------- column sums of A (CTA 0), where they are wanted
    // Ordinary loads may read what this CTA's own copies brought once full[s], which lives here, has completed. CTA 1 would need its copies' completion
    // passed on, with a release and an acquire at cluster scope per stage: a BERT layer 1650 us instead of 1520, and in the MMA warp's loop
    // 1930. So CTA 0 adds up alone. The tiles of one row have the same two halves of A in shared memory; in even tile columns CTA 0 takes the first, in
    // odd ones the second, and either half's stages are shared by the columns of its parity: of `sharing` columns the j-th takes every
    // sharing-th group of four rows, in turn by two pairs of warps. A warp takes 64 columns, a lane 8 of them in one row of each group, which come
    // from two of a row's 16-byte chunks in turn (128-byte swizzle). It adds up 16 rows or a few more, up to four such sums, and those, so that no
    // chain is long.
    // A stage's MMAs take longer than a share of its sums, so hardly anything waits for these. The product alone, with the column sums as kernels of
    // their own, with these, us, each with its ordered sums: 16384 rows to 3072 x 1024 80.9, 103.4, 79.0; to 4096 x 1024 96.1, 122.2, 97.1; to 768 x 768 29.9, 40.6,
    // 30.8; 1024 rows to 768 x 768 12.4, 15.6, 12.8; 50176 to 512 x 512, where one tile column has all groups of a half, 31.5, 57.9, 35.8. Whole stages in turn
    // instead of groups of rows held a stage for longer than its MMAs (16384 rows to 4096 x 1024 122). Both CTAs adding up for themselves, with the
    // order between them left to chance, took 98.3 there and 29.7 for 768 x 768.
    if (rank == 0 && p.aux) {
      const int w = (warp - 2 - EPI_WARPS) & 1, turn = (warp - 2 - EPI_WARPS) >> 1, row = lane >> 3, chunk = lane & 7;
      const uint8_t* const mine = base + w * 16384 + row * 128;
      const int even = (chunk ^ row) * 16, odd = 512 + (chunk ^ (row + 4)) * 16;
      uint32_t s = 0, phase = 0;
      bool ok = true;
      for (int i = pair; i < p.items && ok; i += pairs) {
        const Item it = item_at<A_MN>(p, i, tiles, kblocks);
        const int column = it.n0 / BN, sharing = (tiles_n + 1 - (column & 1)) / 2, first = (column >> 1) + sharing * turn;
        int rows = 0, held = 0;
        float sum[8] = {}, some[8] = {}, v[8] = {};
        for (int kb = it.kb0; kb < it.kb1; kb++) {
          ok = __all_sync(0xffffffffu, mbar_wait_abortable(&sm->abort, &sm->full[s], phase, p.error, 5)) != 0;
          if (!ok) break;
          const uint8_t* const at = mine + s * STAGE_BYTES;
#pragma unroll 4
          for (int r = first; r < 32; r += 2 * sharing) {
            const uint4 x = *reinterpret_cast<const uint4*>(at + (r >> 1) * 1024 + (r & 1 ? odd : even));
            const uint32_t y[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
            for (int j = 0; j < 4; j++) { v[2 * j] += __uint_as_float(y[j] << 16); v[2 * j + 1] += __uint_as_float(y[j] & 0xffff0000u); }
            rows++;
          }
          __syncwarp();
          if (lane == 0) mbar_arrive(&sm->empty[s]);
          if (rows >= 16) {
#pragma unroll
            for (int j = 0; j < 8; j++) { some[j] += v[j]; v[j] = 0.0f; }
            rows = 0;
            if (++held == 4) {
#pragma unroll
              for (int j = 0; j < 8; j++) { sum[j] += some[j]; some[j] = 0.0f; }
              held = 0;
            }
          }
          if (++s == STAGES) { s = 0; phase ^= 1; }
        }
        if (!ok) break;
#pragma unroll
        for (int j = 0; j < 8; j++) {
          sum[j] += some[j] + v[j];
#pragma unroll
          for (int d = 8; d < 32; d *= 2) sum[j] += __shfl_xor_sync(0xffffffffu, sum[j], d);
        }
        // Two partial sums of a half per two tile columns. Behind the last of an odd number of columns nobody has the second half's: zeros.
        const bool alone = column + 1 == tiles_n && !(column & 1);
        const int m = it.m0 + half_of<A_MN>(it, 0) * 128 + w * 64 + chunk * 8;
        float* const to = reinterpret_cast<float*>(p.aux) + (size_t)(it.slice * ((tiles_n + 1) & ~1) + (column & ~1) + turn) * p.M + m;
        if (lane < 8 && m < p.M) {                            // M is a multiple of 64
          *reinterpret_cast<float4*>(to) = make_float4(sum[0], sum[1], sum[2], sum[3]);
          *reinterpret_cast<float4*>(to + 4) = make_float4(sum[4], sum[5], sum[6], sum[7]);
        }
        if (alone && lane < 8 && m + 128 < p.M)
          *reinterpret_cast<float4*>(to + 128) = *reinterpret_cast<float4*>(to + 132) = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      }
    }
  } else {
    // ----------------------------------------------------------------- epilogue (both CTAs, own 128 rows)
    const int q = warp & 3, ew = warp - 2;
    constexpr int GROUPS = EPI_WARPS / 4;               // of columns
    const bool wide_bias = ((uintptr_t)p.bias & 15) == 0;
    uint8_t* stg = stage_base + ew * kStageWarpBytes;
    uint32_t t = 0;
    bool ok = true;
    // What the epilogue reads besides the accumulator comes by the TMA, a warp's 32 x 32 block into its staging buffer, where each lane takes its row
    // and puts the result's in its place, from where the TMA fetches it. The next block, or the next tile's first one, is asked for as soon as the
    // buffer has been read, so it comes under the wait for the accumulator. Bound by a warp's chain of block, arithmetic and store, four to a
    // scheduler. Read by the lanes themselves a block ahead, which left registers for eight warps (twelve for a GELU' factor), and written by
    // them, us, now: 16384 x 4096 x 1024 with a residual 115, 110, and a bias 135, 113, GELU' 155, 122, and a residual 240, 147; 16384 x 1024 x 1024 32.7,
    // 31.0, 38.7, 33.2, 42.1, 35.8, 53.8, 39.7; 4096 x 768 x 768 11.1, 10.4, 12.1, 11.2, 13.9, 12.3, 16.6, 12.7. The results are the same bits.
    [[maybe_unused]] uint32_t side_phase = 0;
    [[maybe_unused]] bool side_due = false;               // the block asked for has not been waited for
    [[maybe_unused]] const bool one = elect_one();
    [[maybe_unused]] auto ask = [&](int row0, int n) {    // where there is no such block, nobody will wait for it
      if (n >= p.N || row0 >= p.M) return;
      if (one) {
        mbar_expect_tx(&sm->side[ew], kStageWarpBytes);
        tma_load_2d(smem_u32(stg), &tmap_side, smem_u32(&sm->side[ew]), n, row0);
      }
      side_due = true;
    };
    [[maybe_unused]] auto ask_first = [&](int i) {
      if (i >= p.items) return;
      const Item it = item_at<A_MN>(p, i, tiles, kblocks);
      ask(it.m0 + half_of<A_MN>(it, rank) * 128 + q * 32, it.n0 + (ew / 4) * ((it.half ? BN / 2 : BN) / GROUPS));
    };
    if (SIDE) ask_first(pair);
    // A warp's 32 x 32 results to the matrix of `map`, through the staging buffer that the last store but one (sixteen warps: the last one) has left.
    // Two passes over the buffer and the lanes' own stores took, us, now: bias, GELU and its argument kept 16384 x 4096 x 1024 142, 124, x 1024 x 1024 38.4,
    // 33.4, x 512 x 512 18.8, 15.1, 4096 x 768 x 768 13.7, 11.6, bias and GELU 118, 109, 33.7, 30.7, 15.6, 14.1, 12.4, 11.5, a bias 97.9, 93.7, 29.4, 27.1, 13.7,
    // 11.3, 11.0, 9.8, plain 106, 105, 28.2, 27.9, 11.3, 10.3, 9.6, 8.8. Sixteen warps with one block of the accumulator each: GELU 116, 124; without
    // a GELU sixteen warps instead of eight and two buffers: bias 112, 122.
    constexpr int BUFFERS = WIDE ? 1 : 2;
    [[maybe_unused]] int buffer = 0;
    [[maybe_unused]] auto emit = [&](const float (&v)[32], const CUtensorMap* map, int n, int row0) {
      uint8_t* const to = stage_base + (ew * BUFFERS + buffer) * kStageWarpBytes;
      if (one) asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(BUFFERS - 1) : "memory");
      __syncwarp();
#pragma unroll
      for (int k = 0; k < 4; k++) {
        float u[8];
#pragma unroll
        for (int e = 0; e < 8; e++) u[e] = v[8 * k + e];
        *reinterpret_cast<uint4*>(to + stage_offset(lane, k)) = pack8(u);
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (one) tma_store_2d(map, to, n, row0);
      if (BUFFERS == 2) buffer ^= 1;
    };
    // The next item's place is worked out before this one's wait. A GELU after 4096 x 768 x 768 12.7 -> 12.4 us (12.2 before the tiles came in
    // groups), 16384 x 512 x 512 16.4 -> 15.7 (15.5), 8192 x 3072 x 768 38.2 -> 37.3 (37.5).
    Item next = item_at<A_MN>(p, pair, tiles, kblocks);
    for (int i = pair; i < p.items && ok; i += pairs, t++) {
      const Item it = next;
      if (i + pairs < p.items) next = item_at<A_MN>(p, i + pairs, tiles, kblocks);
      const int m0 = it.m0 + half_of<A_MN>(it, rank) * 128, n0 = it.n0;
      // this warp's
      const int cols = (it.half ? BN / 2 : BN) / GROUPS, chunks = cols / 32, col0 = (ew / 4) * cols;
      const uint32_t acc = t & 1, aphase = (t >> 1) & 1;
      const int mw = m0 + q * 32;                         // the warp's first row
      ok = mbar_wait_abortable(&sm->abort, &sm->tmem_full[acc], aphase, p.error, 4);
      ok = __all_sync(0xffffffffu, ok);   // the tensor-memory loads below need the whole warp
      if (!ok) break;
      tc_fence_after();
      const int m = m0 + q * 32 + lane;
      const bool row_ok = m < p.M;
      const uint32_t taddr = tmem_base + ((uint32_t)(q * 32) << 16) + acc * BN + col0;
      auto process = [&](const uint32_t (&r)[32], int c) {
        const int n = n0 + col0 + c * 32;
        if (n >= p.N || mw >= p.M) return;                // warp-uniform; the launcher guarantees N % 32 == 0
        float v[32];
#pragma unroll
        for (int j = 0; j < 32; j++) v[j] = __uint_as_float(r[j]);
        if constexpr (A_MN) {                              // a weight gradient, fp32
          if (p.halves && it.kb1 - it.kb0 > 1) {
            uint32_t other[32];
            tc_ld32(taddr + BN + c * 32, other);
            tc_wait_ld();
#pragma unroll
            for (int j = 0; j < 32; j++) v[j] += __uint_as_float(other[j]);
          }
          uint32_t o[32];
#pragma unroll
          for (int j = 0; j < 32; j++) o[j] = __float_as_uint(v[j]);
          warp_store_rows_f32(stage_base + ew * 4096, lane, o, reinterpret_cast<float*>(p.C) + it.slice * p.slice_stride + (size_t)mw * p.ldc + n, p.ldc,
                              p.M - mw);
          return;
        }
        if (p.flags & kBias) {
          if (wide_bias) {                                 // n is a multiple of 32
#pragma unroll
            for (int j = 0; j < 32; j += 4) {
              const float4 b = *reinterpret_cast<const float4*>(p.bias + n + j);
              v[j] += b.x; v[j + 1] += b.y; v[j + 2] += b.z; v[j + 3] += b.w;
            }
          } else {
#pragma unroll
            for (int j = 0; j < 32; j++) v[j] += p.bias[n + j];
          }
        }
        if (p.flags & kAuxOut) emit(v, &tmap_side, n, mw);
        if (p.flags & kGelu) gelu(v);                    // not together with kGeluGrad
        emit(v, &tmap_c, n, mw);
      };
      if constexpr (SIDE != kNothing) {
#pragma unroll 1
        for (int c = 0; c < chunks; c++) {
          const int n = n0 + col0 + c * 32;
          if (n < p.N && mw < p.M) {                       // warp-uniform; the launcher guarantees N % 32 == 0
            ok = mbar_wait_abortable(&sm->abort, &sm->side[ew], side_phase, p.error, 5);
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            side_phase ^= 1;
            side_due = false;
            const size_t off = (size_t)m * p.ldc + n;
#pragma unroll
            for (int h = 0; h < 2; h++) {
              uint32_t r[16];
              uint4 res[2] = {};
              if (SIDE == kArgument && (p.flags & kResidual) && row_ok)   // the buffer holds the argument: a lane reads its own row
#pragma unroll
                for (int k = 0; k < 2; k++) res[k] = *reinterpret_cast<const uint4*>(p.residual + off + h * 16 + k * 8);
              tc_ld16(taddr + c * 32 + h * 16, r);
              float bias[16];                              // a residual: under the wait for the accumulator; no registers for it with a GELU' factor
              auto add_bias = [&](float* to, int from) {   // eight columns
                if (wide_bias) {                           // n is a multiple of 32
#pragma unroll
                  for (int e = 0; e < 8; e += 4) {
                    const float4 b = *reinterpret_cast<const float4*>(p.bias + from + e);
                    to[e] += b.x; to[e + 1] += b.y; to[e + 2] += b.z; to[e + 3] += b.w;
                  }
                } else {
#pragma unroll
                  for (int e = 0; e < 8; e++) to[e] += p.bias[from + e];
                }
              };
              if constexpr (SIDE == kSum) {
#pragma unroll
                for (int e = 0; e < 16; e++) bias[e] = -0.0f;   // added to anything leaves it as it is
                if (p.flags & kBias) {
                  add_bias(bias, n + h * 16);
                  add_bias(bias + 8, n + h * 16 + 8);
                }
              }
              tc_wait_ld();
#pragma unroll
              for (int k = 0; k < 2; k++) {
                const int e0 = h * 16 + k * 8;
                float v[8], x[8];
#pragma unroll
                for (int e = 0; e < 8; e++) v[e] = SIDE == kSum ? __uint_as_float(r[8 * k + e]) + bias[8 * k + e] : __uint_as_float(r[8 * k + e]);
                if (SIDE == kArgument && (p.flags & kBias)) add_bias(v, n + e0);
                own_chunk(stg, lane, 2 * h + k, x);
                if ((p.flags & kAuxOut) && row_ok) *reinterpret_cast<uint4*>(p.aux + off + e0) = pack8(v);
                if constexpr (SIDE == kArgument) {
                  gelu_grad8(v, x);
                  if (p.flags & kResidual) add8(v, res[k]);
                } else {
                  if (p.flags & kGelu) gelu(v);
#pragma unroll
                  for (int e = 0; e < 8; e++) v[e] += x[e];
                }
                *reinterpret_cast<uint4*>(stg + stage_offset(lane, 2 * h + k)) = pack8(v);
              }
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (one) {
              tma_store_2d(&tmap_c, stg, n, mw);
              asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
            }
          }
          if (c + 1 < chunks) ask(mw, n + 32); else ask_first(i + pairs);
          __syncwarp();
        }
        if (!ok) break;
        tc_fence_before();
        mbar_arrive_cluster(map_to_cta(smem_u32(&sm->tmem_empty[acc]), 0));
        continue;
      }
      // tensor-memory loads one block ahead of the arithmetic (sixteen warps hide them from one another)
      uint32_t ra[32];
      tc_ld32(taddr, ra);
      uint32_t rb[32];
#pragma unroll 1
      for (int c = 0; c < chunks; c += 2) {
        tc_wait_ld();
        if (!WIDE && c + 1 < chunks) tc_ld32(taddr + (c + 1) * 32, rb);
        process(ra, c);
        if (c + 1 < chunks) {
          if (WIDE) tc_ld32(taddr + (c + 1) * 32, rb);
          tc_wait_ld();
          if (!WIDE && c + 2 < chunks) tc_ld32(taddr + (c + 2) * 32, ra);
          process(rb, c + 1);
        }
      }
      // this CTA's half of the accumulator has been read out: tell the MMA thread in CTA 0
      tc_fence_before();
      mbar_arrive_cluster(map_to_cta(smem_u32(&sm->tmem_empty[acc]), 0));
    }
    if (!A_MN) {                                           // nothing may be in flight when the CTA ends
      if (side_due)
        for (uint32_t it = 0; it < kSpinLimit; it++) if (mbar_try_wait(&sm->side[ew], side_phase)) break;
      if (one) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    }
  }

  __syncwarp();
  tc_fence_before();
  __syncthreads();
  cluster_sync();            // the peer no longer reads this CTA's shared memory or signals its barriers
  if (warp == 1) {
    __syncwarp();
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(TMEM_COLS) : "memory");
  }
}

// K-major matrix [rows][K] (K a multiple of 64) as {64, rows, K / 64}; box = 64 x 128 rows x 2 chunks (32 KB; half a tile: 64 rows).
static int make_map_kfold(CUtensorMap* map, const void* ptr, uint64_t rows, uint64_t K, uint64_t ld, uint32_t box_rows = 128) {
  EncodeTiledFn fn = encode_tiled_fn();
  if (!fn) return -10;
  if (((uintptr_t)ptr & 15) || (ld * 2) % 16 || K % 64) return -11;
  cuuint64_t dims[3] = {64, rows, K / 64};
  cuuint64_t strides[2] = {ld * 2, 128};
  cuuint32_t box[3] = {64, box_rows, 2};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(ptr), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : -12;
}

// MN-major matrix [K][cols] (cols a multiple of 64) as {64, K, cols / 64}; box = 64 x 128 K-rows x 2 column groups (32 KB; half a tile: one).
static int make_map_mnfold(CUtensorMap* map, const void* ptr, uint64_t K, uint64_t cols, uint64_t ld, uint32_t groups = 2) {
  EncodeTiledFn fn = encode_tiled_fn();
  if (!fn) return -10;
  if (((uintptr_t)ptr & 15) || (ld * 2) % 16 || cols % 64) return -11;
  cuuint64_t dims[3] = {64, K, cols / 64};
  cuuint64_t strides[2] = {ld * 2, 128};
  cuuint32_t box[3] = {64, 128, groups};
  cuuint32_t estr[3] = {1, 1, 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(ptr), dims, strides, box, estr,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : -12;
}

// Row-major matrix [rows][cols] in blocks of 32 x 32 (64-byte rows, the staging buffers' swizzle).
static int make_map_blocks(CUtensorMap* map, const void* ptr, uint64_t rows, uint64_t cols, uint64_t ld) {
  EncodeTiledFn fn = encode_tiled_fn();
  if (!fn) return -10;
  if (((uintptr_t)ptr & 15) || (ld * 2) % 16 || cols % 32) return -11;
  cuuint64_t dims[2] = {cols, rows};
  cuuint64_t strides[1] = {ld * 2};
  cuuint32_t box[2] = {32, 32};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : -12;
}

using KernelFn = void (*)(CUtensorMap, CUtensorMap, CUtensorMap, Params, CUtensorMap, CUtensorMap);
static_assert(sizeof(Smem) <= 512, "the staging buffers begin 512 bytes behind the operands");
constexpr size_t kSmemBytes = (size_t)STAGES * STAGE_BYTES + 512 + (size_t)Epilogue<kNothing, true>::WARPS * kStageWarpBytes + 1024;

static KernelFn pick(bool b_mn, int side, bool wide) {
  if (side == kArgument) return b_mn ? gemm2_bf16_kernel<false, true, kArgument, false> : gemm2_bf16_kernel<false, false, kArgument, false>;
  if (side == kSum) return b_mn ? gemm2_bf16_kernel<false, true, kSum, false> : gemm2_bf16_kernel<false, false, kSum, false>;
  if (wide) return b_mn ? gemm2_bf16_kernel<false, true, kNothing, true> : gemm2_bf16_kernel<false, false, kNothing, true>;
  return b_mn ? gemm2_bf16_kernel<false, true, kNothing, false> : gemm2_bf16_kernel<false, false, kNothing, false>;
}

static int launch(KernelFn kernel, int threads, int max_pairs, const CUtensorMap& ma, const CUtensorMap& mb, const CUtensorMap& mh,
                  const Params& p, const CUtensorMap& side, const CUtensorMap& mc, void* stream) {
  const int pairs = p.items < max_pairs ? p.items : max_pairs;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2 * pairs, 1, 1);
  cfg.blockDim = dim3(threads, 1, 1);
  cfg.dynamicSmemBytes = kSmemBytes;
  cfg.stream = (cudaStream_t)stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  static const bool pdl = [] { const char* e = getenv("GCOW_PDL"); return !(e && e[0] == '0'); }();
  cfg.attrs = attr; cfg.numAttrs = pdl ? 2 : 1;
  return (int)cudaLaunchKernelEx(&cfg, kernel, ma, mb, mh, p, side, mc);
}

}  // namespace gemm2
}  // namespace gcow

using namespace gcow::gemm2;

extern "C" {

// Number of CTA pairs that can run at once on the current device (0: cluster launches are not possible).
int gcow_gemm2_max_pairs() {
  static std::once_flag once;
  static int pairs = 0;
  std::call_once(once, [] {
    for (const KernelFn kernel : {pick(false, kNothing, false), pick(false, kNothing, true), pick(false, kSum, false), pick(false, kArgument, false),
                                  pick(true, kNothing, false), pick(true, kNothing, true), pick(true, kSum, false), pick(true, kArgument, false),
                                  (KernelFn)gemm2_bf16_kernel<true, true, kNothing, false>}) {
      if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBytes) != cudaSuccess) {
        cudaGetLastError();
        return;
      }
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2, 1, 1);
    cfg.blockDim = dim3(Epilogue<kNothing, true>::THREADS, 1, 1);
    cfg.dynamicSmemBytes = kSmemBytes;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = 2; attr.val.clusterDim.y = 1; attr.val.clusterDim.z = 1;
    cfg.attrs = &attr; cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, gemm2_bf16_kernel<false, false, kNothing, true>, &cfg) == cudaSuccess) pairs = n;
    else cudaGetLastError();
  });
  return pairs;
}

// C[M,N] = A[M,K] * op(B) (+ bias) (GELU) (+ residual), bf16 in and out, on CTA pairs. A is K-major [M][K]; B is
// [N][K] (b_mn == 0) or [K][N] (b_mn == 1, N a multiple of 64).
// K a multiple of 64, N a multiple of 32, lda/ldb/ldc multiples of 8, 16-byte aligned bases.
// flags as gcow_gemm_bf16 (2 bias, 4 GELU, 8 residual, 32 aux receives the pre-GELU value, 64 multiply by GELU'(aux)).
// Returns 0, a negative argument error (-2: not supported here, use the one-CTA kernel) or a CUDA error code.
int gcow_gemm2_bf16(const void* A, const void* B, void* C, int M, int N, int K, int lda, int ldb, int ldc,
                    const float* bias, const void* residual, void* aux, int flags, uint32_t* error, int b_mn, void* stream) {
  if (M <= 0 || N <= 0 || K <= 0) return 0;
  if (K % 64 || N % 32 || lda % 8 || ldb % 8 || ldc % 8 || ((uintptr_t)C & 15) || (b_mn && N % 64)) return -2;
  if (flags & ~(kBias | kGelu | kResidual | kAuxOut | kGeluGrad) || ((flags & kGelu) && (flags & kGeluGrad))) return -2;
  if ((flags & kBias) && !bias) return -1;
  if ((flags & kResidual) && (!residual || ((uintptr_t)residual & 15))) return -1;
  if ((flags & (kAuxOut | kGeluGrad)) && (!aux || ((uintptr_t)aux & 15))) return -1;
  const int max_pairs = gcow_gemm2_max_pairs();
  if (max_pairs <= 0) return -2;
  CUtensorMap ma, mb;
  int rc = make_map_kfold(&ma, A, (uint64_t)M, (uint64_t)K, (uint64_t)lda);
  if (rc) return rc;
  rc = b_mn ? make_map_mnfold(&mb, B, (uint64_t)K, (uint64_t)N, (uint64_t)ldb)
            : make_map_kfold(&mb, B, (uint64_t)N, (uint64_t)K, (uint64_t)ldb);
  if (rc) return rc;
  Params p = {};
  p.C = (__nv_bfloat16*)C; p.bias = bias; p.residual = (const __nv_bfloat16*)residual; p.aux = (__nv_bfloat16*)aux;
  p.M = M; p.N = N; p.K = K; p.ldc = ldc; p.flags = flags; p.error = error;
  // A last round of tiles that would leave half of the pairs idle is cut into halves of 128 columns, one for every pair (16384 x
  // 1024 x 1024 is 3.46 rounds of 74: with a residual 43 -> 40 us, times GELU' 45 -> 41, plain 28 both ways).
  const int tiles = ((M + BM - 1) / BM) * ((N + BN - 1) / BN), rest = tiles % max_pairs;
  p.whole = rest && 2 * rest <= max_pairs ? tiles - rest : tiles;
  p.items = p.whole + 2 * (tiles - p.whole);
  p.order = quick(tile_order(M, N, K, BM, BN));
  CUtensorMap mh = mb;
  if (p.items > p.whole) {
    rc = b_mn ? make_map_mnfold(&mh, B, (uint64_t)K, (uint64_t)N, (uint64_t)ldb, 1)
              : make_map_kfold(&mh, B, (uint64_t)N, (uint64_t)K, (uint64_t)ldb, 64);
    if (rc) return rc;
  }
  // Its own instance for launches that read nothing besides the accumulator: those hold two of its blocks in registers and two staging buffers a
  // warp, with eight warps; a side operand comes through the one buffer of each of sixteen.
  const int side = flags & kGeluGrad ? kArgument : flags & kResidual ? kSum : kNothing;
  const bool wide = !side && (flags & kGelu);
  CUtensorMap mside = mb, mc = mb;
  const void* const other = side == kSum ? residual : flags & (kAuxOut | kGeluGrad) ? aux : nullptr;
  rc = make_map_blocks(&mc, C, (uint64_t)M, (uint64_t)N, (uint64_t)ldc);
  if (!rc && other) rc = make_map_blocks(&mside, other, (uint64_t)M, (uint64_t)N, (uint64_t)ldc);
  if (rc) return -2;
  const int threads = wide || side ? Epilogue<kSum, false>::THREADS : Epilogue<kNothing, false>::THREADS;
  return launch(pick(b_mn, side, wide), threads, max_pairs, ma, mb, mh, p, mside, mc, stream);
}

// How many slabs of equal length the one-CTA kernel's weight gradient cuts K rows into for an M x N result: it doubles while
// the tiles still fit one wave of 148 CTAs and a slab keeps at least 512 rows.
int gcow_wgrad_slabs(int64_t M, int64_t N, int64_t K) {
  const int64_t tiles = ((M + 127) / 128) * ((N + 255) / 256);
  int s = 1;
  while (s < 64 && tiles * s * 2 <= 148 && K % (2 * s) == 0 && (K / (2 * s)) % 64 == 0 && K / (2 * s) >= 512) s *= 2;
  return s;
}

// How many slices of the reduction gcow_gemm2_wgrad cuts an M x N result over K rows into; 0: not taken (an operand narrower
// than a tile, or no cluster launches). Fewer tiles than pairs leave the others idle, and slices cost a pass over their M x N
// partial results: the count that a model of the two puts lowest, in us, fitted to 1024 to 50176 rows and results of 256 x 256 to
// 4096 x 4096 with 1 to 64 slices, launches with their sums in a chain: 0.7 per stage of 128 rows, 4 for a further round of tiles, and for the ordered
// sum 0.0014 s^2 + (1.17 s - 0.8) per million elements, half as much again where the partial results no longer fit the L2. An earlier model, of a
// slower kernel (0.71, 1.5 a round, 1.8 + 0.003 s^2 + (4.5 + 0.35 s) per million), cut less: 1024 rows to 768 x 768 one slice 12.8 us, four 10.2; 3000 to
// 2304 x 768 one 22.1, two 17.9; 4096 to 768 x 3072 one 28.1, two 22.0; 8192 to 3072 x 1024 one 47.2, three 45.2; 6144 to 4096 x 4096 still one, 153, two
// 172. It stays as the bound on a slice: where it cut more its count stays (8192 to 512 x 512 sixteen 16.7, thirteen 13.8), since fewer slices are longer
// sums, less exact ones than results had.
// No accumulator takes more stages than one of the slabs above: the tensor core cuts the running sum at every step, and the error
// grows with the number of steps (relative 2-norm, noise: 512 rows 4.7e-7, 1024 1.0e-6, 4096 4.4e-6). Where every pair has one
// item at most, its slice is shared by two accumulators: 1024 rows to 1024 x 1024 in one slice 14.2 us, in two slices 17.3, on
// the one-CTA kernel in two slabs 18.8.
int gcow_gemm2_wgrad_slices(int M, int N, int K) {
  const int max_pairs = gcow_gemm2_max_pairs();
  if (max_pairs <= 0 || M < 256 || N < 256 || M % 64 || N % 64 || K < 1024) return 0;
  const long long tiles = (long long)((M + BM - 1) / BM) * ((N + BN - 1) / BN);
  const int kblocks = (K + BK - 1) / BK, slab = K / gcow_wgrad_slabs(M, N, K), longest = (slab + BK - 1) / BK;
  const auto stages = [&](int s) { const int per = (kblocks + s - 1) / s; return tiles * s <= max_pairs ? (per + 1) / 2 : per; };   // per accumulator
  const auto rounds = [&](int s) { return (double)((tiles * s + max_pairs - 1) / max_pairs); };
  const auto cheapest = [&](int most, auto cost) {
    int best = 1;
    double least = 1e30;
    for (int s = 1; s <= 64 && kblocks / s >= 2; s++) {
      const int per = (kblocks + s - 1) / s;
      if ((s - 1) * per >= kblocks || stages(s) > most) continue;   // an empty slice; one too long
      const double c = cost(s, rounds(s), (double)per);
      if (c < least) { least = c; best = s; }
    }
    return best;
  };
  const double size = (double)M * N * 1e-6;
  const int before = cheapest(longest, [&](int s, double r, double per) { return r * per * 0.71 + (r - 1) * 1.5 + (s > 1 ? 1.8 + 0.003 * s * s + size * (4.5 + 0.35 * s) : 0.0); });
  return cheapest(stages(before), [&](int s, double r, double per) {
    return r * per * 0.7 + (r - 1) * 4.0 + (s > 1 ? 0.0014 * s * s + size * (1.17 * s - 0.8) * (size * s > 24 ? 1.5 : 1.0) : 0.0);
  });
}

// Partial column sums per slice that gcow_gemm2_wgrad leaves for a result of N columns; 0: it has none to give, one tile column sees half of A's.
int gcow_gemm2_wgrad_sums(int N) { return N <= BN ? 0 : ((N + BN - 1) / BN + 1) & ~1; }

// parts[slice][M][N] fp32 = A^T B over the slice's rows, A [K][M], B [K][N] bf16 with contiguous rows: the weight gradient of a
// linear layer. `slices` as gcow_gemm2_wgrad_slices has it. sums (or null): [slices * gcow_gemm2_wgrad_sums(N)][M] fp32, which add up to the
// column sums of A, the bias gradient.
int gcow_gemm2_wgrad(const void* A, const void* B, float* parts, float* sums, int M, int N, int K, int lda, int ldb, int slices, uint32_t* error,
                     void* stream) {
  if ((sums && N <= BN) || M <= 0 || N <= 0 || K <= 0 || slices <= 0 || M % 64 || N % 64 || lda % 8 || ldb % 8 || (((uintptr_t)parts | (uintptr_t)sums) & 15)) return -2;
  const int max_pairs = gcow_gemm2_max_pairs();
  if (max_pairs <= 0) return -2;
  CUtensorMap ma, mb;
  int rc = make_map_mnfold(&ma, A, (uint64_t)K, (uint64_t)M, (uint64_t)lda);
  if (!rc) rc = make_map_mnfold(&mb, B, (uint64_t)K, (uint64_t)N, (uint64_t)ldb);
  if (rc) return rc;
  Params p = {};
  p.C = (__nv_bfloat16*)parts;
  p.M = M; p.N = N; p.K = K; p.ldc = N; p.error = error;
  const int kblocks = (K + BK - 1) / BK;
  p.slice_blocks = (kblocks + slices - 1) / slices;
  if ((slices - 1) * p.slice_blocks >= kblocks) return -2;   // an empty slice would leave its part unwritten
  p.whole = p.items = ((M + BM - 1) / BM) * ((N + BN - 1) / BN) * slices;
  p.order = quick(tile_order(M, N, K, BM, BN));
  p.slice_stride = (size_t)M * N;
  p.halves = p.items <= max_pairs;
  p.aux = (__nv_bfloat16*)sums;
  return launch(gemm2_bf16_kernel<true, true, kNothing, false>, kThreads<true, kNothing, false>, max_pairs, ma, mb, mb, p, mb, mb, stream);
}

}  // extern "C"
