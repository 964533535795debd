// Tile kernels of the ZFP codec (sm_100a): every mode the one-store fixed-rate 1-D kernels do not cover - 2-D in any
// mode, fixed accuracy / precision, odd rates.
//
// Encode: a warp takes 32 * kPer consecutive blocks, codes each into a slot in shared memory (tile_coder.cuh), prefix-sums
// the lengths and packs the slots into one bit string in shared memory.
//   * Fixed rate: the string's place in the stream is known and word aligned, so the warp writes it there: one launch, no
//     scratch, no barrier.
//   * Variable rate: the warp writes its string, its length and its blocks' lengths (16 bits each) to scratch, all
//     coalesced, and the CTA its total; a second kernel adds up the totals before its share of the tiles and moves the
//     strings into place, shifted, together with the blocks' bit offsets. A word that two strings share is written by
//     the later one, which reads the earlier one's last 32 bits (a string that is followed by another has at least 32
//     bits, one per block). The strings are a fraction of the input and mostly still in L2, so this costs little, and
//     nothing waits: with the lengths passed on inside one kernel (decoupled look-back) the polling of a thousand CTAs
//     and the wait of every tile for its predecessors took longer than the coding itself (1-D, 25.6 M values at
//     tolerance 1e-6: 226 to 343 us for that kernel).
//
// Decode: a warp copies the segment of the stream that holds its 32 * kPer blocks into shared memory, coalesced, and each
// lane reads its blocks from there.
//
// Array walk and partial edge blocks follow sw/src/zfp.c:31-56,79-103 and sw/src/encode.c:41-88.
#include <cuda_runtime.h>
#include <stdint.h>
#include <atomic>
#include "tile_coder.cuh"

namespace gcow {

constexpr int kTileThreads = 256, kTileWarps = kTileThreads / 32;
// Blocks per lane: a 1-D block is little work, so four per lane make the steps per string (scan, copy) a small share; a 2-D
// block is sixteen values and up to 17 words of slot, so one.
template <int DIM> struct TileShape {
  static constexpr int kPer = DIM == 1 ? 4 : 1, kWarpBlocks = 32 * kPer, kBlocks = kTileThreads * kPer;
};

__device__ const TwinTable d_twin{};
__device__ const RunTable d_run{};

struct TileArgs {
  uint64_t nx, ny, blocks;
  uint32_t bx, tiles;             // blocks per row of blocks (2-D); tiles
  uint32_t slot_words, warp_words;  // encode: words per slot, per packed string; decode: window capacity, window pitch
  uint32_t pitch;                 // encode at variable rate: words from one string to the next in scratch
  ZfpParams p;
  int vec;                        // 2-D: values per load that the row pitch and the base address allow (4, 2 or 1); 1-D: 4 or 1
};

__device__ __forceinline__ void tile_load_1d(float* f, const float* __restrict__ in, const TileArgs& a, uint64_t b) {
  const uint64_t x0 = 4 * b;
  if (x0 + 4 <= a.nx) {
    if (a.vec == 4) {
      const float4 v = __ldg(reinterpret_cast<const float4*>(in) + b);
      f[0] = v.x; f[1] = v.y; f[2] = v.z; f[3] = v.w;
    } else {
#pragma unroll
      for (int i = 0; i < 4; i++) f[i] = __ldg(in + x0 + i);
    }
  } else {
    const uint32_t c = (uint32_t)(a.nx - x0);
    f[0] = f[1] = f[2] = f[3] = 0;
    for (uint32_t i = 0; i < c; i++) f[i] = in[x0 + i];
    pad_partial(f, c, 1);
  }
}
__device__ __forceinline__ void tile_store_1d(const float* f, float* __restrict__ out, const TileArgs& a, uint64_t b) {
  const uint64_t x0 = 4 * b;
  if (x0 + 4 <= a.nx) {
    if (a.vec == 4) {
      reinterpret_cast<float4*>(out)[b] = make_float4(f[0], f[1], f[2], f[3]);
    } else {
#pragma unroll
      for (int i = 0; i < 4; i++) out[x0 + i] = f[i];
    }
  } else {
    for (uint64_t i = 0; x0 + i < a.nx; i++) out[x0 + i] = f[i];
  }
}
__device__ __forceinline__ void tile_load_2d(float* f, const float* __restrict__ in, const TileArgs& a, uint64_t b) {
  const uint64_t by = a.blocks <= 0xffffffffull ? (uint64_t)((uint32_t)b / a.bx) : b / a.bx;
  const uint64_t x0 = 4 * (b - by * a.bx), y0 = 4 * by;
  const float* src = in + y0 * a.nx + x0;
  if (x0 + 4 <= a.nx && y0 + 4 <= a.ny) {
    if (a.vec == 4) {
#pragma unroll
      for (int y = 0; y < 4; y++) {
        const float4 v = __ldg(reinterpret_cast<const float4*>(src + y * a.nx));
        f[4 * y] = v.x; f[4 * y + 1] = v.y; f[4 * y + 2] = v.z; f[4 * y + 3] = v.w;
      }
    } else if (a.vec == 2) {
#pragma unroll
      for (int y = 0; y < 4; y++) {
        const float2 v = __ldg(reinterpret_cast<const float2*>(src + y * a.nx));
        const float2 w = __ldg(reinterpret_cast<const float2*>(src + y * a.nx + 2));
        f[4 * y] = v.x; f[4 * y + 1] = v.y; f[4 * y + 2] = w.x; f[4 * y + 3] = w.y;
      }
    } else {
#pragma unroll
      for (int y = 0; y < 4; y++)
#pragma unroll
        for (int x = 0; x < 4; x++) f[4 * y + x] = __ldg(src + y * a.nx + x);
    }
    return;
  }
  const uint32_t cx = (uint32_t)(a.nx - x0 < 4 ? a.nx - x0 : 4), cy = (uint32_t)(a.ny - y0 < 4 ? a.ny - y0 : 4);
#pragma unroll
  for (int i = 0; i < 16; i++) f[i] = 0;
#pragma unroll
  for (uint32_t y = 0; y < 4; y++) {
    if (y < cy) {
#pragma unroll
      for (uint32_t x = 0; x < 4; x++) if (x < cx) f[4 * y + x] = src[y * a.nx + x];
      if (cx < 4) pad_partial(f + 4 * y, cx, 1);
    }
  }
  if (cy < 4) {
#pragma unroll
    for (int x = 0; x < 4; x++) pad_partial(f + x, cy, 4);
  }
}
__device__ __forceinline__ void tile_store_2d(const float* f, float* __restrict__ out, const TileArgs& a, uint64_t b) {
  const uint64_t by = a.blocks <= 0xffffffffull ? (uint64_t)((uint32_t)b / a.bx) : b / a.bx;
  const uint64_t x0 = 4 * (b - by * a.bx), y0 = 4 * by;
  float* dst = out + y0 * a.nx + x0;
  if (x0 + 4 <= a.nx && y0 + 4 <= a.ny) {
    if (a.vec == 4) {
#pragma unroll
      for (int y = 0; y < 4; y++)
        *reinterpret_cast<float4*>(dst + y * a.nx) = make_float4(f[4 * y], f[4 * y + 1], f[4 * y + 2], f[4 * y + 3]);
    } else if (a.vec == 2) {
#pragma unroll
      for (int y = 0; y < 4; y++) {
        *reinterpret_cast<float2*>(dst + y * a.nx) = make_float2(f[4 * y], f[4 * y + 1]);
        *reinterpret_cast<float2*>(dst + y * a.nx + 2) = make_float2(f[4 * y + 2], f[4 * y + 3]);
      }
    } else {
#pragma unroll
      for (int y = 0; y < 4; y++)
#pragma unroll
        for (int x = 0; x < 4; x++) dst[y * a.nx + x] = f[4 * y + x];
    }
    return;
  }
#pragma unroll
  for (uint32_t y = 0; y < 4; y++)
#pragma unroll
    for (uint32_t x = 0; x < 4; x++)
      if (x0 + x < a.nx && y0 + y < a.ny) dst[y * a.nx + x] = f[4 * y + x];
}

// Scratch of the variable-rate encoder: the warps' strings, their lengths, the tiles' lengths, the blocks' lengths.
struct TileStrings {
  uint32_t* strings;
  uint32_t* unit_bits;
  uint32_t* tile_bits;
  uint16_t* lens;
};

// The stream ends with this string: its open word, and zeros up to a 64-bit boundary.
__device__ __forceinline__ void close_stream(uint32_t* __restrict__ out, const uint32_t* packed, uint64_t start, uint32_t total, uint32_t prev) {
  const uint32_t o = (uint32_t)(start & 31u), words = (total + 31) >> 5;
  const uint64_t bits = start + total, w64 = (bits + 63) >> 6;
  for (uint64_t w = bits >> 5; w < 2 * w64; w++) {
    const uint32_t i = (uint32_t)(w - (start >> 5));
    const uint32_t here = i < words ? packed[i] : 0u, below = i == 0 ? prev : i - 1 < words ? packed[i - 1] : 0u;
    out[w] = o ? __funnelshift_l(below, here, o) : here;
  }
}

template <int DIM, bool FIXED, bool BUDGET>
__global__ void __launch_bounds__(kTileThreads)
encode_tiles_kernel(const float* __restrict__ in, const TileArgs a, uint32_t* __restrict__ out, uint64_t* __restrict__ block_bits,
                    const TileStrings st, const uint16_t* __restrict__ enc_tab, const uint32_t* __restrict__ pair_tab) {
  constexpr int kPer = TileShape<DIM>::kPer, WB = TileShape<DIM>::kWarpBlocks, NB = TileShape<DIM>::kBlocks;
  constexpr int kTabWords = DIM == 1 ? kEncPairTabSize : kTwinTabSize;
  extern __shared__ __align__(16) uint32_t smem[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // table | per warp: slots [slot_words][WB], lengths [WB], packed string [warp_words]
  uint32_t* const tab = smem;
  uint32_t* const slots = smem + kTabWords + warp * (a.slot_words * WB + WB + a.warp_words);
  uint32_t* const lens = slots + a.slot_words * WB;
  uint32_t* const packed = lens + WB;
  __shared__ uint32_t s_total[2][kTileWarps];               // alternating: a warp can be one tile ahead of the sum

  if (DIM == 1) {
    for (int i = tid; i < kEncPairTabSize / 4; i += kTileThreads)
      reinterpret_cast<uint4*>(tab)[i] = reinterpret_cast<const uint4*>(pair_tab)[i];
  } else {
    if (tid < kTwinTabSize / 4) reinterpret_cast<uint4*>(tab)[tid] = reinterpret_cast<const uint4*>(d_twin.v)[tid];
  }
  __syncthreads();
  int turn = 0;
  for (uint32_t tile = blockIdx.x; tile < a.tiles; tile += gridDim.x, turn ^= 1) {
    const uint64_t b0 = (uint64_t)tile * NB + warp * WB;
    const uint32_t nb = a.blocks > b0 ? (a.blocks - b0 < WB ? (uint32_t)(a.blocks - b0) : WB) : 0;
#pragma unroll 1
    for (int j = 0; j < kPer; j++) {
      const uint32_t i = lane + 32 * j;
      uint32_t bits = 0;
      if (i < nb) {
        float f[1 << (2 * DIM)];
        if (DIM == 1) {
          tile_load_1d(f, in, a, b0 + i);
          bits = encode_slot_1d(f, a.p, tab, enc_tab, slots + i, WB);
        } else {
          tile_load_2d(f, in, a, b0 + i);
          bits = encode_slot_2d<BUDGET>(f, a.p, tab, slots + i, WB);
        }
      }
      lens[i] = bits;                                       // the block's own length, before padding to minbits
    }

    // lengths -> offsets within the warp's string
    uint32_t off[kPer], len[kPer], total = 0;
#pragma unroll
    for (int j = 0; j < kPer; j++) {
      const uint32_t i = lane + 32 * j;
      len[j] = lens[i];
      if (FIXED) {
        off[j] = i * a.p.maxbits;
      } else {
        uint32_t x = len[j];
        if (i < nb && x < a.p.minbits) x = a.p.minbits;
        const uint32_t v = x;
        if (i < nb) st.lens[b0 + i] = (uint16_t)v;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
          const uint32_t y = __shfl_up_sync(0xffffffffu, x, d);
          if (lane >= d) x += y;
        }
        off[j] = total + x - v;
        total += __shfl_sync(0xffffffffu, x, 31);
      }
    }
    if (FIXED) total = nb * a.p.maxbits;
    const uint32_t words = (total + 31) >> 5;
    for (uint32_t i = lane; i < words / 4 + 1; i += 32) reinterpret_cast<uint4*>(packed)[i] = make_uint4(0, 0, 0, 0);
    __syncwarp();
#pragma unroll
    for (int j = 0; j < kPer; j++) {
      const uint32_t nw = (len[j] + 31) >> 5, o = off[j] & 31u;
      uint32_t* dst = packed + (off[j] >> 5);
      const uint32_t* src = slots + lane + 32 * j;
      uint32_t carry = 0;
#pragma unroll 1
      for (uint32_t w = 0; w < nw; w++) {
        const uint32_t v = *src;
        src += WB;
        atomicOr(dst++, carry | (v << o));
        carry = funnel_l0(v, o);
      }
      if (carry) atomicOr(dst, carry);
    }
    __syncwarp();
    if (FIXED) {
      const uint64_t start = b0 * a.p.maxbits;              // a multiple of 32 bits
      const bool ends = nb && b0 + nb == a.blocks;
      uint32_t* const dst = out + (start >> 5);
      for (uint32_t i = lane; i < total >> 5; i += 32) dst[i] = packed[i];
      if (ends && lane == 0) close_stream(out, packed, start, total, 0);
      if (block_bits) {
#pragma unroll
        for (int j = 0; j < kPer; j++) {
          const uint32_t i = lane + 32 * j;
          if (i < nb) block_bits[b0 + i] = start + off[j];
        }
        if (ends && lane == 0) block_bits[a.blocks] = start + total;
      }
    } else {
      const uint64_t unit = (uint64_t)tile * kTileWarps + warp;
      uint32_t* const dst = st.strings + unit * a.pitch;
      for (uint32_t i = lane; i < words; i += 32) dst[i] = packed[i];
      if (lane == 0) {
        s_total[turn][warp] = total;
        if (nb) st.unit_bits[unit] = total;
      }
      __syncthreads();
      if (tid == 0) {
        uint32_t sum = 0;
#pragma unroll
        for (int w = 0; w < kTileWarps; w++) sum += s_total[turn][w];
        st.tile_bits[tile] = sum;
      }
    }
    __syncwarp();
  }
}

// Second kernel of the variable-rate encoder: every CTA takes a contiguous share of the tiles, at most kPlaceUnits strings
// at a time, whose starts it works out in shared memory first; then every load of a string depends on nothing but that
// table, and a warp keeps several of them in flight.
constexpr int kPlaceUnits = 1024;

template <int DIM>
__global__ void __launch_bounds__(kTileThreads, DIM == 1 ? 4 : 5)
place_strings_kernel(const TileStrings st, const TileArgs a, uint32_t* __restrict__ out, uint64_t* __restrict__ block_bits,
                     uint64_t* total_out) {
  constexpr int kPer = TileShape<DIM>::kPer, WB = TileShape<DIM>::kWarpBlocks;
  constexpr int kWords = DIM == 1 ? 8 : 3;                  // words per lane and step: a 1-D string is some 200 words, a 2-D one 70
  __shared__ unsigned long long s_sum[kTileWarps];
  __shared__ uint32_t s_warp[kTileWarps];
  __shared__ uint32_t s_bits[kPlaceUnits];                  // a string's length ...
  __shared__ uint32_t s_from[kPlaceUnits];                  // ... and start after the first one of the batch
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t t0 = (uint32_t)((uint64_t)a.tiles * blockIdx.x / gridDim.x);
  const uint32_t t1 = (uint32_t)((uint64_t)a.tiles * (blockIdx.x + 1) / gridDim.x);
  unsigned long long base = 0;
#pragma unroll 4
  for (uint32_t i = tid; i < t0 / 4; i += kTileThreads) {
    const uint4 v = reinterpret_cast<const uint4*>(st.tile_bits)[i];
    base += (unsigned long long)v.x + v.y + v.z + v.w;
  }
  if (tid < (t0 & 3u)) base += st.tile_bits[(t0 & ~3u) + tid];
#pragma unroll
  for (int d = 16; d; d >>= 1) base += __shfl_xor_sync(0xffffffffu, base, d);
  if (lane == 0) s_sum[warp] = base;
  __syncthreads();
  base = 0;
#pragma unroll
  for (int w = 0; w < kTileWarps; w++) base += s_sum[w];

  const uint64_t units = (a.blocks + WB - 1) / WB;
  const uint64_t u_end = (uint64_t)t1 * kTileWarps < units ? (uint64_t)t1 * kTileWarps : units;
  for (uint64_t u0 = (uint64_t)t0 * kTileWarps; u0 < u_end; u0 += kPlaceUnits) {
    const uint32_t nu = u_end - u0 < kPlaceUnits ? (uint32_t)(u_end - u0) : kPlaceUnits;
    // starts of this batch's strings: four consecutive ones per thread
    uint32_t v[4], sum = 0;
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const uint32_t i = tid * 4 + j;
      v[j] = i < nu ? st.unit_bits[u0 + i] : 0;
      sum += v[j];
    }
    uint32_t x = sum;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, x, d);
      if (lane >= d) x += y;
    }
    if (lane == 31) s_warp[warp] = x;
    __syncthreads();
    uint32_t from = x - sum, all = 0;
#pragma unroll
    for (int w = 0; w < kTileWarps; w++) {
      if (w < warp) from += s_warp[w];
      all += s_warp[w];
    }
#pragma unroll
    for (int j = 0; j < 4; j++) {
      s_bits[tid * 4 + j] = v[j];
      s_from[tid * 4 + j] = from;
      from += v[j];
    }
    __syncthreads();
    // the caller's host thread waits for the stream's length: it gets it before the strings are moved
    if (total_out && u0 + nu == units && tid == 0) {
      *(volatile uint64_t*)total_out = base + all;
      __threadfence_system();
    }

    // The loads of a warp's next string are issued before the current one is written.
    struct Fetched { uint32_t w[kWords], len[kPer], q0, q1; } cur, nxt;
    auto fetch = [&](uint32_t k, Fetched& f) {
      const uint64_t unit = u0 + k, b0 = unit * WB;
      const uint32_t nb = a.blocks - b0 < WB ? (uint32_t)(a.blocks - b0) : WB, words = (s_bits[k] + 31) >> 5;
      const uint32_t* const src = st.strings + unit * a.pitch;
      const uint16_t* const lens = st.lens + b0;
#pragma unroll
      for (int j = 0; j < kPer; j++) f.len[j] = lane + 32 * j < nb ? lens[lane + 32 * j] : 0;
#pragma unroll
      for (int j = 0; j < kWords; j++) f.w[j] = 32 * j + lane < words ? src[32 * j + lane] : 0u;
      f.q0 = f.q1 = 0;
      if (unit) {                                           // the words with the 32 bits before this string
        const uint32_t pt = k ? s_bits[k - 1] : st.unit_bits[unit - 1];
        const uint32_t* const q = src - a.pitch + ((pt - 32) >> 5);
        f.q0 = q[0];
        f.q1 = pt & 31u ? q[1] : 0u;
        f.q0 = window32(f.q0, f.q1, pt & 31u);
      }
    };
    if (warp < nu) fetch(warp, cur);
    for (uint32_t k = warp; k < nu; k += kTileWarps) {
      if (k + kTileWarps < nu) fetch(k + kTileWarps, nxt);
      const uint64_t unit = u0 + k, b0 = unit * WB, start = base + s_from[k];
      const uint32_t nb = a.blocks - b0 < WB ? (uint32_t)(a.blocks - b0) : WB, total = s_bits[k];
      const uint32_t* const src = st.strings + unit * a.pitch;
      const uint32_t o = (uint32_t)(start & 31u), words = (total + 31) >> 5, full = (o + total) >> 5;
      uint32_t* const dst = out + (start >> 5);
      uint32_t last = cur.q0;                               // the word before the next chunk
#pragma unroll
      for (int j = 0; j < kWords; j++) {
        const uint32_t i = 32 * j + lane;
        uint32_t below = __shfl_up_sync(0xffffffffu, cur.w[j], 1);
        if (lane == 0) below = last;
        last = __shfl_sync(0xffffffffu, cur.w[j], 31);
        if (i < full) dst[i] = __funnelshift_l(below, cur.w[j], o);
      }
#pragma unroll 1
      for (uint32_t i0 = 32 * kWords; i0 < full; i0 += 32) {  // a string longer than most
        const uint32_t i = i0 + lane, w = i < words ? src[i] : 0u;
        uint32_t below = __shfl_up_sync(0xffffffffu, w, 1);
        if (lane == 0) below = last;
        last = __shfl_sync(0xffffffffu, w, 31);
        if (i < full) dst[i] = __funnelshift_l(below, w, o);
      }
      uint64_t at = start;
#pragma unroll
      for (int j = 0; j < kPer; j++) {
        uint32_t y = cur.len[j];
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
          const uint32_t z = __shfl_up_sync(0xffffffffu, y, d);
          if (lane >= d) y += z;
        }
        if (lane + 32 * j < nb) block_bits[b0 + lane + 32 * j] = at + y - cur.len[j];
        at += __shfl_sync(0xffffffffu, y, 31);
      }
      if (b0 + nb == a.blocks && lane == 0) {
        block_bits[a.blocks] = start + total;
        close_stream(out, src, start, total, cur.q0);
      }
      cur = nxt;
    }
    base += all;
    __syncthreads();
  }
}

// 1-D tables in shared memory: the lean coder's windows and nibble pairs, and one plane per lookup.
// Before, with one plane per lookup throughout and a bit-matrix transpose per eight planes, 25.6 M values took: noise at
// tolerance 1e-6 121 us (now 101), at 1e-3 95 (93), at 6 bits/value 117 (97); a random walk at 1e-6 218 (138).
template <int DIM, bool BUDGET>
__global__ void __launch_bounds__(kTileThreads)
decode_tiles_kernel(const uint32_t* __restrict__ in, float* __restrict__ out, const TileArgs a,
                    const uint64_t* __restrict__ block_bits, int shift, const uint16_t* __restrict__ plane_tab, const uint32_t* __restrict__ loop_tab) {
  constexpr int kPer = TileShape<DIM>::kPer, WB = TileShape<DIM>::kWarpBlocks, NB = TileShape<DIM>::kBlocks;
  constexpr int kTabWords = DIM == 1 ? kTileDecTab1 : kRunTabSize;
  extern __shared__ __align__(16) uint32_t smem[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  uint32_t* const words = smem + kTabWords + warp * a.warp_words;
  const uint32_t cap = a.slot_words;
  if (DIM == 1) {
    for (int i = tid; i < 384; i += kTileThreads) reinterpret_cast<DecWindow*>(smem + kTileRows)[i] = make_tile_row(plane_tab, i);
    for (int i = tid; i < kDecTiny / 4; i += kTileThreads)   // windows and nibble pairs
      reinterpret_cast<uint4*>(smem)[i] = reinterpret_cast<const uint4*>(loop_tab)[i];
  } else {
    for (int i = tid; i < kRunTabSize / 4; i += kTileThreads) reinterpret_cast<uint4*>(smem)[i] = reinterpret_cast<const uint4*>(d_run.v)[i];
  }
  __syncthreads();
  for (uint32_t tile = blockIdx.x; tile < a.tiles; tile += gridDim.x) {
    const uint64_t b0 = (uint64_t)tile * NB + warp * WB;
    if (b0 >= a.blocks) return;                             // tiles only grow
    const uint32_t nb = a.blocks - b0 < WB ? (uint32_t)(a.blocks - b0) : WB;
    uint64_t at[kPer];
#pragma unroll
    for (int j = 0; j < kPer; j++) {
      const uint32_t i = lane + 32 * j < nb ? lane + 32 * j : nb - 1;
      at[j] = block_bits ? block_bits[b0 + i] : (b0 + i) * a.p.maxbits;
    }
    const uint64_t start = __shfl_sync(0xffffffffu, at[0], 0);
    const uint64_t end = block_bits ? block_bits[b0 + nb] : (b0 + nb) * a.p.maxbits;
    const uint64_t w0 = start >> 5, w1 = (end + 31) >> 5;
    const uint32_t nw = w1 - w0 < cap ? (uint32_t)(w1 - w0) : cap;
    const uint32_t* const src = in + w0;
    __syncwarp();
#pragma unroll 4
    for (uint32_t i = lane; i < nw; i += 32) words[i] = __ldg(src + i);
    if (lane < 4) words[nw + lane] = 0;
    __syncwarp();
#pragma unroll 1
    for (int j = 0; j < kPer; j++) {
      const uint32_t i = lane + 32 * j;
      if (i >= nb) break;
      const uint64_t rel = (j == 0 ? at[0] : j == 1 ? at[kPer > 1 ? 1 : 0] : j == 2 ? at[kPer > 2 ? 2 : 0] : at[kPer > 3 ? 3 : 0]) - (w0 << 5);
      const uint32_t pos = rel < (uint64_t)cap * 32 ? (uint32_t)rel : cap * 32;
      float f[1 << (2 * DIM)];
      if (DIM == 1) {
        decode_window_1d(f, a.p, smem, plane_tab, words, pos, shift);
        tile_store_1d(f, out, a, b0 + i);
      } else {
        decode_window_2d<BUDGET>(f, a.p, smem, words, pos, shift);
        tile_store_2d(f, out, a, b0 + i);
      }
    }
  }
}

}  // namespace gcow

using namespace gcow;

extern "C" int gcow_codec_tables4(const void** etab, const void** dtab, const void** epair, const void** dloop);

namespace {

template <int DIM> constexpr int blocks_per_tile() { return TileShape<DIM>::kBlocks; }

TileArgs tile_args(const void* values, uint64_t nx, uint64_t ny, const ZfpParams& p, uint64_t blocks, int dim) {
  TileArgs a;
  a.nx = nx; a.ny = ny; a.blocks = blocks; a.p = p;
  a.bx = dim == 2 ? (uint32_t)((nx + 3) / 4) : 1;
  a.slot_words = a.warp_words = a.pitch = 0;
  const uint64_t per = dim == 1 ? blocks_per_tile<1>() : blocks_per_tile<2>();
  a.tiles = (uint32_t)((blocks + per - 1) / per);
  const uintptr_t base = (uintptr_t)values;
  if (dim == 1) a.vec = (base & 15) == 0 ? 4 : 1;
  else a.vec = (base & 15) == 0 && nx % 4 == 0 ? 4 : (base & 7) == 0 && nx % 2 == 0 ? 2 : 1;
  return a;
}

// Words of a warp's packed string or window.
uint32_t warp_words_for(const ZfpParams& p, int dim) {
  const uint32_t wb = dim == 1 ? TileShape<1>::kWarpBlocks : TileShape<2>::kWarpBlocks;
  return (wb * max_block_bits(p, dim) + 31) / 32;
}
struct TileScratch { uint64_t strings, unit_bits, tile_bits, lens, bytes; };   // byte offsets
TileScratch tile_scratch(const ZfpParams& p, uint64_t blocks, int dim) {
  const uint64_t wb = dim == 1 ? TileShape<1>::kWarpBlocks : TileShape<2>::kWarpBlocks;
  const uint64_t units = (blocks + wb - 1) / wb, tiles = (units + kTileWarps - 1) / kTileWarps;
  TileScratch t;
  t.tile_bits = 0;                                            // first: read 16 bytes at a time
  t.strings = (tiles * 4 + 15) & ~15ull;
  t.unit_bits = t.strings + (blocks * max_block_bits(p, dim) + 31) / 32 * 4;
  t.lens = t.unit_bits + units * 4;
  t.bytes = t.lens + blocks * 2 + 16;                         // 16: the base is rounded up
  return t;
}
constexpr uint32_t kPackedPad = 4;                            // the word after the string, and whole 16-byte rows
constexpr uint32_t kReadAhead = kTileMaxBlockBits / 32 + 8;   // a block never reads further than this past its start
uint32_t round4(uint32_t v) { return (v + 3) & ~3u; }

template <auto kKernel>
int grid_of(uint32_t smem, uint32_t tiles, int* err) {
  static std::atomic<uint64_t> allowed{0};                  // one bit per device: the large dynamic allocation is permitted
  int dev = 0;
  *err = (int)cudaGetDevice(&dev);
  if (*err) return 0;
  if (dev >= 64 || !((allowed.load(std::memory_order_relaxed) >> dev) & 1)) {
    *err = (int)cudaFuncSetAttribute(kKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    if (*err) return 0;
    if (dev < 64) allowed.fetch_or(1ull << dev, std::memory_order_relaxed);
  }
  // 228 KB of shared memory and 2048 threads per SM; more CTAs than fit would only queue
  uint32_t per_sm = (228u * 1024) / (smem + 1024);
  if (per_sm > 2048 / kTileThreads) per_sm = 2048 / kTileThreads;
  if (per_sm < 1) per_sm = 1;
  const uint32_t g = 148 * per_sm;
  return (int)(tiles < g ? tiles : g);
}

}  // namespace

extern "C" {

// Whether the tile kernels take these parameters (1) or the slot / scan / scatter kernels have to (0): blocks padded
// beyond the longest code a block can have would need slots of any size.
int gcow_tile_usable(const int32_t* params, uint64_t blocks, int dim) {
  const ZfpParams p = {(uint32_t)params[0], (uint32_t)params[1], (uint32_t)params[2], params[3]};
  const uint32_t limit = dim == 1 ? 160u : kTileMaxBlockBits;
  return max_block_bits(p, dim) <= limit && blocks <= 0xffffffffull * 64 ? 1 : 0;
}

// Scratch of gcow_encode_tiles in bytes: 0 at fixed rate; else the strings (as many words as the longest possible stream),
// a length per string and per tile, and 16 bits per block.
uint64_t gcow_encode_tiles_scratch_bytes(const int32_t* params, uint64_t blocks, int dim) {
  if (params[0] == params[1]) return 0;
  const ZfpParams p = {(uint32_t)params[0], (uint32_t)params[1], (uint32_t)params[2], params[3]};
  return tile_scratch(p, blocks, dim).bytes;
}

// A word of pinned host memory of the calling thread, set to all ones: where an encode call leaves the stream's length for
// the thread that made it. One per thread, given back when the thread ends.
int gcow_host_word(uint64_t** word) {
  struct Word {
    uint64_t* p = nullptr;
    ~Word() { if (p) (void)cudaFreeHost(p); }
  };
  static thread_local Word w;
  if (!w.p) {
    const cudaError_t e = cudaHostAlloc((void**)&w.p, 64, cudaHostAllocPortable | cudaHostAllocMapped);
    if (e != cudaSuccess) { w.p = nullptr; return (int)e; }
  }
  *(volatile uint64_t*)w.p = ~0ull;
  *word = w.p;
  return 0;
}

// Waits until the device has written the word. The stream is asked now and then, so a launch that failed, or ended without
// writing, ends the wait.
int gcow_wait_host_word(volatile uint64_t* word, void* stream, uint64_t* value) {
  for (;;) {
    for (int i = 0; i < 512; i++) {
      if ((*value = *word) != ~0ull) return 0;
#if defined(__x86_64__)
      __builtin_ia32_pause();
#endif
    }
    const cudaError_t e = cudaStreamQuery((cudaStream_t)stream);
    if (e == cudaSuccess) return (*value = *word) != ~0ull ? 0 : -1;
    if (e != cudaErrorNotReady) return (int)e;
  }
}

uint64_t gcow_max_stream_bytes(const int32_t* params, uint64_t blocks, int dim) {
  const ZfpParams p = {(uint32_t)params[0], (uint32_t)params[1], (uint32_t)params[2], params[3]};
  return max_output_bytes(p, blocks, dim);
}

// Encode without touching anything of `out` but the stream itself (its last word zero padded to 64 bits). `block_bits`
// (blocks + 1, device) receives every block's start bit and the total; it may be null at fixed rate.
// `total_out` (host memory that the device can write, or null): at variable rate also receives the total, early.
int gcow_encode_tiles(const float* in, uint64_t nx, uint64_t ny, const int32_t* params, void* out, void* scratch,
                      uint64_t* block_bits, uint64_t* total_out, void* stream) {
  cudaStream_t s = (cudaStream_t)stream;
  const ZfpParams p = {(uint32_t)params[0], (uint32_t)params[1], (uint32_t)params[2], params[3]};
  const int dim = ny ? 2 : 1;
  const uint64_t blocks = ny ? num_blocks_2d(nx, ny) : num_blocks_1d(nx);
  if (!blocks) return 0;
  if (!gcow_tile_usable(params, blocks, dim)) return -3;
  const bool fixed = is_fixed_rate(p);
  if (!fixed && (!block_bits || !scratch)) return -1;
  const void *et, *dt, *pt, *lt;
  if (int rc = gcow_codec_tables4(&et, &dt, &pt, &lt)) return rc;
  TileArgs a = tile_args(in, nx, ny, p, blocks, dim);
  a.slot_words = tile_slot_words(p, dim);
  a.warp_words = round4(warp_words_for(p, dim) + kPackedPad);
  const uint32_t wb = dim == 1 ? TileShape<1>::kWarpBlocks : TileShape<2>::kWarpBlocks;
  const uint32_t smem = ((dim == 1 ? kEncPairTabSize : kTwinTabSize) + kTileWarps * (a.slot_words * wb + wb + a.warp_words)) * 4;
  const TileScratch ts = tile_scratch(p, blocks, dim);
  char* const sp = (char*)(((uintptr_t)scratch + 15) & ~(uintptr_t)15);
  a.pitch = wb / 32 * max_block_bits(p, dim);
  TileStrings st = {};
  if (!fixed) st = {(uint32_t*)(sp + ts.strings), (uint32_t*)(sp + ts.unit_bits), (uint32_t*)(sp + ts.tile_bits), (uint16_t*)(sp + ts.lens)};
  int err = 0;
#define GCOW_ENCODE(D, F, B)                                                                                   \
  do {                                                                                                         \
    const int g = grid_of<&encode_tiles_kernel<D, F, B>>(smem, a.tiles, &err);                                 \
    if (err) return err;                                                                                       \
    encode_tiles_kernel<D, F, B><<<g, kTileThreads, smem, s>>>(in, a, (uint32_t*)out, block_bits, st,         \
                                                               (const uint16_t*)et, (const uint32_t*)pt);      \
  } while (0)
  const bool cuts = tile_budget_cuts(p, dim);
  if (dim == 1) { if (fixed) GCOW_ENCODE(1, true, true); else GCOW_ENCODE(1, false, true); }
  else if (fixed) { if (cuts) GCOW_ENCODE(2, true, true); else GCOW_ENCODE(2, true, false); }
  else { if (cuts) GCOW_ENCODE(2, false, true); else GCOW_ENCODE(2, false, false); }
#undef GCOW_ENCODE
  if (!fixed) {
    const uint32_t most = 148 * (dim == 1 ? 4 : 5), g = a.tiles < most ? a.tiles : most;
    if (dim == 1) place_strings_kernel<1><<<g, kTileThreads, 0, s>>>(st, a, (uint32_t*)out, block_bits, total_out);
    else place_strings_kernel<2><<<g, kTileThreads, 0, s>>>(st, a, (uint32_t*)out, block_bits, total_out);
  }
  return (int)cudaGetLastError();
}

// Decode; block_bits == nullptr means fixed rate (block b starts at b * maxbits). Reads no word past the one that holds
// the last block's last bit.
int gcow_decode_tiles(const void* in, float* out, uint64_t nx, uint64_t ny, const int32_t* params,
                      const uint64_t* block_bits, int shift, void* stream) {
  cudaStream_t s = (cudaStream_t)stream;
  const ZfpParams p = {(uint32_t)params[0], (uint32_t)params[1], (uint32_t)params[2], params[3]};
  const int dim = ny ? 2 : 1;
  const uint64_t blocks = ny ? num_blocks_2d(nx, ny) : num_blocks_1d(nx);
  if (!blocks) return 0;
  if (!gcow_tile_usable(params, blocks, dim)) return -3;
  if (!block_bits && !is_fixed_rate(p)) return -2;
  const void *et, *dt, *pt, *lt;
  if (int rc = gcow_codec_tables4(&et, &dt, &pt, &lt)) return rc;
  TileArgs a = tile_args(out, nx, ny, p, blocks, dim);
  a.slot_words = warp_words_for(p, dim) + 1;                 // window capacity: one more for the bits before the first block
  a.warp_words = round4(a.slot_words + kReadAhead);
  const uint32_t smem = ((dim == 1 ? (uint32_t)kTileDecTab1 : (uint32_t)kRunTabSize) + kTileWarps * a.warp_words) * 4;
  int err = 0;
#define GCOW_DECODE(D, B)                                                                                      \
  do {                                                                                                         \
    const int g = grid_of<&decode_tiles_kernel<D, B>>(smem, a.tiles, &err);                                    \
    if (err) return err;                                                                                       \
    decode_tiles_kernel<D, B><<<g, kTileThreads, smem, s>>>((const uint32_t*)in, out, a, block_bits, shift, (const uint16_t*)dt, (const uint32_t*)lt); \
  } while (0)
  if (dim == 1) GCOW_DECODE(1, true);
  else if (tile_budget_cuts(p, 2)) GCOW_DECODE(2, true);
  else GCOW_DECODE(2, false);
#undef GCOW_DECODE
  return (int)cudaGetLastError();
}

}  // extern "C"
