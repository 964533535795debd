// Tile kernels of the ZFP codec (sm_100a): every mode the one-store fixed-rate 1-D kernels do not cover - 2-D in any
// mode, fixed accuracy / precision, odd rates.
//
// Encode: a warp takes 32 * kPer consecutive blocks.
//   * Fixed rate: every block is coded into a slot in shared memory (tile_coder.cuh). Blocks of whole words: every lane stores its
//     block where it belongs, 16 bytes at a time. Other rates: the warp packs its slots into one bit string, whose place in
//     the stream is known and word aligned. One launch, no scratch.
//   * Variable rate: the warp's blocks grow into one bit string in shared memory, 32 at a time (StringBuilder), and leave as a
//     part of ONE string per tile (a CTA's 256 * kPer blocks), shifted by the length of the warps before it; a word that two
//     warps share is written by the later one, which takes the earlier one's last 32 bits from shared memory (a string that
//     is followed by another has at least 32 bits, one per block). Every block's offset within its warp's string (16 bits)
//     and every warp's within the tile go to scratch with it, all coalesced. A second kernel adds up the tiles' lengths
//     before its share of them and moves their strings into place the same way, together with the blocks' bit offsets.
//     Nothing waits: with the lengths passed on inside one kernel (decoupled look-back) the polling of a thousand CTAs and the
//     wait of every tile for its predecessors took longer than the coding itself (1-D, 25.6 M values at tolerance 1e-6:
//     226 to 343 us for that kernel).
//
// Decode: a warp copies the segment of the stream that holds its 32 * kPer blocks into shared memory, coalesced, and each
// lane reads its blocks from there.
//
// Array walk and partial edge blocks follow sw/src/zfp.c:31-56,79-103 and sw/src/encode.c:41-88.
#include <cuda_runtime.h>
#include <stdint.h>
#include <atomic>
#include "tile_coder.cuh"
#include "../ops/pdl.cuh"

namespace gcow {

constexpr int kTileThreads = 256, kTileWarps = kTileThreads / 32;
// Blocks per lane, kPer. A 1-D block is little work, so four per lane make the steps per string (copy, totals) a small share -
// but one per lane where four would leave SMs without a CTA, since a lane's blocks follow one another. A 2-D block is
// sixteen values and up to 17 words of slot, so one.
constexpr uint64_t kWideBlocks = 148ull * 4 * kTileThreads;   // more than this: four per lane
inline int tile_per(uint64_t blocks, int dim) { return dim == 1 && blocks > kWideBlocks ? 4 : 1; }

// Blocks of a tile's first 32 of a warp that may leave the 1-D straight line before the warp stops trying it. 25.6 M values decoded,
// us, plane loop alone, straight line always first, with this rule: N(0, 1e-3) at tolerance 1e-6 101, 80.4, 81.4; values near 1 at
// tolerance 1e-3 133, 146, 128, at precision 8 99, 121, 95; a random walk at 1e-3 132, 144, 126; one smooth block in eight
// among noise 156, 179, 164.
// Encoder, likewise (with the straight line always first, a group of zero blocks went through the atomic operations too): N(0, 1e-3) at
// tolerance 1e-6 139, 134.9, 136.5; values within 1e-6 of 1 at 1e-6 255, 302, 252; denormals at precision 16 146, 176, 155; zeros at
// precision 16 79, 110, 76, at tolerance 1e-3 93, 110, 77.
constexpr int kLeftMost = 4;

__device__ const TwinTable d_twin{};
__device__ const RunTable d_run{};

struct TileArgs {
  uint64_t nx, ny, blocks;
  uint32_t bx, tiles;             // blocks per row of blocks (2-D); tiles
  uint32_t slot_words, warp_words;  // encode: words per slot, per packed string; decode: window capacity, window pitch
  uint32_t pitch;                 // encode at variable rate: words from one tile's string to the next in scratch
  ZfpParams p;
  int wide;                       // encode, kDirect: blocks of whole 16 bytes at an aligned address
  Divisor row;                    // 2-D: by bx
  int vec;                        // 2-D: values per load that the row pitch and the base address allow (4, 2 or 1); 1-D: 4 or 1
};

__device__ __forceinline__ void tile_load_1d(float* f, const float* in, const TileArgs& a, uint64_t b) {
  const uint64_t x0 = 4 * b;
  if (x0 + 4 <= a.nx) {
    if (a.vec == 4) {
      const float4 v = reinterpret_cast<const float4*>(in)[b];
      f[0] = v.x; f[1] = v.y; f[2] = v.z; f[3] = v.w;
    } else {
#pragma unroll
      for (int i = 0; i < 4; i++) f[i] = in[x0 + i];
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
// The row of blocks that block b is in. A division by a number the compiler does not know is some twenty instructions, of about 850 a
// block takes.
__device__ __forceinline__ uint64_t block_row(const TileArgs& a, uint64_t b) {
  return a.blocks <= 0x80000000ull ? (uint64_t)a.row.under((uint32_t)b) : b / a.bx;
}
__device__ __forceinline__ void tile_load_2d(float* f, const float* in, const TileArgs& a, uint64_t b) {
  const uint64_t by = block_row(a, b);
  const uint64_t x0 = 4 * (b - by * a.bx), y0 = 4 * by;
  const float* src = in + y0 * a.nx + x0;
  if (x0 + 4 <= a.nx && y0 + 4 <= a.ny) {
    if (a.vec == 4) {
#pragma unroll
      for (int y = 0; y < 4; y++) {
        const float4 v = *reinterpret_cast<const float4*>(src + y * a.nx);
        f[4 * y] = v.x; f[4 * y + 1] = v.y; f[4 * y + 2] = v.z; f[4 * y + 3] = v.w;
      }
    } else if (a.vec == 2) {
#pragma unroll
      for (int y = 0; y < 4; y++) {
        const float2 v = *reinterpret_cast<const float2*>(src + y * a.nx);
        const float2 w = *reinterpret_cast<const float2*>(src + y * a.nx + 2);
        f[4 * y] = v.x; f[4 * y + 1] = v.y; f[4 * y + 2] = w.x; f[4 * y + 3] = w.y;
      }
    } else {
#pragma unroll
      for (int y = 0; y < 4; y++)
#pragma unroll
        for (int x = 0; x < 4; x++) f[4 * y + x] = src[y * a.nx + x];
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
  const uint64_t by = block_row(a, b);
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

// Scratch of the variable-rate encoder: the tiles' strings and lengths, the warps' offsets in them, the blocks' in their warp's.
struct TileStrings {
  uint32_t* strings;
  uint32_t* tile_bits;
  uint32_t* warp_at;
  uint16_t* block_at;
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

// The last 32 bits of a string of at least 32.
__device__ __forceinline__ uint32_t last_bits(const uint32_t* string, uint32_t bits) {
  const uint32_t* const q = string + ((bits - 32) >> 5);
  return bits & 31u ? __funnelshift_r(q[0], q[1], bits) : q[0];
}

// The words of w, zero past the code, to bit `at` of a zeroed string.
template <int NW>
__device__ __forceinline__ void put_bits(uint32_t* string, uint32_t at, const uint32_t (&w)[NW]) {
  uint32_t* const dst = string + (at >> 5);
  uint32_t below = 0;
#pragma unroll
  for (int i = 0; i <= NW; i++) {
    const uint32_t here = i < NW ? w[i < NW ? i : 0] : 0u, v = __funnelshift_l(below, here, at);
    if (v) atomicOr(dst + i, v);
    below = here;
  }
}

// A warp's string as it grows, 32 blocks (one per lane, in order) at a time. Words are stored once, whole: a word that two
// blocks share is stored by the later one, which gets the earlier one's last bits by a shuffle; `carry` holds the last,
// open word of the string so far. That takes blocks of 32 to 128 bits (a shorter one could share its word with two
// others); a group of blocks of one bit is a ballot, and any other group is put together by atomic operations on zeroed words.
struct StringBuilder {
  uint32_t* string;
  uint32_t at, carry;          // bits so far; the word they end in (0 where they end on its boundary)
  __device__ __forceinline__ explicit StringBuilder(uint32_t* s) : string(s), at(0), carry(0) {}
  // This lane's block: `len` bits with its padding (0: none, behind the last one); w: all of it, zero past its end, if in_w;
  // put(place) adds the block to zeroed words otherwise. Returns the block's place.
  template <class Put>
  __device__ __forceinline__ uint32_t add(int lane, uint32_t len, bool in_w, const uint32_t (&w)[4], Put&& put) {
    uint32_t x = len;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, x, d);
      if (lane >= d) x += y;
    }
    const uint32_t place = at + x - len, end = at + __shfl_sync(0xffffffffu, x, 31), o = place & 31u;
    if (__all_sync(0xffffffffu, in_w && len - 32u <= 96u)) {
      const uint32_t n = (o + len) >> 5;                   // words that end in this block: 1 to 4
      const uint32_t w0 = w[0] << o, w1 = __funnelshift_l(w[0], w[1], o), w2 = __funnelshift_l(w[1], w[2], o),
                     w3 = __funnelshift_l(w[2], w[3], o), w4 = __funnelshift_l(w[3], 0u, o);
      const uint32_t open = n == 1 ? w1 : n == 2 ? w2 : n == 3 ? w3 : w4;
      uint32_t below = __shfl_up_sync(0xffffffffu, open, 1);
      if (lane == 0) below = carry;
      carry = __shfl_sync(0xffffffffu, open, 31);
      uint32_t* const dst = string + (place >> 5);
      dst[0] = w0 | below;
      if (n > 1) dst[1] = w1;
      if (n > 2) dst[2] = w2;
      if (n > 3) dst[3] = w3;
    } else if (__all_sync(0xffffffffu, len <= 1u)) {       // blocks of one bit: the group is a word
      const uint32_t bits = __ballot_sync(0xffffffffu, w[0] & 1u), here = at & 31u;
      if (here + (end - at) >= 32u) {
        if (lane == 0) string[at >> 5] = carry | (bits << here);
        carry = funnel_l0(bits, here);
      } else {
        carry |= bits << here;
      }
    } else {
      for (uint32_t i = (at >> 5) + lane; i <= end >> 5; i += 32) string[i] = i == at >> 5 ? carry : 0u;
      __syncwarp();
      put(place);
      __syncwarp();
      carry = string[end >> 5];
      __syncwarp();
    }
    at = end;
    return place;
  }
  // The open word joins the others; the lanes may read the string.
  __device__ __forceinline__ void close(int lane) {
    if (lane == 0 && (at & 31u)) string[at >> 5] = carry;
    __syncwarp();
  }
};

// CTAs per SM of the 2-D coders: 48 registers, which hold a block without a spill, where the compiler left to itself takes up to 62 and
// four CTAs fit. 7654 x 7654 at tolerance 1e-3: encoding 153.7 -> 148.4 us, decoding 123.5 -> 115.8; at 1e-1 118.4 -> 112.3 and 72.6 -> 66.2;
// 2047 x 3001 at 8 bits/value decoding 22.4 -> 21.7. Six (40 registers, 20 to 40 bytes of spills): 161.9, 116.3, 128.1, 63.6. The 1-D
// coders take 40 to 48 registers by themselves and lose by being told.
// Where four CTAs per SM hold all tiles at once the unbounded instance stays: more places than that only let some SMs take more tiles than
// others (1500 x 1500: 1e-3 13.4 and 7.9 us unbounded, 14.4 and 8.7 bounded, 16 bits/value decoding 13.4 and 15.0; 2000 x 2000:
// 17.7 and 12.2, 17.6 and 11.9; just above the line, 1600 x 1600, decoding at 4 bits/value is slower bounded, 11.3 and 12.0, at 16 bits/value, 1e-3 and 1e-1
// faster, 15.0 and 14.4, 8.3 and 7.8, 4.9 and 4.0).
constexpr int kCtas2d = 5;

enum TileMode { kVariable, kPacked, kDirect };              // variable rate; fixed rate; fixed rate in whole words

template <int DIM, int PER, TileMode MODE, bool BUDGET, int CTAS>
__global__ void __launch_bounds__(kTileThreads, CTAS)
encode_tiles_kernel(const float* in, const TileArgs a, uint32_t* __restrict__ out, uint64_t* __restrict__ block_bits,
                    const TileStrings st, const uint16_t* __restrict__ enc_tab, const uint32_t* __restrict__ pair_tab) {
  constexpr int WB = 32 * PER, NB = kTileThreads * PER;
  constexpr int kTabWords = DIM == 1 ? kEncPairTabSize : kTwinTabSize;
  constexpr int SW = MODE == kVariable ? 32 : WB;           // variable rate: a slot per lane, used again for its next block
  extern __shared__ __align__(16) uint32_t smem[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // table | per warp: slots [slot_words][SW], packed string [warp_words] (none for kDirect)
  uint32_t* const tab = smem;
  uint32_t* const slots = smem + kTabWords + warp * (a.slot_words * SW + a.warp_words);
  uint32_t* const packed = slots + a.slot_words * SW;
  __shared__ uint32_t s_total[2][kTileWarps], s_last[2][kTileWarps];   // alternating: a warp can be one tile ahead of the others

  pdl_trigger();                                            // the kernel that moves the strings may set itself up
  if (DIM == 1) {
    for (int i = tid; i < kEncPairTabSize / 4; i += kTileThreads)
      reinterpret_cast<uint4*>(tab)[i] = reinterpret_cast<const uint4*>(pair_tab)[i];
  } else {
    if (tid < kTwinTabSize / 4) reinterpret_cast<uint4*>(tab)[tid] = reinterpret_cast<const uint4*>(d_twin.v)[tid];
  }
  if (MODE == kPacked)
    for (uint32_t i = lane; i < a.warp_words / 4; i += 32) reinterpret_cast<uint4*>(packed)[i] = make_uint4(0, 0, 0, 0);
  __syncthreads();
  pdl_wait();                                               // the tables came under the tail of the stream's last kernel
  int turn = 0;
  bool straight = !BUDGET;                                  // 1-D: as in the decoder
  for (uint32_t tile = blockIdx.x; tile < a.tiles; tile += gridDim.x, turn ^= 1) {
    const uint64_t b0 = (uint64_t)tile * NB + warp * WB;
    const uint32_t nb = a.blocks > b0 ? (a.blocks - b0 < WB ? (uint32_t)(a.blocks - b0) : WB) : 0;
    if (MODE == kVariable) {
      StringBuilder string(packed);
#pragma unroll 1
      for (int j = 0; j < PER; j++) {
        const uint32_t i = lane + 32 * j;
        const bool there = i < nb;
        uint32_t bits = 0, w[4] = {0, 0, 0, 0};
        bool in_w = false;
        bool left = false;                                  // by the straight line
        if (there) {
          float f[1 << (2 * DIM)];
          if (DIM == 1) {
            tile_load_1d(f, in, a, b0 + i);
            in_w = straight && encode_code_1d(f, a.p, tab, w, bits);
            left = !in_w;
            if (!in_w) bits = encode_slot_1d(f, a.p, tab, enc_tab, slots + lane, 32);
          } else {
            tile_load_2d(f, in, a, b0 + i);
            bits = encode_slot_2d<BUDGET>(f, a.p, tab, slots + lane, 32);
          }
          if (!in_w && bits <= 128u) {
            in_w = true;
#pragma unroll
            for (uint32_t k = 0; k < 4; k++) w[k] = 32 * k < bits ? slots[lane + 32 * k] : 0u;
          }
        }
        if (DIM == 1 && !BUDGET && j == 0 && straight) straight = __popc(__ballot_sync(0xffffffffu, left)) < kLeftMost;
        const uint32_t place = string.add(lane, there && bits < a.p.minbits ? a.p.minbits : bits, in_w, w, [&](uint32_t at) {
          if (!there) return;
          if (in_w) put_bits(packed, at, w);
          else for (uint32_t k = 0; 32 * k < bits; k++) put_bits(packed, at + 32 * k, {slots[lane + 32 * k]});
        });
        if (there) st.block_at[b0 + i] = (uint16_t)place;
      }
      string.close(lane);
      const uint32_t total = string.at, words = (total + 31) >> 5;
      if (lane == 0) {
        s_total[turn][warp] = total;
        s_last[turn][warp] = total >= 32 ? last_bits(packed, total) : 0u;
      }
      __syncthreads();
      uint32_t at = 0, all = 0;
#pragma unroll
      for (int w = 0; w < kTileWarps; w++) {
        if (w == warp) at = all;
        all += s_total[turn][w];
      }
      if (tid == 0) st.tile_bits[tile] = all;
      if (lane == 0 && nb) st.warp_at[(uint64_t)tile * kTileWarps + warp] = at;
      // whole words up to this string's end (the tile's last string: and the open one)
      const uint32_t o = at & 31u, prev = at ? s_last[turn][warp - 1] : 0u;
      const uint32_t n = at + total == all ? (o + total + 31) >> 5 : (o + total) >> 5;
      uint32_t* const dst = st.strings + (uint64_t)tile * a.pitch + (at >> 5);
      if (nb)
        for (uint32_t i = lane; i < n; i += 32) dst[i] = __funnelshift_l(i ? packed[i - 1] : prev, i < words ? packed[i] : 0u, o);
      __syncwarp();
      continue;
    }

    uint32_t lens[PER] = {};                                // the blocks' own lengths, before padding to minbits
#pragma unroll 1
    for (int j = 0; j < PER; j++) {
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
#pragma unroll
      for (int k = 0; k < PER; k++) lens[k] = PER == 1 || k == j ? bits : lens[k];
    }

    if (MODE == kDirect) {
      const uint32_t bw = a.p.maxbits >> 5;                 // words per block
#pragma unroll
      for (int j = 0; j < PER; j++) {
        const uint32_t i = lane + 32 * j;
        if (i >= nb) break;
        const uint32_t* const src = slots + i;
        uint32_t* const dst = out + (b0 + i) * bw;
        const uint32_t nw = (lens[j] + 31) >> 5;
        auto word = [&](uint32_t w) { return w < nw ? src[w * WB] : 0u; };
        if (a.wide) {
          for (uint32_t w = 0; w < bw; w += 4) *reinterpret_cast<uint4*>(dst + w) = make_uint4(word(w), word(w + 1), word(w + 2), word(w + 3));
        } else {
          for (uint32_t w = 0; w < bw; w++) dst[w] = word(w);
        }
        if (block_bits) block_bits[b0 + i] = (b0 + i) * a.p.maxbits;
        if (b0 + i + 1 == a.blocks) {
          if (block_bits) block_bits[a.blocks] = a.blocks * a.p.maxbits;
          if ((a.blocks * bw) & 1u) dst[bw] = 0;            // zeros up to a 64-bit boundary
        }
      }
      continue;
    }

    const uint32_t total = nb * a.p.maxbits, words = (total + 31) >> 5;
    __syncwarp();
#pragma unroll
    for (int j = 0; j < PER; j++) {
      const uint32_t off = (lane + 32 * j) * a.p.maxbits, nw = (lens[j] + 31) >> 5, o = off & 31u;
      uint32_t* dst = packed + (off >> 5);
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
    const uint64_t start = b0 * a.p.maxbits;                // a multiple of 32 bits
    const bool ends = nb && b0 + nb == a.blocks;
    uint32_t* const dst = out + (start >> 5);
    for (uint32_t i = lane; i < total >> 5; i += 32) dst[i] = packed[i];
    if (ends && lane == 0) close_stream(out, packed, start, total, 0);
    if (block_bits) {
#pragma unroll
      for (int j = 0; j < PER; j++) {
        const uint32_t i = lane + 32 * j;
        if (i < nb) block_bits[b0 + i] = start + i * a.p.maxbits;
      }
      if (ends && lane == 0) block_bits[a.blocks] = start + total;
    }
    __syncwarp();
    for (uint32_t i = lane; i < words; i += 32) packed[i] = 0;
    __syncwarp();
  }
}

// Second kernel of the variable-rate encoder: every CTA takes a contiguous share of the tiles, at most kTileThreads of them at a
// time, whose starts it works out in shared memory first; then nothing depends on anything but that table, and the
// warps run through the strings at their own pace, each with parts of PART blocks and as large a share of their tile's words.
// Bound by latency and by the bytes: a part is a few loads in a row, all of them ahead of the stores, and most of a small array's time is the
// wait for the coder and the sum of the tiles before. With the whole CTA on one tile (154 instructions a warp for some 40 words and
// 32 offsets, now a fifth of that) both kernels took, us, 7654 x 7654 at tolerance 1e-3 148.6, now 142, at 1e-1 112.6, now 102.4; 510 x 510 9.3, now
// 8.8; 25.6 M values at tolerance 1e-6 132.7, now 129.7, at 1e-3 112.6, now 109.7. Six CTAs per SM with 128 blocks of four
// a lane 131 and 114.4, four 134.7 and 115.7, with 64 blocks 142 and 122.
// The next kernel is let in once the tiles before are added up: with 244 tiles a decoder that came at the start found the SMs unevenly
// taken (1 M values at tolerance 1e-3, encoder and decoder 26.5 us, now 20.5; 510 x 510 14.5, now 13.4); at the very end, 7654 x 7654 at 1e-1
// 103.2 instead of 102.2 and 1000 values 10.5 instead of 8.9.
constexpr int kPlaceCtas = 5;
template <int PER, int PART>
__global__ void __launch_bounds__(kTileThreads, kPlaceCtas)
place_strings_kernel(const TileStrings st, const TileArgs a, uint32_t* __restrict__ out, uint64_t* __restrict__ block_bits,
                     uint64_t* total_out) {
  constexpr int NB = kTileThreads * PER, kParts = NB / PART, kWords = PER == 4 ? 8 : 4;
  __shared__ unsigned long long s_sum[kTileWarps];
  __shared__ uint32_t s_warp[kTileWarps];
  __shared__ uint32_t s_bits[kTileThreads];                 // a string's length ...
  __shared__ uint32_t s_from[kTileThreads];                 // ... and start after the first one of the batch
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const bool wide = ((uintptr_t)block_bits & 15) == 0;
  const uint32_t t0 = (uint32_t)((uint64_t)a.tiles * blockIdx.x / gridDim.x);
  const uint32_t t1 = (uint32_t)((uint64_t)a.tiles * (blockIdx.x + 1) / gridDim.x);
  pdl_wait();
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
  pdl_trigger();

  for (uint32_t u0 = t0; u0 < t1; u0 += kTileThreads) {
    const uint32_t nu = t1 - u0 < kTileThreads ? t1 - u0 : kTileThreads;
    const uint32_t v = tid < nu ? st.tile_bits[u0 + tid] : 0;
    uint32_t x = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, x, d);
      if (lane >= d) x += y;
    }
    if (lane == 31) s_warp[warp] = x;
    __syncthreads();
    uint32_t from = x - v, all = 0;
#pragma unroll
    for (int w = 0; w < kTileWarps; w++) {
      if (w < warp) from += s_warp[w];
      all += s_warp[w];
    }
    s_bits[tid] = v;
    s_from[tid] = from;
    __syncthreads();
    // the caller's host thread waits for the stream's length: it gets it before the strings are moved
    if (total_out && u0 + nu == a.tiles && tid == 0) {
      *(volatile uint64_t*)total_out = base + all;
      __threadfence_system();
    }
#pragma unroll 1
    for (uint32_t item = warp; item < nu * kParts; item += kTileWarps) {
      const uint32_t k = item / kParts, part = item % kParts, tile = u0 + k, total = s_bits[k];
      const uint64_t start = base + s_from[k];
      const uint32_t* const src = st.strings + (uint64_t)tile * a.pitch;
      const uint32_t o = (uint32_t)(start & 31u), full = (o + total) >> 5;   // at most the string's words
      uint32_t* const dst = out + (start >> 5);
      // the offsets of two blocks a lane at a time, ahead of the words, and all of them ahead of their stores
      constexpr int kPairs = (PART + 63) / 64;
      const uint64_t b0 = (uint64_t)tile * NB + part * PART + 2 * lane, b1 = PART < 64 && lane >= PART / 2 ? 0 : a.blocks;
      uint32_t at[kPairs], from[kPairs];
#pragma unroll
      for (int j = 0; j < kPairs; j++) {
        const uint64_t b = b0 + 64 * j;
        at[j] = b + 1 < b1 ? *reinterpret_cast<const uint32_t*>(st.block_at + b) : b < b1 ? st.block_at[b] : 0u;
        from[j] = b < b1 ? st.warp_at[(uint64_t)tile * kTileWarps + (part * PART + 64 * j + 2 * lane) / (32 * PER)] : 0u;
      }
      const uint32_t each = (full + 32 * kParts - 1) / (32 * kParts) * 32, i0 = part * each, i1 = i0 + each < full ? i0 + each : full;
      uint32_t prev = 0;                                    // the word before this part's first
      if (part == 0) {
        if (tile) prev = last_bits(src - a.pitch, k ? s_bits[k - 1] : st.tile_bits[tile - 1]);
      } else if (i0 < i1) {
        prev = src[i0 - 1];
      }
      uint32_t carry = prev;
#pragma unroll 1
      for (uint32_t i = i0 + lane; i - lane < i1; i += 32 * kWords) {
        uint32_t here[kWords];
#pragma unroll
        for (int j = 0; j < kWords; j++) here[j] = i + 32 * j < i1 ? src[i + 32 * j] : 0u;
#pragma unroll
        for (int j = 0; j < kWords; j++) {
          uint32_t below = __shfl_up_sync(0xffffffffu, here[j], 1);
          if (lane == 0) below = carry;
          carry = __shfl_sync(0xffffffffu, here[j], 31);
          if (i + 32 * j < i1) dst[i + 32 * j] = __funnelshift_l(below, here[j], o);
        }
      }
#pragma unroll
      for (int j = 0; j < kPairs; j++) {
        const uint64_t b = b0 + 64 * j, first = start + from[j] + (at[j] & 0xffffu), second = start + from[j] + (at[j] >> 16);
        if (wide && b + 1 < b1) {
          *reinterpret_cast<ulonglong2*>(block_bits + b) = make_ulonglong2(first, second);
        } else {
          if (b < b1) block_bits[b] = first;
          if (b + 1 < b1) block_bits[b + 1] = second;
        }
      }
      if (tile + 1 == a.tiles && part == 0 && lane == 0) {
        block_bits[a.blocks] = start + total;
        close_stream(out, src, start, total, prev);
      }
    }
    base += all;
    __syncthreads();
  }
}

// 1-D tables in shared memory: the lean coder's windows and nibble pairs, and one plane per lookup.
// Before, with one plane per lookup throughout and a bit-matrix transpose per eight planes, 25.6 M values took: noise at
// tolerance 1e-6 121 us, with windows 101, with the straight line first 81; at 1e-3 95, 93, 70; at 6 bits/value 117, 97, 84; a
// random walk at 1e-6 218, 144, 135.
template <int DIM, int PER, bool BUDGET, int CTAS>
__global__ void __launch_bounds__(kTileThreads, CTAS)
decode_tiles_kernel(const uint32_t* in, float* __restrict__ out, const TileArgs a,
                    const uint64_t* block_bits, int shift, const uint16_t* __restrict__ plane_tab, const uint32_t* __restrict__ loop_tab) {
  constexpr int kPer = PER, WB = 32 * PER, NB = kTileThreads * PER;
  constexpr int kTabWords = DIM == 1 ? kTileDecTab1 : kRunTabSize;
  extern __shared__ __align__(16) uint32_t smem[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  uint32_t* const words = smem + kTabWords + warp * a.warp_words;
  const uint32_t cap = a.slot_words;
  pdl_trigger();
  if (DIM == 1) {
    for (int i = tid; i < 384; i += kTileThreads) reinterpret_cast<DecWindow*>(smem + kTileRows)[i] = make_tile_row(plane_tab, i);
    for (int i = tid; i < kDecTiny / 4; i += kTileThreads)   // windows and nibble pairs
      reinterpret_cast<uint4*>(smem)[i] = reinterpret_cast<const uint4*>(loop_tab)[i];
  } else {
    for (int i = tid; i < kRunTabSize / 4; i += kTileThreads) reinterpret_cast<uint4*>(smem)[i] = reinterpret_cast<const uint4*>(d_run.v)[i];
  }
  __syncthreads();
  pdl_wait();
  // 1-D: whether this warp tries the straight line. A block that leaves it costs the warp both forms, so a group with a few of
  // those ends the attempts: the next blocks are like these ones.
  bool straight = !BUDGET;
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
    for (uint32_t i = lane; i < nw; i += 32) words[i] = src[i];
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
        const bool left = !straight || !decode_code_1d(f, a.p, smem, words, pos, shift);
        if (left) decode_window_1d(f, a.p, smem, plane_tab, words, pos, shift);
        if (j == 0 && straight) straight = __popc(__ballot_sync(nb < 32 ? (1u << nb) - 1u : 0xffffffffu, left)) < kLeftMost;
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

TileArgs tile_args(const void* values, uint64_t nx, uint64_t ny, const ZfpParams& p, uint64_t blocks, int dim) {
  TileArgs a;
  a.nx = nx; a.ny = ny; a.blocks = blocks; a.p = p;
  a.bx = dim == 2 ? (uint32_t)((nx + 3) / 4) : 1;
  a.slot_words = a.warp_words = a.pitch = 0;
  a.wide = 0;
  a.row = divisor(a.bx);
  const uint64_t per = (uint64_t)kTileThreads * tile_per(blocks, dim);
  a.tiles = (uint32_t)((blocks + per - 1) / per);
  const uintptr_t base = (uintptr_t)values;
  if (dim == 1) a.vec = (base & 15) == 0 ? 4 : 1;
  else a.vec = (base & 15) == 0 && nx % 4 == 0 ? 4 : (base & 7) == 0 && nx % 2 == 0 ? 2 : 1;
  return a;
}

// Words of a warp's packed string or window.
uint32_t warp_words_for(const ZfpParams& p, uint64_t blocks, int dim) {
  return tile_per(blocks, dim) * max_block_bits(p, dim);     // 32 blocks per unit of it
}
struct TileScratch { uint64_t strings, warp_at, tile_bits, block_at, bytes; };   // byte offsets
TileScratch tile_scratch(const ZfpParams& p, uint64_t blocks, int dim) {
  const uint64_t per = (uint64_t)kTileThreads * tile_per(blocks, dim), tiles = (blocks + per - 1) / per;
  const uint64_t wb = per / kTileWarps, warps = (blocks + wb - 1) / wb;
  TileScratch t;
  t.tile_bits = 0;                                            // first: read 16 bytes at a time
  t.strings = (tiles * 4 + 15) & ~15ull;
  t.warp_at = t.strings + (blocks * max_block_bits(p, dim) + 31) / 32 * 4;
  t.block_at = t.warp_at + warps * 4;
  t.bytes = t.block_at + blocks * 2 + 16;                     // 16: the base is rounded up
  return t;
}
constexpr uint32_t kPackedPad = 4;                            // the word after the string, and whole 16-byte rows
constexpr uint32_t kReadAhead = kTileMaxBlockBits / 32 + 8;   // a block never reads further than this past its start
uint32_t round4(uint32_t v) { return (v + 3) & ~3u; }

// CTAs of a launch whose CTAs go through the tiles in steps of the grid: four times as many as are resident at once, by what
// registers, threads and shared memory allow. A number between two multiples of that leaves the GPU nearly empty at the end
// (2-D encoder, five per SM fit, six launched: a sixth of the work ran at one CTA per SM). Why four is said below.
template <auto kKernel>
int grid_of(uint32_t smem, uint32_t tiles, int* err) {
  static std::atomic<int> held[64];                         // by device: CTAs per SM that registers and threads allow, 0: not asked yet
  int dev = 0, most = 0;
  *err = (int)cudaGetDevice(&dev);
  if (*err) return 0;
  if (dev < 64) most = held[dev].load(std::memory_order_relaxed);
  if (!most) {
    *err = (int)cudaFuncSetAttribute(kKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    if (!*err) *err = (int)cudaOccupancyMaxActiveBlocksPerMultiprocessor(&most, kKernel, kTileThreads, 0);
    if (*err) return 0;
    if (most < 1) most = 1;
    if (dev < 64) held[dev].store(most, std::memory_order_relaxed);
  }
  const int fit = (int)(228u * 1024 / (smem + 1280));       // shared memory of an SM; 1280: the system's 1 KB and static arrays
  // Four CTAs per place: with one, every place takes the same number of tiles, and the last round of 25.6 M values at tolerance
  // 1e-6 (7.03 tiles a place) stood almost empty: round trip 233 us, with two 216, three 212, four 212, eight 214; a 7654 x 7654
  // field at 1e-3 297, 288, 284, 281, 279.
  const uint32_t g = 4u * 148u * (uint32_t)(fit < 1 ? 1 : fit < most ? fit : most);
  return (int)(tiles < g ? tiles : g);
}

// The coders' split between L1 and shared memory for the kernel behind them too: an SM whose next kernel wants another one has to run
// empty first (510 x 510 at tolerance 1e-3 and back 15.0 -> 13.9 us, 100 000 values at 1e-6 11.3 -> 10.3).
template <auto kKernel>
int all_shared() {
  static std::atomic<bool> done[64];                        // by device
  int dev = 0, err = (int)cudaGetDevice(&dev);
  if (err || (dev < 64 && done[dev].load(std::memory_order_relaxed))) return err;
  err = (int)cudaFuncSetAttribute(kKernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
  if (!err && dev < 64) done[dev].store(true, std::memory_order_relaxed);
  return err;
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

// Scratch of gcow_encode_tiles in bytes: 0 at fixed rate; else a length per tile, the tiles' strings (as many words as the longest
// possible stream), an offset per warp and one of 16 bits per block.
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
  const int per = tile_per(blocks, dim);
  const bool cuts = tile_budget_cuts(p, dim);
  const TileMode mode = !fixed ? kVariable : p.maxbits % 32 ? kPacked : kDirect;
  a.slot_words = tile_slot_words(p, dim);
  a.warp_words = mode == kDirect ? 0 : round4(warp_words_for(p, blocks, dim) + kPackedPad);
  a.wide = p.maxbits % 128 == 0 && ((uintptr_t)out & 15) == 0;
  const uint32_t slots = mode == kVariable ? 32 : 32 * per;
  const uint32_t smem = ((dim == 1 ? kEncPairTabSize : kTwinTabSize) + kTileWarps * (a.slot_words * slots + a.warp_words)) * 4;
  const TileScratch ts = tile_scratch(p, blocks, dim);
  char* const sp = (char*)(((uintptr_t)scratch + 15) & ~(uintptr_t)15);
  a.pitch = kTileWarps * per * max_block_bits(p, dim);
  TileStrings st = {};
  if (!fixed) st = {(uint32_t*)(sp + ts.strings), (uint32_t*)(sp + ts.tile_bits), (uint32_t*)(sp + ts.warp_at), (uint16_t*)(sp + ts.block_at)};
  int err = 0;
#define GCOW_ENCODE(D, P, F, B, C)                                                                                \
  do {                                                                                                         \
    const int g = grid_of<&encode_tiles_kernel<D, P, F, B, C>>(smem, a.tiles, &err);                              \
    if (err) return err;                                                                                       \
    launch_dependent(encode_tiles_kernel<D, P, F, B, C>, dim3(g), dim3(kTileThreads), smem, s, in, a, (uint32_t*)out, block_bits, st, \
                     (const uint16_t*)et, (const uint32_t*)pt);                                                \
  } while (0)
#define GCOW_ENCODE_MODE(D, P, B, C)                                    \
  do {                                                                \
    if (mode == kVariable) GCOW_ENCODE(D, P, kVariable, B, C);           \
    else if (mode == kPacked) GCOW_ENCODE(D, P, kPacked, B, C);          \
    else GCOW_ENCODE(D, P, kDirect, B, C);                               \
  } while (0)
  if (dim == 1 && mode == kVariable && !cuts) { if (per == 4) GCOW_ENCODE(1, 4, kVariable, false, 0); else GCOW_ENCODE(1, 1, kVariable, false, 0); }
  else if (dim == 1) { if (per == 4) GCOW_ENCODE_MODE(1, 4, true, 0); else GCOW_ENCODE_MODE(1, 1, true, 0); }
  else if (a.tiles > 4 * 148) { if (cuts) GCOW_ENCODE_MODE(2, 1, true, kCtas2d); else GCOW_ENCODE_MODE(2, 1, false, kCtas2d); }
  else if (cuts) GCOW_ENCODE_MODE(2, 1, true, 0);
  else GCOW_ENCODE_MODE(2, 1, false, 0);
#undef GCOW_ENCODE_MODE
#undef GCOW_ENCODE
  if (!fixed) {
    const uint32_t most = 148 * kPlaceCtas, g = a.tiles < most ? a.tiles : most;
    // Where every CTA has a tile of its own, one warp to an eighth of it.
#define GCOW_PLACE(P, N)                                                                                          \
  do {                                                                                                         \
    if ((err = all_shared<&place_strings_kernel<P, N>>())) return err;                                         \
    launch_dependent(place_strings_kernel<P, N>, dim3(g), dim3(kTileThreads), 0, s, st, a, (uint32_t*)out, block_bits, total_out); \
  } while (0)
    if (a.tiles > most) { if (per == 4) GCOW_PLACE(4, 256); else GCOW_PLACE(1, 128); }
    else if (per == 4) GCOW_PLACE(4, 128);
    else GCOW_PLACE(1, 32);
#undef GCOW_PLACE
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
  const int per = tile_per(blocks, dim);
  const bool cuts = tile_budget_cuts(p, dim);
  a.slot_words = warp_words_for(p, blocks, dim) + 1;                 // window capacity: one more for the bits before the first block
  a.warp_words = round4(a.slot_words + kReadAhead);
  const uint32_t smem = ((dim == 1 ? (uint32_t)kTileDecTab1 : (uint32_t)kRunTabSize) + kTileWarps * a.warp_words) * 4;
  int err = 0;
#define GCOW_DECODE(D, P, B, C)                                                                                      \
  do {                                                                                                         \
    const int g = grid_of<&decode_tiles_kernel<D, P, B, C>>(smem, a.tiles, &err);                                 \
    if (err) return err;                                                                                       \
    launch_dependent(decode_tiles_kernel<D, P, B, C>, dim3(g), dim3(kTileThreads), smem, s, (const uint32_t*)in, out, a, block_bits, shift, \
                     (const uint16_t*)dt, (const uint32_t*)lt);                                                \
  } while (0)
  if (dim == 1 && per == 4) { if (cuts) GCOW_DECODE(1, 4, true, 0); else GCOW_DECODE(1, 4, false, 0); }
  else if (dim == 1) { if (cuts) GCOW_DECODE(1, 1, true, 0); else GCOW_DECODE(1, 1, false, 0); }
  else if (a.tiles > 4 * 148) { if (cuts) GCOW_DECODE(2, 1, true, kCtas2d); else GCOW_DECODE(2, 1, false, kCtas2d); }
  else if (cuts) GCOW_DECODE(2, 1, true, 0);
  else GCOW_DECODE(2, 1, false, 0);
#undef GCOW_DECODE
  return (int)cudaGetLastError();
}

}  // extern "C"
