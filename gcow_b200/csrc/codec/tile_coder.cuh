// Block coders of the tile kernels (tile_kernels.cu): any mode, 1-D blocks of 4 and
// 2-D blocks of 4x4, host + device.
//
// A block is coded into 32-bit words of its own ("slot", word j at slot[j * stride])
// and read back from a window of 32-bit words at any bit position. Both use one
// property of the embedded coder: after a plane, the running count n is one past the
// highest coefficient that any plane so far has touched. A plane x therefore splits
// at n into verbatim bits and a rest r = x >> n, and the code of the rest is a
// function of r alone:
//   r == 0                one 0 bit (nothing when n == N)
//   otherwise, h = highest set bit of r:  a 1 bit, then the bits 0..h of r with a 1
//   inserted after every one-bit, the last inserted one turned into a 0; when n + h
//   is the last coefficient the final two bits are not sent (implied).
// (sw/src/encode.c:279-339 is the serial form: group tests and unary runs.)
#pragma once
#include "../divisor.h"
#include "zfp_block.cuh"

namespace gcow {

// The largest block the tile kernels take: the unpadded maximum of a 2-D block (9 header
// bits + 15 group tests + 16 * 32 plane bits = 536), rounded up to words.
constexpr uint32_t kTileMaxBlockBits = 544;

// Words of one slot: the longest unpadded code, or what may have been emitted when the budget is found to be exceeded
// (1-D: eight planes of at most seven bits at once, 2-D: one code of at most 32 bits), and one more written by the end.
inline uint32_t tile_slot_words(const ZfpParams& p, int dim) {
  const uint32_t n = dim == 1 ? 4 : 16, prec = p.maxprec < 32 ? p.maxprec : 32;
  const uint32_t natural = kHeaderBits + (n - 1) + n * prec;
  const uint32_t past = p.maxbits + (dim == 1 ? 55 : 31);
  return (natural <= p.maxbits || natural < past ? natural : past) / 32 + 1;
}
// Whether a block can reach maxbits.
inline bool tile_budget_cuts(const ZfpParams& p, int dim) {
  const uint32_t n = dim == 1 ? 4 : 16, prec = p.maxprec < 32 ? p.maxprec : 32;
  return kHeaderBits + (n - 1) + n * prec > p.maxbits;
}

// A rest's ones doubled, a byte at a time: entry v = the byte with every one-bit doubled, its length << 16.
constexpr int kTwinTabSize = 256;
GCOW_HD constexpr uint32_t make_twin_entry(uint32_t v) {
  uint32_t r = 0, len = 0;
  for (uint32_t i = 0; i < 8; i++) {
    const uint32_t b = (v >> i) & 1u;
    r |= (b * 3u) << len;
    len += 1 + b;
  }
  return r | (len << 16);
}
// The decoder's inverse, behind a positive group test: indexed by the next kRunBits bits of the stream, of which it takes as
// many tokens as are whole: "0" a zero, "11" a one with another positive test behind it, "10" the last one. Entry: the
// coefficients' bits | their number << 10 | bits used << 14 | 1 << 31 if the last one was among them.
constexpr int kRunBits = 10, kRunTabSize = 1 << kRunBits;
GCOW_HD constexpr uint32_t make_run_entry(uint32_t v) {
  uint32_t r = 0, used = 0, n = 0;
  while (used < (uint32_t)kRunBits) {
    if (!((v >> used) & 1u)) { used++; n++; continue; }
    if (used + 2 > (uint32_t)kRunBits) break;
    const uint32_t more = (v >> (used + 1)) & 1u;
    r |= 1u << n++;
    used += 2;
    if (!more) return r | (n << 10) | (used << 14) | 0x80000000u;
  }
  return r | (n << 10) | (used << 14);
}

template <int SIZE, uint32_t (*MAKE)(uint32_t)>
struct alignas(16) CodeTable {
  uint32_t v[SIZE];
  constexpr CodeTable() : v() { for (int i = 0; i < SIZE; i++) v[i] = MAKE((uint32_t)i); }
};
using TwinTable = CodeTable<kTwinTabSize, make_twin_entry>;
using RunTable = CodeTable<kRunTabSize, make_run_entry>;

// Bit i of the low half to bit 2i, and back (odd bits of the argument are ignored).
GCOW_HD uint32_t spread2(uint32_t x) {
  x = (x | (x << 8)) & 0x00ff00ffu;
  x = (x | (x << 4)) & 0x0f0f0f0fu;
  x = (x | (x << 2)) & 0x33333333u;
  return (x | (x << 1)) & 0x55555555u;
}
GCOW_HD uint32_t compact2(uint32_t x) {
  x &= 0x55555555u;
  x = (x | (x >> 1)) & 0x33333333u;
  x = (x | (x >> 2)) & 0x0f0f0f0fu;
  x = (x | (x >> 4)) & 0x00ff00ffu;
  return (x | (x >> 8)) & 0xffffu;
}

GCOW_HD uint32_t popc32(uint32_t x) {
#if defined(__CUDA_ARCH__)
  return (uint32_t)__popc(x);
#else
  return (uint32_t)__builtin_popcount(x);
#endif
}
GCOW_HD uint32_t funnel_l0(uint32_t v, uint32_t s) {   // the bits of v << s above bit 31, 0 <= s < 32
#if defined(__CUDA_ARCH__)
  return __funnelshift_l(v, 0u, s);
#else
  return s ? v >> (32 - s) : 0u;
#endif
}
GCOW_HD uint32_t window32(uint32_t lo, uint32_t hi, uint32_t s) {   // low word of (hi:lo) >> s, 0 <= s < 32
#if defined(__CUDA_ARCH__)
  return __funnelshift_r(lo, hi, s);
#else
  return s ? (lo >> s) | (hi << (32 - s)) : lo;
#endif
}

// Appends codes of up to 32 bits to a slot.
struct SlotWriter {
  uint32_t* at;        // next word
  uint32_t stride;
  uint32_t acc, fill;  // fill < 32 bits pending
  uint32_t full;       // bits in completed words
  GCOW_HD SlotWriter(uint32_t* slot, uint32_t s) : at(slot), stride(s), acc(0), fill(0), full(0) {}
  // the header and z zero bits behind it, 0 <= z <= 32, as the first thing in the slot
  GCOW_HD void begin(uint32_t head, uint32_t z) {
    acc = head;
    fill = kHeaderBits + z;
    if (fill >= 32) flush(0);
  }
  GCOW_HD void flush(uint32_t next) {
    *at = acc;
    at += stride;
    acc = next;
    fill -= 32;
    full += 32;
  }
  GCOW_HD void put(uint32_t code, uint32_t len) {       // len <= 32, code < 2^len
    acc |= code << fill;
    const uint32_t hi = funnel_l0(code, fill);
    fill += len;
    if (fill >= 32) flush(hi);
  }
  GCOW_HD uint32_t bits() const { return full + fill; }
};

// Ends a slot at `limit` bits (what lies past the budget is dropped) and returns its length.
GCOW_HD uint32_t finish_slot(const SlotWriter& s, uint32_t* slot, uint32_t stride, uint32_t limit) {
  uint32_t total = s.bits();
  *s.at = s.acc;
  if (total > limit) {
    total = limit;
    if (total & 31u) slot[(total >> 5) * stride] &= low_mask32(total & 31u);
  }
  return total;
}

// Cast of a block to integers relative to 2^(emax - 30). The clamping conversion (values out
// of range, NaN) is only needed where the block is not ordinary: a non-finite member or a vanishing maximum.
template <int N>
GCOW_HD void cast_block(int32_t* q, const float* f, int emax, bool ordinary) {
  const float scale = pow2f(30 - emax);
  if (ordinary) {
#pragma unroll
    for (int i = 0; i < N; i++) {
#if defined(__CUDA_ARCH__)
      q[i] = __float2int_rz(scale * f[i]);
#else
      q[i] = (int32_t)(scale * f[i]);
#endif
    }
  } else {
#pragma unroll
    for (int i = 0; i < N; i++) q[i] = trunc_to_i32(scale * f[i]);
  }
}
template <int N>
GCOW_HD int block_emax_fmax(const float* f) {              // block_emax with the hardware maximum (NaN members are skipped)
  float m = 0;
#pragma unroll
  for (int i = 0; i < N; i++) m = fmaxf(m, fabsf(f[i]));
  return scalar_exponent(m);
}
// The exponent of a block's largest magnitude (emax), NaN members skipped, and whether the plain conversion serves.
template <int N>
GCOW_HD int block_exponent(const float* f, bool& ordinary) {
  const uint32_t mb = block_max_bits<N>(f, 29, ordinary);    // scale * f is below 2^31 and the scale a normal float
  return ordinary ? (int)(mb >> 23) - 126 : block_emax_fmax<N>(f);
}

// ------------------------------------------------------------------- 1-D encoder
// The planes below the leading all-zero ones are coded two per lookup for the first eight, a
// last odd plane with the same table (the second plane masked away: an absent plane codes like a
// zero plane minus that plane's own zero bits), and verbatim nibbles follow once n >= 3.
GCOW_HD uint32_t encode_slot_1d(const float* f, const ZfpParams& p, const uint32_t* epair, const uint16_t* etab,
                                uint32_t* slot, uint32_t stride) {
  bool ordinary;
  const int emax = block_exponent<4>(f, ordinary);
  const uint32_t prec = block_precision(emax, p.maxprec, p.minexp, 1);
  const uint32_t biased = prec ? (uint32_t)(emax + kEBias) : 0;
  if (!biased) { *slot = 0; return 1; }
  int32_t q[4];
  uint32_t u[4];
  cast_block<4>(q, f, emax, ordinary);
  fwd_lift(q[0], q[1], q[2], q[3]);
#pragma unroll
  for (int i = 0; i < 4; i++) u[i] = int2nb(q[i]);
  const uint32_t planes = prec < 32u ? prec : 32u;
  const uint32_t mm = u[0] | u[1] | u[2] | u[3];
  uint32_t z = mm ? clz32(mm) : 32u;
  if (z > planes) z = planes;
  SlotWriter s(slot, stride);
  s.begin(2u * biased + 1u, z);
  uint32_t left = planes - z;
  if (left && s.bits() < p.maxbits) {                      // z < 32
    const uint32_t m = pow2_factor(z);
    const uint32_t R = byte_perm(byte_perm(u[0] * m, u[1] * m, 0x0073), byte_perm(u[2] * m, u[3] * m, 0x0073), 0x5410);
    // byte i = the next eight planes of coefficient i
    uint32_t n = 0;
    if (left >= 8) {
      uint32_t e[4], prev = 0;
#pragma unroll
      for (int j = 0; j < 4; j++) prev = e[j] = pair_entry(epair, R, j, prev);
      s.put(prepend_code(e[0], prepend_code(e[1], 0)), (e[0] + e[1]) & 63u);   // at most 28 bits
      s.put(prepend_code(e[2], prepend_code(e[3], 0)), (e[2] + e[3]) & 63u);
      n = (prev >> 8) & 0xffu;
      left -= 8;
      uint32_t k = 24 - z;                                 // planes k-1 .. k-left remain
      while (left && s.bits() < p.maxbits) {
        uint32_t T = plane_group8(u, k);
        uint32_t cnt = left < 8 ? left : 8;
        k -= cnt;
        left -= cnt;
        while (n < 3 && cnt) {                             // very smooth block: one plane per lookup
          const uint32_t e = etab[n * 16 + (T & 15u)];
          s.put(e & 0x7fu, (e >> 7) & 7u);
          n = e >> 10;
          T >>= 4;
          cnt--;
        }
        s.put(T & low_mask32(4 * cnt), 4 * cnt);
      }
    } else {
      uint32_t prev = 0;
#pragma unroll
      for (int j = 0; j < 4; j++) {
        if (left > 2u * j) {
          const bool single = left == 2u * j + 1;
          prev = pair_entry(epair, single ? R & 0xaaaaaaaau : R, j, prev);
          n = (prev >> 8) & 0xffu;
          uint32_t len = prev & 31u;
          if (single) len -= n < 4 ? n + 1 : 4u;
          s.put(prepend_code(prev, 0) & low_mask32(len), len);
        }
      }
    }
  }
  return finish_slot(s, slot, stride, p.maxbits);
}

// 64 bits to bit `at` of w, past what it holds; what leaves the 128 bits falls off.
GCOW_HD void append64(uint32_t (&w)[4], uint32_t at, uint32_t lo, uint32_t hi) {
  const uint32_t a = lo << (at & 31u), b = funnel_l(lo, hi, at), c = funnel_l0(hi, at & 31u);
  if (at >> 5 == 1u) { w[1] |= a; w[2] |= b; w[3] |= c; }   // ordinary data
  else if (at < 32u) { w[0] |= a; w[1] |= b; w[2] |= c; }
  else if (at < 96u) { w[2] |= a; w[3] |= b; }
  else if (at < 128u) w[3] |= a;
}
// The same code in registers, hardly a branch on ordinary data: the first eight planes behind the leading zeros two per lookup,
// the next eight likewise while n < 3, then verbatim nibbles. w: the code from bit 0, zeros past its `length`. False where the
// serial form above has to do it: a non-finite or tiny maximum, a NaN member, more than sixteen planes with n < 3 or
// sixteen verbatim ones, a code of more than 128 bits. No budget: the block's code must not reach maxbits.
GCOW_HD bool encode_code_1d(const float* f, const ZfpParams& p, const uint32_t* epair, uint32_t (&w)[4], uint32_t& length) {
  bool ok;
  const uint32_t mb = block_max_bits<4>(f, 29, ok), ex = mb >> 23;
  const float scale = bits_f32(0x8d800000u - (mb & 0xff800000u));   // 2^(30 - emax), emax = ex - 126; used with 29 <= ex <= 254
  const float p0 = scale * f[0], p1 = scale * f[1], p2 = scale * f[2], p3 = scale * f[3];
  const uint32_t prec = block_precision((int)ex - 126, p.maxprec, p.minexp, 1), planes = prec < 32u ? prec : 32u;
  if (planes == 0 || mb == 0) {                             // the block is a single 0 bit
    w[0] = w[1] = w[2] = w[3] = 0;
    length = 1;
    return true;
  }
  int32_t q[4];
#if defined(__CUDA_ARCH__)
  q[0] = __float2int_rz(p0); q[1] = __float2int_rz(p1); q[2] = __float2int_rz(p2); q[3] = __float2int_rz(p3);
#else
  if (!ok) return false;                                    // out of range for this conversion
  q[0] = (int32_t)p0; q[1] = (int32_t)p1; q[2] = (int32_t)p2; q[3] = (int32_t)p3;
#endif
  fwd_lift(q[0], q[1], q[2], q[3]);
  uint32_t u[4];
#pragma unroll
  for (int i = 0; i < 4; i++) u[i] = int2nb(q[i]);
  const uint32_t mm = u[0] | u[1] | u[2] | u[3];
  uint32_t z = mm ? clz32(mm) : 32u;
  if (z > planes) z = planes;
  const uint32_t left = planes - z, first = left < 8u ? left : 8u;
  ok = ok && z < 23u;                                       // the header's shift
  // A plane that the block does not have codes like a zero plane, min(n + 1, 4) zeros, which are taken off again.
  auto planes8 = [&](uint32_t at, uint32_t here, uint32_t prev, uint32_t& lo, uint32_t& hi, uint32_t& bits) {
    const uint32_t m = pow2_factor(at);
    const uint32_t R = byte_perm(byte_perm(u[0] * m, u[1] * m, 0x0073), byte_perm(u[2] * m, u[3] * m, 0x0073), 0x5410) &
                       (((0xff00u >> here) & 0xffu) * 0x01010101u);
    uint32_t e[4], sum = 0;
#pragma unroll
    for (int j = 0; j < 4; j++) sum += prev = e[j] = pair_entry(epair, R, j, prev);
    lo = hi = 0;
#pragma unroll
    for (int j = 3; j >= 0; j--) {
      hi = funnel_l(lo, hi, e[j]);
      lo = prepend_code(e[j], lo);
    }
    const uint32_t n = (prev >> 8) & 0xffu;
    bits = (sum & 0xffu) - (8u - here) * (n < 4u ? n + 1u : 4u);
    return prev;
  };
  uint32_t lo, hi, bits;
  uint32_t prev = planes8(z, first, 0, lo, hi, bits);
  const uint32_t s = kHeaderBits + z;
  w[0] = (2u * ex + 3u) | (lo << (s & 31u));                // flag bit + biased exponent (emax + 127 = ex + 1)
  w[1] = funnel_l(lo, hi, s);
  w[2] = funnel_l0(hi, s & 31u);
  w[3] = 0;
  length = s + bits;
  uint32_t k = 24u - z, rest = left - first;                // planes k-1 .. k-rest remain
  if (rest && ((prev >> 8) & 0xffu) < 3u) {
    const uint32_t next = rest < 8u ? rest : 8u;
    prev = planes8(z + 8u, next, prev & 0xff00u, lo, hi, bits);
    append64(w, length, lo, hi);
    length += bits;
    rest -= next;
    k -= 8u;
    ok = ok && (!rest || ((prev >> 8) & 0xffu) >= 3u);
  }
  if (rest) {                                               // verbatim nibbles
    const uint32_t t0 = plane_group8(u, k) & low_mask32(4u * rest);
    const uint32_t t1 = rest > 8u ? plane_group8(u, k - 8u) & low_mask32(4u * rest - 32u) : 0u;
    append64(w, length, t0, t1);
    length += 4u * rest;
  }
  return ok && rest <= 16u && length <= 128u;
}

// -------------------------------------------------------- 16 x 16 bit transposition
// In: w[j] = row j in the low half, row j + 8 in the high half (j = 0..7). Out: w[j] = column j
// in the low half, column j + 8 in the high half. The same function inverts itself.
GCOW_HD uint32_t select_bits(uint32_t a, uint32_t b, uint32_t m) { return (a & m) | (b & ~m); }
GCOW_HD void swap_quads(uint32_t* w, int a, int b, int s, uint32_t m) {
  const uint32_t x = w[a], y = w[b];
  w[a] = select_bits(x, y << s, m);
  w[b] = select_bits(x >> s, y, m);
}
GCOW_HD void transpose16(uint32_t* w) {
#pragma unroll
  for (int j = 0; j < 8; j++) w[j] = byte_perm(w[j], 0, 0x3120);   // bytes: row j low, row j+8 low, row j high, row j+8 high
#pragma unroll
  for (int j = 0; j < 4; j++) swap_quads(w, j, j + 4, 4, 0x0f0f0f0fu);
#pragma unroll
  for (int j = 0; j < 8; j++) if (!(j & 2)) swap_quads(w, j, j + 2, 2, 0x33333333u);
#pragma unroll
  for (int j = 0; j < 8; j += 2) swap_quads(w, j, j + 1, 1, 0x55555555u);
}
// After the transposition the low half of w[j] is column j of rows 0..15 read as bytes: rows 0..7 in
// byte 0, rows 8..15 in byte 1 - i.e. column j as a 16-bit word - and the high half is column j + 8.
GCOW_HD void transpose16_inv(uint32_t* w) {
#pragma unroll
  for (int j = 0; j < 8; j += 2) swap_quads(w, j, j + 1, 1, 0x55555555u);
#pragma unroll
  for (int j = 0; j < 8; j++) if (!(j & 2)) swap_quads(w, j, j + 2, 2, 0x33333333u);
#pragma unroll
  for (int j = 0; j < 4; j++) swap_quads(w, j, j + 4, 4, 0x0f0f0f0fu);
#pragma unroll
  for (int j = 0; j < 8; j++) w[j] = byte_perm(w[j], 0, 0x3120);
}

// ------------------------------------------------------------------- 2-D encoder
// On smooth data the first coefficient leads the others by many planes (3 to 9 on a 64 x 64 to 7654 x 7654 surface): as long
// as nothing else has been touched a plane is its bit and a 0, so the whole run is one bit-spread word instead of a step of
// the loop per plane. The planes behind it are taken sixteen at a time by one bit-matrix transposition, then one code per
// plane; `twin` is the table of make_twin_entry. kBudget: the block may have to be cut at maxbits.
// Bound by instructions (issue slots 69 % used). With every plane a step of the loop, and rests of more than eight bits
// doubled one bit at a time: 7654 x 7654 at tolerance 1e-3 184 -> 136 us, decoder 181 -> 130; 2047 x 3001 at 8 bits/value
// 30 -> 23 and 38 -> 25.
template <bool kBudget>
GCOW_HD uint32_t encode_slot_2d(const float* f, const ZfpParams& p, const uint32_t* twin, uint32_t* slot, uint32_t stride) {
  bool ordinary;
  const int emax = block_exponent<16>(f, ordinary);
  const uint32_t prec = block_precision(emax, p.maxprec, p.minexp, 2);
  const uint32_t biased = prec ? (uint32_t)(emax + kEBias) : 0;
  if (!biased) { *slot = 0; return 1; }
  int32_t q[16];
  uint32_t u[16];
  cast_block<16>(q, f, emax, ordinary);
  Xform<2>::fwd(q);
  fwd_reorder<2>(u, q);
  uint32_t others = 0;
#pragma unroll
  for (int i = 1; i < 16; i++) others |= u[i];
  const uint32_t planes = prec < 32u ? prec : 32u, mm = u[0] | others;
  uint32_t z = mm ? clz32(mm) : 32u, zo = others ? clz32(others) : 32u;
  if (z > planes) z = planes;
  if (zo > planes) zo = planes;
  SlotWriter s(slot, stride);
  s.begin(2u * biased + 1u, z);
  uint32_t n = 0, sh = z;
  if (zo > z && (!kBudget || s.bits() < p.maxbits)) {       // planes z .. zo-1 hold the first coefficient alone
    n = 1;
    sh = zo;
    uint32_t b = shr_sat(brev32(u[0]), z), run = zo - z, c = run < 15u ? run : 15u;
    s.put((spread2(b & low_mask32(c)) << 1) | 1u, 2 * c + 1);
    while ((run -= c) && (!kBudget || s.bits() < p.maxbits)) {
      b >>= c;
      c = run < 16u ? run : 16u;
      s.put(spread2(b & low_mask32(c)), 2 * c);
    }
  }
  int left = (int)(planes - sh);
#pragma unroll 1
  for (; left > 0 && (!kBudget || s.bits() < p.maxbits); sh += 16, left -= 16) {
    uint32_t w[8];
#pragma unroll
    for (int j = 0; j < 8; j++) w[j] = byte_perm(shl_sat(u[j], sh), shl_sat(u[j + 8], sh), 0x7632);   // the top halves
    transpose16(w);
#pragma unroll
    for (int t = 0; t < 16; t++) {
      if (t >= left) break;
      const uint32_t x = t < 8 ? w[7 - t] >> 16 : w[15 - t] & 0xffffu;
      const uint32_t r = x >> n;
      uint32_t code = x, len = n + (n < 16u ? 1u : 0u);
      if (r) {
        // 1, then the rest up to its highest one with the ones doubled, the last of them with a 0 in the twin's place
        const uint32_t e = twin[r & 0xffu];
        const uint32_t d = (e & 0xffffu) | ((twin[r >> 8] & 0xffffu) << (e >> 16));
        const uint32_t top = 32u - clz32(d);
        code = (x & ((1u << n) - 1u)) | (((2u * d + 1u) ^ shl_sat(1u, top)) << n);
        len = n + top + 1u;
        n += 32u - clz32(r);
        if (n == 16u) {                                     // the last coefficient: its one-bit is implied, no closing test
          len -= 2u;
          code &= (1u << len) - 1u;
        }
      }
      s.put(code, len);
      if (kBudget && s.bits() >= p.maxbits) break;
    }
  }
  return finish_slot(s, slot, stride, kBudget ? p.maxbits : 0xffffffffu);
}

// ---------------------------------------------------------------------- decoders
// Window of 32-bit words read at any bit position; the caller guarantees two readable words after
// the last one that holds bits of the block.
struct WindowReader {
  const uint32_t* w;   // the word after `hi`
  uint32_t lo, hi, o;  // o < 32: position in lo
  GCOW_HD WindowReader(const uint32_t* words, uint32_t pos) : w(words + (pos >> 5) + 2), o(pos & 31u) { lo = w[-2]; hi = w[-1]; }
  GCOW_HD uint32_t peek() const { return window32(lo, hi, o); }
  GCOW_HD void skip(uint32_t n) {                          // n <= 32
    o += n;
    if (o >= 32) {
      lo = hi;
      hi = *w++;
      o -= 32;
    }
  }
};

// One block of 4 from a window. `tab`: the lean coder's decoder windows and nibble pairs, then at kTileRows one plane per
// lookup in the same form (rows n = 0..2 of 128 entries, the next seven bits) for where a window would run past the last
// plane or the budget; `dtab`: the decoder's budget table, for the last bits of a budget (may be global memory). Planes gather
// in U, byte i those of coefficient i; once n >= 3 the rest is verbatim nibbles, two per lookup.
constexpr int kTileRows = kDecTiny, kTileDecTab1 = kTileRows + 3 * 128 * 2;
// Entry i (0..383) of the one-plane rows, from the decoder's budget table.
GCOW_HD DecWindow make_tile_row(const uint16_t* dtab, uint32_t i) {
  const uint32_t e = dtab[((i >> 7) * 8 + 7) * 128 + (i & 127)], n = e >> 7;
  return {spread_nibble(e & 15u), 1u | (n < 3 ? (n + 1) << 12 : 0u) | ((e >> 4) & 7u) << 16};
}
GCOW_HD void decode_window_1d(float* f, const ZfpParams& p, const uint32_t* tab, const uint16_t* dtab, const uint32_t* words,
                              uint32_t pos, int shift) {
  WindowReader src(words, pos);
  const uint32_t head = src.peek();
  if (!(head & 1u)) {
    f[0] = f[1] = f[2] = f[3] = 0;
    return;
  }
  const int emax = (int)((head >> 1) & 0xffu) - kEBias;
  const uint32_t prec = block_precision(emax, p.maxprec, p.minexp, 1), planes = prec < 32u ? prec : 32u;
  uint32_t bits = p.maxbits - kHeaderBits;                 // budget left
  src.skip(kHeaderBits);
  const uint32_t S = src.peek();                           // leading all-zero planes
  uint32_t z = S ? (uint32_t)ctz32(S) : 32u;
  if (z > planes) z = planes;
  if (z > bits) z = bits;
  src.skip(z);
  bits -= z;
  const uint32_t* const nib = tab + kDecNibbles;
  uint32_t u[4] = {0, 0, 0, 0};
  uint32_t U = 0, held = 0, gone = z, row = 0x1000;        // planes in U; planes above the next one; (n + 1) * 4096, 0 once n >= 3
  auto flush = [&]() {                                     // U to its place: the planes down to 32 - gone
    const uint32_t m = pow2_factor(32u - gone);
    u[0] += (U & 0xffu) * m; u[1] += ((U >> 8) & 0xffu) * m; u[2] += ((U >> 16) & 0xffu) * m; u[3] += (U >> 24) * m;
    U = held = 0;
  };
  while (row && gone < planes && bits) {
    if (held > 3) flush();                                 // at most seven planes: the tail wants the bytes' top bits clear
    const bool wide = planes - gone >= 4 && bits >= 9;     // a window holds at most four planes and nine bits
    if (wide || bits >= 7) {
      const uint32_t v = src.peek(), at = wide ? row - 0x1000u + 8u * (v & 511u) : kTileRows * 4u + ((row - 0x1000u) >> 2) + 8u * (v & 127u);
      const DecWindow d = *reinterpret_cast<const DecWindow*>(reinterpret_cast<const char*>(tab) + at);
      const uint32_t n = d.meta & 15u, used = d.meta >> 16;
      U = (U << n) | d.u;
      held += n;
      gone += n;
      src.skip(used);
      bits -= used;
      row = d.meta & 0x3000u;
    } else {                                               // the budget may end inside this plane
      const uint32_t e = dtab[((((row >> 12) - 1u) * 8 + bits) << 7) + (src.peek() & low_mask32(bits))], used = (e >> 4) & 7u, n = e >> 7;
      U = 2 * U + (nib[e & 15u] >> 1);
      held++;
      gone++;
      src.skip(used);
      bits -= used;
      row = n < 3 ? (n + 1) << 12 : 0u;
    }
  }
  // A nibble cut by the budget after its first three bits: with n == 3 the missing bit is a group test that reads as 0,
  // with n == 4 a verbatim bit that reads as 0 - the same nibble.
  const uint32_t want = 4 * (planes - gone), tail = want < bits ? want : bits;
  if (tail | U) {
    const uint32_t t = src.peek() & low_mask32(tail);
    const uint32_t W = ((nib[t & 255u] * 4u + nib[(t >> 8) & 255u]) * 4u + nib[(t >> 16) & 255u]) * 4u + nib[t >> 24];
    const uint32_t m = gone < 24u ? pow2_factor(24u - gone) : 1u, r = gone < 24u ? 0u : gone - 24u;
    u[0] += shr_sat(byte_perm_sx(W, U, 0xcc40) * m, r); u[1] += shr_sat(byte_perm_sx(W, U, 0xdd51) * m, r);
    u[2] += shr_sat(byte_perm_sx(W, U, 0xee62) * m, r); u[3] += shr_sat(byte_perm_sx(W, U, 0xff73) * m, r);
  }
  if (tail > 32) {                                         // more than eight planes left: gone < 24
    src.skip(32);
    const uint32_t t = src.peek() & low_mask32(tail - 32), k = 24u - gone;
    const uint32_t V = ((nib[t & 255u] * 4u + nib[(t >> 8) & 255u]) * 4u + nib[(t >> 16) & 255u]) * 4u + nib[t >> 24];
    u[0] |= shr_sat(V << 24, 32u - k); u[1] |= shr_sat((V & 0xff00u) << 16, 32u - k);
    u[2] |= shr_sat((V & 0xff0000u) << 8, 32u - k); u[3] |= shr_sat(V & 0xff000000u, 32u - k);
    for (uint32_t done = 64, kk = k - 8; done < tail; done += 32, kk -= 8) {
      src.skip(32);
      deposit_group8(u, src.peek() & low_mask32(tail - done), kk);
    }
  }
  int32_t q[4];
#pragma unroll
  for (int i = 0; i < 4; i++) q[i] = nb2int(u[i]);
  inv_lift(q[0], q[1], q[2], q[3]);
  inv_cast<4>(f, q, emax, shift);
}

// The same as a straight line, for blocks that no budget cuts. What a block ends with need not be found: its planes below the
// last one are read from whatever follows it and masked off. False (f is not written) where the loop above has to do it:
// more than three windows or seven planes with n < 3, more than 23 leading zero planes, a code past the 96 bits held.
GCOW_HD bool decode_code_1d(float* f, const ZfpParams& p, const uint32_t* tab, const uint32_t* words, uint32_t pos, int shift) {
  const uint32_t* const w = words + (pos >> 5);
  const uint32_t o = pos & 31u, w1 = w[1], w2 = w[2];
  uint32_t x0 = window32(w[0], w1, o), x1 = window32(w1, w2, o), x2 = window32(w2, w[3], o);
  const uint32_t head = x0;
  if (!(head & 1u)) {
    f[0] = f[1] = f[2] = f[3] = 0;
    return true;
  }
  const uint32_t e8 = (head >> 1) & 0xffu;                   // emax + 127
  const uint32_t prec = block_precision((int)e8 - kEBias, p.maxprec, p.minexp, 1), planes = prec < 32u ? prec : 32u;
  auto skip = [&](uint32_t n) {                            // n < 32
    x0 = window32(x0, x1, n);
    x1 = window32(x1, x2, n);
    x2 >>= n;
  };
  skip(kHeaderBits);
  const uint32_t z = (uint32_t)ctz32(x0 | 0x1000000u);
  if (planes > z + 23u || shift < -29) return false;       // more than sixteen verbatim; 2^(emax - 30 - shift) may be infinite
  skip(z);
  uint32_t U = 0, row = 0x1000, sum = (kHeaderBits + z) << 16; // the sum as in decode_block_1d_try
#pragma unroll
  for (int c = 0; c < 3; c++) {
    if (c == 0 || (row && z + (sum & 0xffu) < planes)) {
      const DecWindow d = *reinterpret_cast<const DecWindow*>(reinterpret_cast<const char*>(tab) + (row - 0x1000u) + 8u * (x0 & 511u));
      U = c ? funnel_l(0u, U, d.meta) | d.u : d.u;
      row = d.meta & 0x3000u;
      sum += d.meta;
      skip(d.meta >> 16);
    }
  }
  const uint32_t gone = z + (sum & 0xffu);
  const int rest = (int)(planes - gone), used = (int)(sum >> 16);   // verbatim planes; below 0: read too far, which the mask undoes
  if (!((!row || rest <= 0) && (sum & 0xffu) <= 7u && z < 24u && rest <= 16 && used + 4 * rest <= 96)) return false;
  const uint32_t* const nib = tab + kDecNibbles;
  const uint32_t W = ((nib[x0 & 255u] * 4u + nib[(x0 >> 8) & 255u]) * 4u + nib[(x0 >> 16) & 255u]) * 4u + nib[x0 >> 24];
  const uint32_t m = gone < 24u ? pow2_factor(24u - gone) : 1u, r = gone < 24u ? 0u : gone - 24u;
  uint32_t u[4];
  u[0] = shr_sat(byte_perm_sx(W, U, 0xcc40) * m, r); u[1] = shr_sat(byte_perm_sx(W, U, 0xdd51) * m, r);
  u[2] = shr_sat(byte_perm_sx(W, U, 0xee62) * m, r); u[3] = shr_sat(byte_perm_sx(W, U, 0xff73) * m, r);
  if (rest > 8) {                                          // gone < 24
    const uint32_t k = 24u - gone;
    uint32_t V = (nib[x1 & 255u] * 4u + nib[(x1 >> 8) & 255u]) * 16u;
    if (rest > 12) V += nib[(x1 >> 16) & 255u] * 4u + nib[x1 >> 24];
    u[0] |= shr_sat(V << 24, 32u - k); u[1] |= shr_sat((V & 0xff00u) << 16, 32u - k);
    u[2] |= shr_sat((V & 0xff0000u) << 8, 32u - k); u[3] |= shr_sat(V & 0xff000000u, 32u - k);
  }
  const uint32_t mask = ~shr_sat(0xffffffffu, planes);
  int32_t q[4];
#pragma unroll
  for (int i = 0; i < 4; i++) q[i] = nb2int(u[i] & mask);
  inv_lift(q[0], q[1], q[2], q[3]);
  const int ef = (int)e8 - 30 - shift;                     // a normal float unless the block is tiny
  const float scale = bits_f32(ef >= 1 ? (uint32_t)ef << 23 : shl_sat(1u, (uint32_t)(ef + 22)));
#pragma unroll
  for (int i = 0; i < 4; i++) f[i] = scale * (float)q[i];
  return true;
}

// One plane of 16 coefficients whose code the budget cuts: bit by bit. A one-bit that is pending where the bits end is placed.
GCOW_HD uint32_t cut_plane_2d(uint32_t b, uint32_t n, uint32_t bits) {
  const uint32_t m = n < bits ? n : bits;
  uint32_t x = b & low_mask32(m);
  b = shr_sat(b, m);
  bits -= m;
  while (bits && n < 16) {
    bits--;
    const uint32_t test = b & 1u;
    b >>= 1;
    if (!test) break;
    while (bits && n < 15) {
      bits--;
      const uint32_t one = b & 1u;
      b >>= 1;
      if (one) break;
      n++;
    }
    x += 1u << n;
    n++;
  }
  return x;
}

// One block of 4x4 from a window of 32-bit words starting at bit `pos`. The run of planes that hold the first coefficient alone
// is read by its pattern (see the encoder), the others are collected as 16-bit words and turned back into coefficients by
// the bit-matrix transposition. `run`: the table of make_run_entry.
template <bool kBudget>
GCOW_HD void decode_window_2d(float* f, const ZfpParams& p, const uint32_t* run, const uint32_t* words, uint32_t pos, int shift) {
  WindowReader src(words, pos);
  const uint32_t head = src.peek();
  if (!(head & 1u)) {
#pragma unroll
    for (int j = 0; j < 16; j++) f[j] = 0;
    return;
  }
  const int emax = (int)((head >> 1) & 0xffu) - kEBias;
  const uint32_t prec = block_precision(emax, p.maxprec, p.minexp, 2);
  const uint32_t planes = prec < 32u ? prec : 32u;
  uint32_t bits = p.maxbits - kHeaderBits;                 // budget left
  src.skip(kHeaderBits);
  const uint32_t S = src.peek();
  uint32_t z = S ? (uint32_t)ctz32(S) : 32u;
  if (z > planes) z = planes;
  if (kBudget && z > bits) z = bits;
  src.skip(z);
  if (kBudget) bits -= z;
  uint32_t u[16];
#pragma unroll
  for (int j = 0; j < 16; j++) u[j] = 0;
  uint32_t n = 0, sh = z, b = src.peek();
  if ((b & 3u) == 3u) {                                    // the first coefficient: its bits and negative group tests in turn
    uint32_t skip = 1, most = 15, c;
    b >>= 1;
    do {
      const uint32_t tests = b & 0xaaaaaaaau;
      c = tests ? (uint32_t)ctz32(tests) >> 1 : most;
      if (c > most) c = most;
      if (c > planes - sh) c = planes - sh;
      if (kBudget && 2 * c + skip > bits) c = bits > skip ? (bits - skip) >> 1 : 0u;
      if (!c) break;
      u[0] |= shr_sat(brev32(compact2(b & low_mask32(2 * c))), sh);
      n = 1;
      sh += c;
      if (kBudget) bits -= 2 * c + skip;
      src.skip(2 * c + skip);
      if (c < most) break;
      b = src.peek();
      skip = 0;
      most = 16;
    } while (true);
  }
  int left = (int)(planes - sh);
  uint32_t nmask = n;                                      // the low n bits
#pragma unroll 1
  for (; left > 0 && (!kBudget || bits); sh += 16, left -= 16) {
    uint32_t w[8];
#pragma unroll
    for (int j = 0; j < 8; j++) w[j] = 0;
#pragma unroll
    for (int t = 0; t < 16; t++) {
      if (t >= left || (kBudget && !bits)) break;
      b = src.peek();
      uint32_t x = b & nmask, used = n, m = n;
      if (n < 16) {
        uint32_t e = b >> n;
        used = n + 1;
        if (e & 1u) {                                      // a positive group test: tokens up to the last one
          uint32_t r = 0, c = 0, entry;
          e >>= 1;
          do {
            entry = run[e & (uint32_t)(kRunTabSize - 1)];
            r |= (entry & 0x3ffu) << c;
            c += (entry >> 10) & 15u;
            const uint32_t k = (entry >> 14) & 15u;
            e >>= k;
            used += k;
          } while (!(entry >> 31) && n + c < 15u);
          m = n + c;
          if (m > 15u || !(entry >> 31)) {                 // the last coefficient: its one-bit is implied and no test follows
            r &= (1u << (15u - n)) - 1u;
            used = 16u + popc32(r);                        // n bits, a test, a bit per coefficient before it, a test per one
            r |= 1u << (15u - n);
            m = 16;
          }
          x |= r << n;
        }
      }
      if (kBudget && used > bits) {
        x = cut_plane_2d(b, n, bits);
        used = bits;
      }
      n = m;
      nmask = (1u << n) - 1u;
      if (kBudget) bits -= used;
      src.skip(used);
      if (t < 8) w[7 - t] |= x << 16; else w[15 - t] |= x;
    }
    transpose16_inv(w);
#pragma unroll
    for (int j = 0; j < 8; j++) {
      u[j] |= shr_sat(w[j] << 16, sh);
      u[j + 8] |= shr_sat(w[j] & 0xffff0000u, sh);
    }
  }
  int32_t q[16];
  inv_reorder<2>(q, u);
  Xform<2>::inv(q);
  inv_cast<16>(f, q, emax, shift);
}

}  // namespace gcow
