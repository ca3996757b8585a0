// Register-level BC4 decode shared by the decode GEMV and the prefill GEMM producers.
#pragma once

#include "tx_common.cuh"

namespace tx {

__device__ __forceinline__ uint4 lds128(unsigned addr) {
  uint4 v;
  asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
  return v;
}
__device__ __forceinline__ uint4 ldg_stream(const uint4 *p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.b32 {%0,%1,%2,%3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ void mma_f16(float (&c)[4], unsigned a0, unsigned a1, unsigned a2, unsigned a3,
                                        unsigned b0, unsigned b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ unsigned hfma2_u(unsigned a, unsigned b, unsigned c) {
  unsigned d;
  asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
}
// (a & mask) | c as one LOP3
__device__ __forceinline__ unsigned and_or(unsigned a, unsigned mask, unsigned c) {
  unsigned d;
  asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(d) : "r"(a), "r"(mask), "r"(c));
  return d;
}
__device__ __forceinline__ unsigned hsub2_u(unsigned a, unsigned b) {
  unsigned d;
  asm("sub.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}

__device__ __forceinline__ unsigned hmul2_u(unsigned a, unsigned b) {
  unsigned d;
  asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}

// ---------------------------------------------------------------------------------------------
// Numerators.  Every decode kernel hands the tensor core the exact integers n = 7*e0 + g*(e1-e0)
// (|n| <= 889) scaled by 2^-16, as fp16: n * 2^-16 is a multiple of 2^-24 below 2^-6, hence exact in
// fp16 (subnormal below 2^-14; HFMA2 and the tensor cores take subnormal fp16 operands at full
// speed).  The epilogues multiply by kNumeratorScale * scale_m * (token scaling).
//
// Per block: base = 7*e0 * 2^-16 and three multipliers delta * 2^(8-p) for the field offsets p = 0, 3, 6
// (a field at offset p, masked in place, reads as g * 2^(p-24); the product with delta * 2^(8-p) is
// g*delta * 2^-16; delta * 256 <= 65024 still fits fp16).  Fields at offsets 10 and 13 come down to 0
// and 3 with one shift.  The pair kept in the spare bits is summed from its three bit planes with
// multipliers delta/2, delta, 2*delta (bit 9 reads as 2^-15).
// ---------------------------------------------------------------------------------------------
constexpr float kNumeratorScale = 65536.0f / 889.0f;   // numerators are n * 2^-16, palette value = n / 889

constexpr unsigned kField0 = 0x00070007u, kField3 = 0x00380038u, kField6 = 0x01C001C0u, kFieldSpare = 0x02000200u;

// Both blocks of a duo at once: low halves belong to the first block, high halves to the second.  The multiply-adds pick
// their half by an operand swizzle, so the constants cost seven instructions a duo instead of seven a block.
struct DuoConstants {
  unsigned base, d0, d3, d6, delta;   // fp16x2
  unsigned m0, m3, m6;                // per majority bit (texture weights only)
};
__device__ __forceinline__ unsigned half_of(unsigned v, int second) {
  const __half2 h = *reinterpret_cast<const __half2 *>(&v);
  const __half2 both = second ? __high2half2(h) : __low2half2(h);
  return *reinterpret_cast<const unsigned *>(&both);
}

// TEXTURE_WEIGHTS: the texture unit's interpolation weights are {0,36,72,114,144,186,222,258}/258 for
// g = 0..7, i.e. (36*g + 6*majority(bits of g))/258; the fast path then uses delta * 252/258 per g step
// plus delta * 42/258 per majority bit, both rounded to fp16 (relative error <= 2^-11; the 16-bit
// widening of the endpoints, 3e-5, is neglected -- tx_dequant and the exact kernels evaluate the
// texture palette exactly).
template <bool TEXTURE_WEIGHTS>
__device__ __forceinline__ DuoConstants duo_constants(unsigned ends) {
  const unsigned e0m = __byte_perm(ends, 0x64646464u, 0x4240);   // fp16x2 (1024+u0) of the first and second block
  const unsigned e1m = __byte_perm(ends, 0x64646464u, 0x4341);
  DuoConstants c;
  c.base = hfma2_u(e0m, 0x07000700u /* 7 * 2^-16 */, 0xAFE0AFE0u /* -8064 * 2^-16 */);   // 7*(u0-128) * 2^-16
  unsigned delta = hsub2_u(e1m, e0m);                              // e1 - e0, exact
  if (TEXTURE_WEIGHTS) delta = hmul2_u(delta, 0x3BD03BD0u);        // * 252/258 = 0.976744 -> fp16 0x3BD0
  c.delta = delta;
  c.d0 = hmul2_u(delta, 0x5C005C00u);                              // * 256
  c.d3 = hmul2_u(delta, 0x50005000u);                              // * 32
  c.d6 = hmul2_u(delta, 0x44004400u);                              // * 4
  c.m0 = c.m3 = c.m6 = 0;
  if (TEXTURE_WEIGHTS) {                                           // d carries 252/258: 42/252 = 1/6
    c.m0 = hmul2_u(c.d0, 0x31553155u);
    c.m3 = hmul2_u(c.d3, 0x31553155u);
    c.m6 = hmul2_u(c.d6, 0x31553155u);
  }
  return c;
}

// majority of the three bits of every field, left at the field's lowest bit (texture weights only)
__device__ __forceinline__ unsigned field_majority(unsigned w, unsigned low_bits) {
  unsigned m;
  const unsigned w1 = w >> 1, w2 = w >> 2;
  asm("lop3.b32 %0, %1, %2, %3, 0xE8;" : "=r"(m) : "r"(w), "r"(w1), "r"(w2));
  return m & low_bits;
}

// BIT: offset of the field
template <bool TEXTURE_WEIGHTS, int BIT>
__device__ __forceinline__ unsigned numerators(unsigned word, const DuoConstants &c, int second) {
  constexpr unsigned mask = 0x00070007u << BIT, low_bits = 0x00010001u << BIT;
  const unsigned multiplier = BIT == 0 ? c.d0 : BIT == 3 ? c.d3 : c.d6;
  unsigned n = hfma2_u(word & mask, half_of(multiplier, second), half_of(c.base, second));
  if (TEXTURE_WEIGHTS) n = hfma2_u(field_majority(word, low_bits), half_of(BIT == 0 ? c.m0 : BIT == 3 ? c.m3 : c.m6, second), n);
  return n;
}

// The eight fp16x2 numerator pairs (weights 2i, 2i+1 in pair i) of the first / second block of a duo.
// High palette mode only; blocks with e0 <= e1 are redone by decode_block_low.
template <bool TEXTURE_WEIGHTS = false>
__device__ __forceinline__ void decode_duo_first(const uint4 duo, const DuoConstants &c, unsigned (&a)[8]) {
  const unsigned s0 = duo.x >> 10;
  a[0] = numerators<TEXTURE_WEIGHTS, 0>(duo.x, c, 0);
  a[1] = numerators<TEXTURE_WEIGHTS, 3>(duo.x, c, 0);
  a[2] = numerators<TEXTURE_WEIGHTS, 6>(duo.x, c, 0);
  a[3] = numerators<TEXTURE_WEIGHTS, 0>(s0, c, 0);
  a[4] = numerators<TEXTURE_WEIGHTS, 3>(s0, c, 0);
  a[5] = numerators<TEXTURE_WEIGHTS, 0>(duo.y, c, 0);
  a[6] = numerators<TEXTURE_WEIGHTS, 3>(duo.y, c, 0);
  a[7] = numerators<TEXTURE_WEIGHTS, 6>(duo.y, c, 0);
}

template <bool TEXTURE_WEIGHTS = false>
__device__ __forceinline__ void decode_duo_second(const uint4 duo, const DuoConstants &c, unsigned (&a)[8]) {
  const unsigned s1 = duo.y >> 10, s2 = duo.z >> 10;
  a[0] = numerators<TEXTURE_WEIGHTS, 0>(s1, c, 1);
  a[1] = numerators<TEXTURE_WEIGHTS, 3>(s1, c, 1);
  a[2] = numerators<TEXTURE_WEIGHTS, 0>(duo.z, c, 1);
  a[3] = numerators<TEXTURE_WEIGHTS, 3>(duo.z, c, 1);
  a[4] = numerators<TEXTURE_WEIGHTS, 6>(duo.z, c, 1);
  a[5] = numerators<TEXTURE_WEIGHTS, 0>(s2, c, 1);
  a[6] = numerators<TEXTURE_WEIGHTS, 3>(s2, c, 1);
  // pair 7: bit k of both g values is the spare bit of word k (reads as 2^-15 per set bit)
  const unsigned half_delta = hmul2_u(c.delta, 0x38003800u), twice_delta = hmul2_u(c.delta, 0x40004000u);
  unsigned n = hfma2_u(duo.x & kFieldSpare, half_of(half_delta, 1), half_of(c.base, 1));
  n = hfma2_u(duo.y & kFieldSpare, half_of(c.delta, 1), n);
  n = hfma2_u(duo.z & kFieldSpare, half_of(twice_delta, 1), n);
  if (TEXTURE_WEIGHTS) {
    // majority of the three planes, at the spare bit: * delta * (1/2) * (1/6)
    unsigned m;
    asm("lop3.b32 %0, %1, %2, %3, 0xE8;" : "=r"(m) : "r"(duo.x), "r"(duo.y), "r"(duo.z));
    n = hfma2_u(m & kFieldSpare, half_of(hmul2_u(c.delta, 0x2D552D55u /* 1/12 */), 1), n);
  }
  a[7] = n;
}

// Low-mode blocks (e0 <= e1; about a fifth of the blocks of a 90 %-sparse matrix, so nearly every unit of such a matrix
// holds some).  Their eight palette entries do not lie on one line, so they are looked up: the entries, palette * 889 * 2^-16
// rounded to fp16, become two 8-byte tables (low and high bytes), and one byte permute takes four of them by the index
// fields.  About 90 instructions a block; the per-weight arithmetic that did this before took about 500 (4250x2896, nine
// weights of ten zero, 29 tokens: 53.4 -> 18.4 us a call).
__device__ __forceinline__ unsigned prmt_u(unsigned a, unsigned b, unsigned selector) {
  unsigned d;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(selector));
  return d;
}
struct LowTable {
  unsigned low0, low1, high0, high1;   // low bytes of entries 0-3 and 4-7, high bytes of the same
  // the fp16x2 values of two pairs of weights from their indices (each at bits 0-2 and 16-18 of its word)
  __device__ __forceinline__ void lookup(unsigned fa, unsigned fb, unsigned &a, unsigned &b) const {
    const unsigned wide = fa | (fb << 4), selector = wide | (wide >> 8);   // nibbles: a even, b even, a odd, b odd
    const unsigned low = prmt_u(low0, low1, selector), high = prmt_u(high0, high1, selector);
    a = prmt_u(low, high, 0x6240);
    b = prmt_u(low, high, 0x7351);
  }
};
// entries in the order of the stored index (0: e0, 7: e1, 1..4: between them, 5 and 6: -1 and +1)
__device__ __forceinline__ LowTable low_table(unsigned ends, int palette) {
  const int e0 = int(ends & 0xffu) - 128, e1 = int((ends >> 8) & 0xffu) - 128, d = e1 - e0;
  const bool hardware = palette == TX_PALETTE_HARDWARE;   // uniform
  float den = 635.0f, rcp = 1.0f / 635.0f;
  int first = 5 * e0, last = 5 * e1, step = d;
  if (hardware) {
    den = 32767.0f;
    rcp = 1.0f / 32767.0f;
    first = widen_snorm8(e0);
    last = widen_snorm8(e1);
    step = 48 * d;
  }
  // (the texture unit counts the upper two entries from the far endpoint)
  const int n[6] = {first, first + step, first + 2 * step, hardware ? last - 2 * step : first + 3 * step,
                    hardware ? last - step : first + 4 * step, last};
  float v[6];
#pragma unroll
  for (int i = 0; i < 6; ++i) v[i] = rn_div_const(float(n[i]), den, rcp) * (889.0f / 65536.0f);
  const __half2 h01 = __floats2half2_rn(v[0], v[1]), h23 = __floats2half2_rn(v[2], v[3]);
  const __half2 h45 = __floats2half2_rn(v[4], -889.0f / 65536.0f), h67 = __floats2half2_rn(889.0f / 65536.0f, v[5]);
  const unsigned t01 = *reinterpret_cast<const unsigned *>(&h01), t23 = *reinterpret_cast<const unsigned *>(&h23);
  const unsigned t45 = *reinterpret_cast<const unsigned *>(&h45), t67 = *reinterpret_cast<const unsigned *>(&h67);
  return {prmt_u(t01, t23, 0x6420), prmt_u(t45, t67, 0x6420), prmt_u(t01, t23, 0x7531), prmt_u(t45, t67, 0x7531)};
}
__device__ __forceinline__ void decode_block_low(const uint4 duo, int second, unsigned (&a)[8], int palette) {
  const LowTable table = low_table(duo.w >> (16 * second), palette);
  if (second == 0) {
    table.lookup(duo.x & kField0, (duo.x >> 3) & kField0, a[0], a[1]);
    table.lookup((duo.x >> 6) & kField0, (duo.x >> 10) & kField0, a[2], a[3]);
    table.lookup((duo.x >> 13) & kField0, duo.y & kField0, a[4], a[5]);
    table.lookup((duo.y >> 3) & kField0, (duo.y >> 6) & kField0, a[6], a[7]);
  } else {
    table.lookup((duo.y >> 10) & kField0, (duo.y >> 13) & kField0, a[0], a[1]);
    table.lookup(duo.z & kField0, (duo.z >> 3) & kField0, a[2], a[3]);
    table.lookup((duo.z >> 6) & kField0, (duo.z >> 10) & kField0, a[4], a[5]);
    const unsigned spare = ((duo.x >> 9) & 0x00010001u) | ((duo.y >> 8) & 0x00020002u) | ((duo.z >> 7) & 0x00040004u);
    table.lookup((duo.z >> 13) & kField0, spare, a[6], a[7]);
  }
}

// e0 <= e1 for block `second` of a duo (biased bytes compare like the signed endpoints)
__device__ __forceinline__ bool duo_block_is_low(const uint4 duo, int second) {
  const unsigned ends = duo.w >> (16 * second);
  return (ends & 0xffu) <= ((ends >> 8) & 0xffu);
}

// amax of |x| over one token row, as the integer order of bf16 magnitudes
__device__ __forceinline__ unsigned chunk_absmax(uint4 c) {
  unsigned m = 0;
  unsigned w[4] = {c.x, c.y, c.z, c.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    m = max(m, w[i] & 0x7fffu);
    m = max(m, (w[i] >> 16) & 0x7fffu);
  }
  return m;
}

// power-of-two scaling that brings a row with bf16 magnitude pattern `amax_bits` below 2^15
__device__ __forceinline__ void token_scaling(unsigned amax_bits, float &mult, float &inverse) {
  int ex = int(amax_bits >> 7) & 0xff;
  if (amax_bits == 0) ex = 141;
  ex = min(max(ex, 15), 254);
  mult = __int_as_float((268 - ex) << 23);      // 2^(14 - (ex-127))
  inverse = __int_as_float((ex - 14) << 23);    // 2^((ex-127) - 14)
}

__device__ __forceinline__ uint4 convert_chunk(uint4 c, float mult) {
  unsigned w[4] = {c.x, c.y, c.z, c.w};
  unsigned o[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float lo = __uint_as_float(w[i] << 16) * mult;
    float hi = __uint_as_float(w[i] & 0xffff0000u) * mult;
    __half2 h = __floats2half2_rn(lo, hi);
    o[i] = *reinterpret_cast<unsigned *>(&h);
  }
  return make_uint4(o[0], o[1], o[2], o[3]);
}

// ---------------------------------------------------------------------------------------------
// Staged form of one token for the single-token decode kernel (gemv_solo_kernel): a 16-byte slot with
// the fp32 multiplier 2^s * 2^24/889, then per 128-column unit and lane quad t the four fp16 values
// (hi_t, hi_{t+4}, lo_t, lo_{t+4}) of 7 * S_block * 2^-24 (32 bytes per unit), then the activations as
// fp16 with the factor 2^-offset of the index field they meet (256 bytes per unit).  The kernel stages
// a bf16 token itself, or copies this form when the producer of the activations wrote it.
// ---------------------------------------------------------------------------------------------
constexpr int kStagedHeader = 16;
__host__ __device__ inline size_t staged_bytes(int KI) { return kStagedHeader + size_t(KI) * (32 + 256); }
constexpr float kSoloScale = 16777216.0f / 889.0f;   // sums are (n * x) * 2^-24, palette value = n / 889

// exponent of the staging factor 2^-e for pair i of the first / second block of a duo (tx_common.cuh)
__device__ __forceinline__ int solo_pair_exponent(int second, int pair) {
  // first: offsets 0,3,6,10->0,13->3 (word 0), 0,3,6 (word 1); second: 10->0,13->3 (word 1), 0,3,6,0,3 (word 2), spare bit 9
  const unsigned table = second ? 0x93063030u : 0x63030630u;       // nibble i = exponent of pair i
  return int((table >> (4 * pair)) & 15u);
}

// Stages one token for gemv_solo_kernel: xs[column] = fp16(x * mult * 2^-e(column)), and per unit and
// lane quad t the four fp16 values (hi_t, hi_{t+4}, lo_t, lo_{t+4}) of 7 * S_block * 2^-24.
// `i` is the 8-column chunk index; chunks 2b and 2b+1 of block b sit in neighbouring lanes.
__device__ __forceinline__ void solo_stage_chunk(int i, uint4 raw, float mult, uint8_t *xs_g, uint8_t *stab_g, bool inside) {
  const int pair0 = 4 * (i & 1), second = (i >> 3) & 1;            // block b = i >> 1, second half of the unit when b & 4
  unsigned w[4] = {raw.x, raw.y, raw.z, raw.w}, o[4];
  float sum = 0.f;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int e = solo_pair_exponent(second, pair0 + j);
    const float down = __int_as_float((127 - e) << 23), up = __int_as_float((127 + e) << 23);
    const float lo = __uint_as_float(w[j] << 16) * mult * down;
    const float hi = __uint_as_float(w[j] & 0xffff0000u) * mult * down;
    const __half2 h = __floats2half2_rn(lo, hi);
    o[j] = *reinterpret_cast<const unsigned *>(&h);
    const float2 back = __half22float2(h);                          // the value the tensor core will see
    sum += (back.x + back.y) * up;
  }
  sum += __shfl_xor_sync(0xffffffffu, sum, 1);                      // both chunks of the block
  if (inside) {
    reinterpret_cast<uint4 *>(xs_g)[i] = make_uint4(o[0], o[1], o[2], o[3]);
    if ((i & 1) == 0) {
      const int block = i >> 1, unit = block >> 3, t = block & 3, high = (block >> 2) & 1;
      const float v = sum * (7.0f / 16777216.0f);
      const __half hi = __float2half_rn(v);
      const __half lo = __float2half_rn(v - __half2float(hi));
      __half *entry = reinterpret_cast<__half *>(stab_g + size_t(unit) * 32 + t * 8);
      entry[high] = hi;
      entry[2 + high] = lo;
    }
  }
}

// ---------------------------------------------------------------------------------------------
// Staged form of a prompt's activations for the tensor-core tiles: fp16 after an exact power-of-two rescale per token, chunk-major
// [K/8][tokens padded to 32][8] with K padded to 128, the order of K in which the tile's producers hold the weights (element 4t + i of step j of a
// 64-column half unit is column 16t + 4j + i), then one fp32 multiplier 2^s * 65536/889 a token.  stage_activations_kernel writes it
// from rows in memory; a kernel that has a row in registers writes it with stage_piece.
// ---------------------------------------------------------------------------------------------
__host__ __device__ inline int padded_prompt(int tokens) { return (tokens + 31) & ~31; }
__host__ __device__ inline size_t staged_prompt_multipliers(int K, int tokens) { return size_t((K + 127) / 128) * 16 * padded_prompt(tokens) * 16; }   // byte offset
__host__ __device__ inline size_t staged_prompt_bytes(int K, int tokens) { return staged_prompt_multipliers(K, tokens) + size_t(padded_prompt(tokens)) * 4; }
// Eight consecutive columns (converted) of piece i of a token; neighbouring lanes hold neighbouring pieces, lane 0 of eight the first of a half unit.
// Lanes q and q ^ 2 swap halves, so that each stores one whole chunk.  `inside`: the piece exists (all lanes of the warp call).
__device__ __forceinline__ void stage_piece(uint4 *staged, int padded_tokens, int tok, int i, uint4 v, bool inside) {
  const int q = i & 7, odd = (q >> 1) & 1;               // block column parity
  const unsigned give0 = odd ? v.x : v.z, give1 = odd ? v.y : v.w;
  const unsigned get0 = __shfl_xor_sync(0xffffffffu, give0, 2), get1 = __shfl_xor_sync(0xffffffffu, give1, 2);
  // even columns keep steps 2(q & 1), odd ones steps 2(q & 1) + 1; chunk 2j + c of the half unit
  const int chunk = (i & ~7) + 2 * (2 * (q & 1) + odd) + (q >> 2);
  if (inside) staged[size_t(chunk) * padded_tokens + tok] = odd ? make_uint4(get0, get1, v.z, v.w) : make_uint4(v.x, v.y, get0, get1);
}

// One row by the CTAs of a cluster (blockIdx.x the share, blockIdx.y the token): every CTA takes a run of half units, the largest magnitudes meet
// through distributed shared memory.  For few tokens: a CTA a row leaves most SMs idle and a long row is a long chain (16 rows of 17408 columns
// took 9.8 us that way).  From kSplitColumns columns on: a linear of 5120 x 17408 with 16 and 64 tokens
// 21.7 -> 19.6 and 26.4 -> 24.1 us, 8192 x 28672 45.0 -> 38.6 and 49.5 -> 43.5, but 2048 x 11008 with 29 13.4 -> 14.1 and 5120 x 5120 with 16 12.0 -> 13.6 (a cluster's
// launch).  At the line, 2048 x 12288 with 16, 32, 64, 96, 128 and 148 tokens: 13.6 -> 11.6, 13.7 -> 14.2, 13.6 -> 13.5, 21.4 -> 22.5, 23.5 -> 23.5, 28.4 -> 26.3; 5120 x 17408
// with 96, 128 and 148: 43.9 -> 42.4, 44.5 -> 41.9, 46.8 -> 47.4.  piece(i): eight columns as bf16 (or, half_in, fp16), asked for once where a thread has up to kSplitHeld of them.
constexpr int kSplitThreads = 256, kSplitHeld = 4, kSplitColumns = 12288;
template <typename Piece>
__device__ __forceinline__ void stage_split_row(uint4 *staged, float *multipliers, int K, int padded_tokens, bool half_in, Piece piece) {
  __shared__ unsigned warp_peak[kSplitThreads / 32], peak_s;
  const int shares = gridDim.x, share = blockIdx.x, tok = blockIdx.y, pieces = (K + 127) / 128 * 16, exist = K / 8;
  const int first = int((long long)share * (pieces / 8) / shares) * 8, last = int((long long)(share + 1) * (pieces / 8) / shares) * 8;
  const auto fetch = [&](int i) { return i < last && i < exist ? piece(i) : make_uint4(0, 0, 0, 0); };
  uint4 held[kSplitHeld];
  unsigned peak = 0;
#pragma unroll
  for (int c = 0; c < kSplitHeld; ++c) held[c] = fetch(first + int(threadIdx.x) + c * kSplitThreads);
  float mult = 1.f, inverse = 1.f;
  if (!half_in) {
#pragma unroll
    for (int c = 0; c < kSplitHeld; ++c) peak = max(peak, chunk_absmax(held[c]));
    for (int i = first + int(threadIdx.x) + kSplitHeld * kSplitThreads; i < last; i += kSplitThreads) peak = max(peak, chunk_absmax(fetch(i)));
    peak = __reduce_max_sync(0xffffffffu, peak);
    if ((threadIdx.x & 31) == 0) warp_peak[threadIdx.x >> 5] = peak;
    __syncthreads();
#pragma unroll
    for (int w = 0; w < kSplitThreads / 32; ++w) peak = max(peak, warp_peak[w]);
    if (shares > 1) {
      if (threadIdx.x == 0) peak_s = peak;
      __syncwarp();              // (the cluster barriers want whole warps)
      asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
      for (int r = 0; r < shares; ++r) {
        unsigned other;
        asm volatile("{\n\t.reg .b32 remote;\n\tmapa.shared::cluster.u32 remote, %1, %2;\n\tld.shared::cluster.u32 %0, [remote];\n\t}"
                     : "=r"(other) : "r"(unsigned(__cvta_generic_to_shared(&peak_s))), "r"(r) : "memory");
        peak = max(peak, other);
      }
      asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");   // (waited for at the end: nobody leaves while another reads)
    }
    token_scaling(peak, mult, inverse);
  }
  const auto store = [&](int i, uint4 v) { stage_piece(staged, padded_tokens, tok, i, half_in ? v : convert_chunk(v, mult), i < last); };
#pragma unroll
  for (int c = 0; c < kSplitHeld; ++c)
    if (first + c * kSplitThreads < last) store(first + int(threadIdx.x) + c * kSplitThreads, held[c]);
  for (int i0 = first + kSplitHeld * kSplitThreads; i0 < last; i0 += kSplitThreads) store(i0 + int(threadIdx.x), fetch(i0 + int(threadIdx.x)));
  if (share == 0 && threadIdx.x == 0) multipliers[tok] = inverse * kNumeratorScale;
  __syncwarp();
  if (!half_in && shares > 1) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// CTAs of a row: up to eight while two CTAs an SM are not exceeded and each has eight half units or more
inline int staging_shares(int K, int tokens, int sm_count) {
  int shares = 8;
  while (shares > 1 && (tokens * shares > 2 * sm_count || (K + 63) / 64 < 8 * shares)) shares /= 2;
  return shares;
}

}  // namespace tx
