// BC4 encoder on the GPU: the reference's "E3" endpoint search (texelator/encoder.py:34-102 endpoint_opt,
// :23-31 nearest, :105-117 pack_blocks, :137-145 row scales), byte-identical to what that code writes.
//
// The reference evaluates the search with PyTorch fp32 tensor operations on 128-row chunks.  To produce
// the same bytes every arithmetic step here is the same single IEEE operation in the same order -- written
// with the round-to-nearest intrinsics so the compiler cannot contract a multiply and an add -- and the
// five weighted sums per block are added the way PyTorch's CPU reduction adds 16 contiguous floats:
// eight lane sums t[j] + t[j+8], then those left to right.  One thread owns one block of 16 weights:
// start at (round(127 max), round(127 min)), nearest palette entry per weight (first lowest on ties),
// activation-weighted 2x2 least squares on the selector coefficients, then the nine integer neighbours
// of the solution in the reference's order, first best wins.  The palette is a [255, 255, 8] fp32 table
// (lut[e1 + 127][e0 + 127][selector]) in device memory, so any measured or computed palette can be used.
//
// What bounds it: instruction issue.  A group of lanes owns a row, so the row's scale is found and used by the same threads and
// the row is read from HBM once.  Two ways through a block:
//
//   encode_block         any palette, any block.  The nine neighbours only need the distance to the nearest entry, not which
//                        entry it is: packed subtractions (two weights per instruction) and three-input minima, ten instructions per
//                        weight and neighbour.  Selectors are found twice (start and winner).  About 2900 instructions.
//   encode_block_spaced  the software palette: weights are assigned by rounding, the nine errors come from a quadratic form and what is
//                        too close to call is evaluated the first way.  About 1600 instructions, 69 % of the issue slots.
//
// us a call, all blocks the first way / as launched: 4096 x 4096 156.2 / 75.7, 12000 x 4096 453 / 209, 34816 x 5120 1548 / 723, 2048 x 1024 23.2 / 16.6;
// 4096 x 4096 with nine weights of ten zero 164.7 / 166.8, under the texture palette 156.0 / 157.2 (the verdict).
#include "tx_common.cuh"

namespace tx {

// the sum of 16 floats in PyTorch's CPU order for a contiguous inner dimension of 16
__device__ __forceinline__ float sum16(const float (&t)[16]) {
  float s = __fadd_rn(t[0], t[8]);
#pragma unroll
  for (int j = 1; j < 8; ++j) s = __fadd_rn(s, __fadd_rn(t[j], t[j + 8]));
  return s;
}

__device__ __forceinline__ unsigned long long pack2(float lo, float hi) {
  return (unsigned long long)__float_as_uint(lo) | ((unsigned long long)__float_as_uint(hi) << 32);
}
__device__ __forceinline__ float lo2(unsigned long long v) { return __uint_as_float(unsigned(v)); }
__device__ __forceinline__ float hi2(unsigned long long v) { return __uint_as_float(unsigned(v >> 32)); }
__device__ __forceinline__ unsigned long long add2(unsigned long long a, unsigned long long b) {   // two round-to-nearest additions
  unsigned long long d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ float min3_abs(float a, float b, float c) {
  float d;
  asm("min.abs.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
__device__ __forceinline__ float max3_abs(float a, float b, float c) {
  float d;
  asm("max.abs.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
__device__ __forceinline__ float min3(float a, float b, float c) {
  float d;
  asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
  float d;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
  return d;
}
__device__ __forceinline__ float min8_abs(const float (&d)[8]) {
  return fminf(min3_abs(min3_abs(min3_abs(d[0], d[1], d[2]), d[3], d[4]), d[5], d[6]), fabsf(d[7]));
}

__device__ __forceinline__ int clamp127(int e) { return min(max(e, -127), 127); }

// distance of every weight to its nearest palette entry; v2[i] packs weights 2i and 2i+1
__device__ __forceinline__ void nearest_distances(const unsigned long long (&v2)[8], const float4 p_lo, const float4 p_hi, unsigned long long (&best2)[8]) {
  const float p[8] = {p_lo.x, p_lo.y, p_lo.z, p_lo.w, p_hi.x, p_hi.y, p_hi.z, p_hi.w};
  unsigned long long minus[8];
#pragma unroll
  for (int s = 0; s < 8; ++s) minus[s] = pack2(-p[s], -p[s]);
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    float even[8], odd[8];
#pragma unroll
    for (int s = 0; s < 8; ++s) {
      const unsigned long long d = add2(v2[i], minus[s]);
      even[s] = lo2(d);
      odd[s] = hi2(d);
    }
    best2[i] = pack2(min8_abs(even), min8_abs(odd));
  }
}

// nearest palette entry of one weight: the lowest selector at the smallest distance (encoder.py:23-31 keeps the first
// with a strict "<"; a weight that is not a number keeps selector 0)
__device__ __forceinline__ int nearest_selector(float v, const float (&p)[8]) {
  float d[8];
#pragma unroll
  for (int s = 0; s < 8; ++s) d[s] = __fsub_rn(v, p[s]);
  const float m = min8_abs(d);
  int sel = 0;
#pragma unroll
  for (int s = 7; s >= 0; --s) sel = fabsf(d[s]) == m ? s : sel;
  return sel;
}

// half of a palette row (entries 0-3 or 4-7); WIDE: the table lies on a 16-byte boundary, so one load fetches it
template <bool WIDE> __device__ __forceinline__ float4 palette_half(const float *row, int half) {
  if (WIDE) return reinterpret_cast<const float4 *>(row)[half];
  return make_float4(row[4 * half], row[4 * half + 1], row[4 * half + 2], row[4 * half + 3]);
}

// value / scale, rounded to nearest: the residual correction of a quotient that is off by at most one unit in the last
// place is the correctly rounded quotient when the reciprocal is correctly rounded (Markstein 1990, "Computation of
// elementary functions on the IBM RISC System/6000 processor"); the product with the reciprocal can be off by two, so
// it takes a first correction too.  The last residual has to be exact: it is a multiple of 2^-46 times the quotient's
// and the scale's power of two, which is representable while the two exponents add up to -103 or more.  The caller keeps
// the scale at 2^-40 or more, and divides where a weight other than zero is below 2^-60 of the scale.
__device__ __forceinline__ float divide_by_scale(float value, float scale, float reciprocal) {
  float q = __fmul_rn(value, reciprocal);
  q = __fmaf_rn(__fmaf_rn(-q, scale, value), reciprocal, q);
  return __fmaf_rn(__fmaf_rn(-q, scale, value), reciprocal, q);
}

// One block of sixteen scaled weights and what was found for it.
struct Block {
  unsigned long long v2[8], h2[8];   // weights and their activation moments, two to a word
  int e0, e1;                        // the start: the block's extremes
  __device__ __forceinline__ float v(int j) const { return j & 1 ? hi2(v2[j / 2]) : lo2(v2[j / 2]); }
  __device__ __forceinline__ float h(int j) const { return j & 1 ? hi2(h2[j / 2]) : lo2(h2[j / 2]); }
  __device__ __forceinline__ void find_extremes() {
    float vmax = -INFINITY, vmin = INFINITY;
#pragma unroll
    for (int j = 0; j < 16; j += 2) {
      vmax = max3(vmax, v(j), v(j + 1));
      vmin = min3(vmin, v(j), v(j + 1));
    }
    e0 = clamp127(int(rintf(__fmul_rn(vmax, 127.f))));
    e1 = clamp127(int(rintf(__fmul_rn(vmin, 127.f))));
  }
};
struct Encoded {
  int e0, e1;
  unsigned long long bits;           // sixteen selectors
};
__device__ __forceinline__ const float *palette_row(const float *lut, int q0, int q1) { return lut + (size_t(q1 + 127) * 255 + (q0 + 127)) * 8; }

// The weighted squared error with a palette, in the reference's order of operations.
// (scalar products and sums: with packed multiplies and adds, .rn on both, 4 blocks of 5.6 million came out one
// neighbour off the reference's, as a fused multiply-add would have it)
__device__ __forceinline__ float exact_error(const Block &b, const float4 p_lo, const float4 p_hi) {
  unsigned long long d2[8];
  nearest_distances(b.v2, p_lo, p_hi, d2);
  float te[16];
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    const float d = j & 1 ? hi2(d2[j / 2]) : lo2(d2[j / 2]);
    te[j] = __fmul_rn(b.h(j), __fmul_rn(d, d));
  }
  return sum16(te);
}

template <bool WIDE> __device__ __forceinline__ unsigned long long exact_selectors(const Block &b, const float *row) {
  const float4 q_lo = palette_half<WIDE>(row, 0), q_hi = palette_half<WIDE>(row, 1);
  const float p[8] = {q_lo.x, q_lo.y, q_lo.z, q_lo.w, q_hi.x, q_hi.y, q_hi.z, q_hi.w};
  unsigned long long bits = 0;
#pragma unroll
  for (int j = 0; j < 16; ++j) bits |= (unsigned long long)nearest_selector(b.v(j), p) << (3 * j);
  return bits;
}

// solution of the weighted 2x2 normal equations (encoder.py:78-86), rounded to endpoints
__device__ __forceinline__ void solve_endpoints(float saa, float sbb, float sab, float say, float sby, int e0, int e1, int &c0, int &c1) {
  const float det = __fsub_rn(__fmul_rn(saa, sbb), __fmul_rn(sab, sab));
  const bool keep = fabsf(det) < 1e-12f;
  const float safe = fmaxf(det, 1e-12f);
  float u = fminf(fmaxf(__fdiv_rn(__fsub_rn(__fmul_rn(say, sbb), __fmul_rn(sby, sab)), safe), -1.f), 1.f);
  float z = fminf(fmaxf(__fdiv_rn(__fsub_rn(__fmul_rn(sby, saa), __fmul_rn(say, sab)), safe), -1.f), 1.f);
  if (keep) {
    u = __fdiv_rn(float(e0), 127.f);
    z = __fdiv_rn(float(e1), 127.f);
  }
  c0 = int(rintf(__fmul_rn(u, 127.f)));
  c1 = int(rintf(__fmul_rn(z, 127.f)));
}

// selector coefficients: value = a*u + b*z + c (encoder.py:53-70); the fractions are Python doubles rounded to fp32
struct Coefficients {
  float a[2][8], b[2][8], c[2][8];   // [high mode][selector]
  float2 by_index[8];                // a and b of the high mode by interpolation index (0: e0 .. 7: e1)
};
__constant__ const Coefficients kCoefficients = {
    {{1.f, 0.f, float(4. / 5), float(3. / 5), float(2. / 5), float(1. / 5), 0.f, 0.f},
     {1.f, 0.f, float(6. / 7), float(5. / 7), float(4. / 7), float(3. / 7), float(2. / 7), float(1. / 7)}},
    {{0.f, 1.f, float(1. / 5), float(2. / 5), float(3. / 5), float(4. / 5), 0.f, 0.f},
     {0.f, 1.f, float(1. / 7), float(2. / 7), float(3. / 7), float(4. / 7), float(5. / 7), float(6. / 7)}},
    {{0.f, 0.f, 0.f, 0.f, 0.f, 0.f, -1.f, 1.f}, {}},   // selectors 6 and 7 of the low mode
    {{1.f, 0.f}, {float(6. / 7), float(1. / 7)}, {float(5. / 7), float(2. / 7)}, {float(4. / 7), float(3. / 7)},
     {float(3. / 7), float(4. / 7)}, {float(2. / 7), float(5. / 7)}, {float(1. / 7), float(6. / 7)}, {0.f, 1.f}}};

// Any palette, any block.
template <bool WIDE> __device__ __forceinline__ Encoded encode_block(Block b, const float *lut, const Coefficients &coef) {
  // the reference clamps the quotients, which moves those alone that are not numbers (to -1)
#pragma unroll
  for (int i = 0; i < 8; ++i) b.v2[i] = pack2(fminf(fmaxf(lo2(b.v2[i]), -1.f), 1.f), fminf(fmaxf(hi2(b.v2[i]), -1.f), 1.f));
  b.find_extremes();
  unsigned long long start_bits = 0;
  int c0, c1;
  {
    // weighted 2x2 normal equations on the start's selectors (encoder.py:72-84)
    const float4 p_lo = palette_half<WIDE>(palette_row(lut, b.e0, b.e1), 0), p_hi = palette_half<WIDE>(palette_row(lut, b.e0, b.e1), 1);
    const float p[8] = {p_lo.x, p_lo.y, p_lo.z, p_lo.w, p_hi.x, p_hi.y, p_hi.z, p_hi.w};
    const int high = b.e0 > b.e1;
    float taa[16], tbb[16], tab[16], tay[16], tby[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const int sel = nearest_selector(b.v(j), p);
      start_bits |= (unsigned long long)sel << (3 * j);
      const float a = coef.a[high][sel], bb = coef.b[high][sel];
      const float target = high ? __fsub_rn(b.v(j), 0.f) : __fsub_rn(b.v(j), coef.c[0][sel]);
      const float ha = __fmul_rn(b.h(j), a), hb = __fmul_rn(b.h(j), bb);
      taa[j] = __fmul_rn(ha, a);
      tbb[j] = __fmul_rn(hb, bb);
      tab[j] = __fmul_rn(ha, bb);
      tay[j] = __fmul_rn(ha, target);
      tby[j] = __fmul_rn(hb, target);
    }
    solve_endpoints(sum16(taa), sum16(tbb), sum16(tab), sum16(tay), sum16(tby), b.e0, b.e1, c0, c1);
  }

  // the nine integer neighbours, delta0 outer, delta1 inner; strict "<" keeps the first best (encoder.py:88-101).
  // The next neighbour's palette is requested before this one's errors are computed.
  float best = INFINITY;
  int out = -1;
  const float *first = palette_row(lut, clamp127(c0 - 1), clamp127(c1 - 1));
  float4 p_lo = palette_half<WIDE>(first, 0), p_hi = palette_half<WIDE>(first, 1);
#pragma unroll 1
  for (int n = 0; n < 9; ++n) {
    const int next = min(n + 1, 8);
    const float *ahead = palette_row(lut, clamp127(c0 + next / 3 - 1), clamp127(c1 + next % 3 - 1));
    const float4 next_lo = palette_half<WIDE>(ahead, 0), next_hi = palette_half<WIDE>(ahead, 1);
    const float err = exact_error(b, p_lo, p_hi);
    if (err < best) {
      best = err;
      out = n;
    }
    p_lo = next_lo;
    p_hi = next_hi;
  }
  Encoded e{b.e0, b.e1, start_bits};
  if (out >= 0) {                                   // (no neighbour wins only when the errors are not numbers)
    e.e0 = clamp127(c0 + out / 3 - 1);
    e.e1 = clamp127(c1 + out % 3 - 1);
    e.bits = exact_selectors<WIDE>(b, palette_row(lut, e.e0, e.e1));
  }
  return e;
}

// ---------------------------------------------------------------------------------------------------------------------
// The same search where the table is the software palette (to within kEntryError: a table made by multiplying with 1/889 is not
// the correctly rounded one) and the endpoints are apart.
//
// The palette's eight entries are then evenly spaced numbers n_g / 889, n_g = (7 - g) e0 + g e1, so the nearest entry of a weight is
// a rounding, and moving both endpoints by at most one moves an entry by at most 7/889, which changes the nearest entry of
// the weights next to a midpoint alone.  So the sixteen weights are assigned once, to the palette of the solution (c0, c1), and
// with r = 889 v - n_g and D = c0 - c1 the error of the neighbour (c0 + s, c1 + t), in units of 1/889 squared, is
//
//     sum h (r - (7 - g) s - g t)^2  -  2 (D + s - t) sum h max(0, x),     x = |r| - D/2 - sign(r) ((7 - g) s + g t) - (s - t)/2
//
// the second sum over the weights whose next entry on the side of r comes closer than their own (D of 20 or more: none has the choice of
// a third).  The first is a quadratic form of five sums; the second is over weights within 7 of a midpoint, 14/D of all.
//
// What decides is the order of nine errors that the reference evaluates in fp32.  `slack` bounds the distance of both evaluations from
// the exact value (below); the neighbours within it of the smallest are evaluated the reference's way, one block in a few hundred.  A
// weight whose place is too near a tie is left to the comparison of distances in the same manner.  Everything
// that enters the normal equations is the reference's arithmetic.
// ---------------------------------------------------------------------------------------------------------------------
constexpr int kApart = 20;
constexpr float kToInteger = 12582912.f;   // 1.5 * 2^23: the sum's lowest bits are the rounded number
constexpr unsigned kNoIndices = 0u - 0x4B400000u * 0x249249u;   // less its own bits (0x4B400000) of eight such sums, three bits apart
constexpr float kEntryError = 0x1p-23f;    // of a table's entry
// A weight's place among the entries, in spacings: 7 * saturate((7 e0 - 889 v) / (7 D)) is off by at most 2^-19.5 (one fused rounding, the
// reciprocal's, two products' of numbers up to 7).  The reference compares distances that are off by kEntryError and by 2^-27 for the
// differences themselves, 1.13e-4 / D spacings in all.  Nearer to a tie than both, the distances are compared.
__device__ __forceinline__ float clear_of_tie(float inverse) { return 0.5f - fmaf(1.2e-4f * 7.f, inverse, 0x1p-19f); }   // inverse: 1 / (7 D)

struct Place {
  float g, y;          // the nearest entry's index, and the place between entry 0 and entry 7 as 0..1 (beyond the ends: 0 or 1)
  unsigned word;       // index in the three lowest bits, the same bits above for all weights
  float off;           // distance from the nearest entry in spacings, 0 beyond the ends
};
__device__ __forceinline__ Place place_of(float v, float seven_e0, float inverse) {   // inverse: 1 / (7 D)
  Place p;
  p.y = __saturatef(__fmul_rn(__fmaf_rn(v, -889.f, seven_e0), inverse));
  const float m = __fmaf_rn(p.y, 7.f, kToInteger);
  p.word = __float_as_uint(m);
  p.g = __fsub_rn(m, kToInteger);
  p.off = fabsf(__fmaf_rn(p.y, 7.f, -p.g));
  return p;
}

// Indices of the weights near a tie again, by the distances from the two entries on either side (equal: the lower selector, which is
// the lower index but for entry 7, selector 1).
__device__ __forceinline__ void settle_ties(const Block &b, const float *row, float seven_e0, float inverse, unsigned (&indices)[2]) {
  const float clear = clear_of_tie(inverse);
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    const float v = b.v(j);
    const Place p = place_of(v, seven_e0, inverse);
    if (p.off < clear) continue;
    const int lower = min(int(7.f * p.y), 6), upper = lower + 1;   // (a place near a tie is not near an entry)
    const float to_lower = fabsf(__fsub_rn(v, row[lower == 0 ? 0 : lower + 1])), to_upper = fabsf(__fsub_rn(v, row[upper == 7 ? 1 : upper + 1]));
    const unsigned g = unsigned(to_upper < to_lower || (to_upper == to_lower && lower > 0 && upper == 7) ? upper : lower), at = 3 * (j & 7);
    indices[j >> 3] = (indices[j >> 3] & ~(7u << at)) | (g << at);
  }
}

// selectors from sixteen interpolation indices of three bits: 0 -> 0, 7 -> 1, g -> g + 1
__device__ __forceinline__ unsigned long long selectors_of(unsigned long long g) {
  constexpr unsigned long long lowest = 0x249249249249ull;
  const unsigned long long b0 = g & lowest, b1 = (g >> 1) & lowest, b2 = (g >> 2) & lowest;
  const unsigned long long s0 = (b1 ^ b2) | (b0 ^ b2);          // not all three bits alike ...
  const unsigned long long first = ~b0 & lowest;                // ... else the lowest bit of g + 1 is flipped
  return (s0 & first) | (~s0 & lowest & b0) | ((b0 ^ b1) << 1) | ((b2 ^ (b0 & b1)) << 2);
}

constexpr int kEncodeThreads = 128;

// `lanes`: those of the warp that have a block in this step, all of which call.
// false: the block is one for encode_block (weights that are not numbers among them: their solution has no two endpoints apart)
template <bool WIDE>
__device__ __forceinline__ bool encode_block_spaced(const Block &b, const float *lut, const Coefficients &coef, float4 (*list)[kEncodeThreads], unsigned lanes, Encoded &e) {
  // (a lane that goes to encode_block takes its warp's time anyway, so the whole warp goes)
  if (__any_sync(lanes, b.e0 - b.e1 < kApart)) return false;
  int c0, c1;
  {
    const float seven_e0 = 7.f * float(b.e0), inverse = __frcp_rn(7.f * float(b.e0 - b.e1));
    float worst = 0.f;
    unsigned indices[2] = {kNoIndices, kNoIndices};     // of weights 0-7 and 8-15, three bits each
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const Place p = place_of(b.v(j), seven_e0, inverse);
      worst = fmaxf(worst, p.off);
      indices[j >> 3] += p.word << (3 * (j & 7));
    }
    if (!(worst < clear_of_tie(inverse))) settle_ties(b, palette_row(lut, b.e0, b.e1), seven_e0, inverse, indices);
    float saa = 0.f, sbb = 0.f, sab = 0.f, say = 0.f, sby = 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) {                       // sum16: weights j and j + 8 first, then those sums in order
      float taa[2], tbb[2], tab[2], tay[2], tby[2];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const float v = b.v(j + 8 * i), h = b.h(j + 8 * i);
        const float2 ab = coef.by_index[indices[i] >> (3 * j) & 7];
        const float ha = __fmul_rn(h, ab.x), hb = __fmul_rn(h, ab.y);
        taa[i] = __fmul_rn(ha, ab.x);
        tbb[i] = __fmul_rn(hb, ab.y);
        tab[i] = __fmul_rn(ha, ab.y);
        tay[i] = __fmul_rn(ha, v);
        tby[i] = __fmul_rn(hb, v);
      }
      const auto add = [&](float &s, const float (&t)[2]) { s = j == 0 ? __fadd_rn(t[0], t[1]) : __fadd_rn(s, __fadd_rn(t[0], t[1])); };
      add(saa, taa);
      add(sbb, tbb);
      add(sab, tab);
      add(say, tay);
      add(sby, tby);
    }
    solve_endpoints(saa, sbb, sab, say, sby, b.e0, b.e1, c0, c1);
  }
  const int apart = c0 - c1;
  if (__any_sync(lanes, apart < kApart)) return false;

  // -- assignment to the solution's palette
  const float D = float(apart), seven_c0 = 7.f * float(c0), inverse = __frcp_rn(7.f * D), near_tie = 0.5f * D - 7.01f;
  float H[2] = {}, Hg[2] = {}, Hgg[2] = {}, R[2] = {}, Rg[2] = {}, S[2] = {};
  unsigned signs = 0;
  int listed = 0;
#pragma unroll
  for (int j = 0; j < 16; ++j) {
    const float v = b.v(j), h = b.h(j);
    const Place p = place_of(v, seven_c0, inverse);
    const float r = __fmaf_rn(v, 889.f, -__fmaf_rn(p.g, -D, seven_c0)), hr = h * r, hg = h * p.g;
    signs |= __float_as_uint(h);
    H[j & 1] += h;
    Hg[j & 1] += hg;
    Hgg[j & 1] = fmaf(hg, p.g, Hgg[j & 1]);
    R[j & 1] += hr;
    Rg[j & 1] = fmaf(hr, p.g, Rg[j & 1]);
    S[j & 1] = fmaf(hr, r, S[j & 1]);
    if (fabsf(r) > near_tie) list[listed++][threadIdx.x] = make_float4(r, p.g, h, p.y);
  }
  // errors of the nine neighbours, less the solution's own
  float gain[9] = {}, listed_h = 0.f;
#pragma unroll 1
  for (int i = 0; i < listed; ++i) {
    const float4 w = list[i][threadIdx.x];
    const float side = w.x > 0.f ? 1.f : -1.f;
    const float by0 = fmaf(-side, 7.f - w.y, -0.5f), by1 = fmaf(-side, w.y, 0.5f);
    const bool inside = w.w > 0.f && w.w < 1.f;                // beyond the ends there is no next entry
    const float x = inside ? fabsf(w.x) - 0.5f * D : -1e30f;
    listed_h += w.z;
#pragma unroll
    for (int n = 0; n < 9; ++n) gain[n] = fmaf(w.z, fmaxf((x + float(n / 3 - 1) * by0) + float(n % 3 - 1) * by1, 0.f), gain[n]);
  }
  const float sum_h = H[0] + H[1], sum_hg = Hg[0] + Hg[1], sum_hgg = Hgg[0] + Hgg[1], sum_s = S[0] + S[1];
  const float along1 = Rg[0] + Rg[1], along0 = fmaf(7.f, R[0] + R[1], -along1);
  const float h01 = fmaf(7.f, sum_hg, -sum_hgg), h00 = fmaf(49.f, sum_h, fmaf(-14.f, sum_hg, sum_hgg));
  float error[9], smallest = INFINITY, most = 0.f;
#pragma unroll
  for (int n = 0; n < 9; ++n) {
    const float s = float(n / 3 - 1), t = float(n % 3 - 1);
    const float form = s * s * h00 + 2.f * s * t * h01 + t * t * sum_hgg - 2.f * s * along0 - 2.f * t * along1;
    error[n] = fmaf(-2.f * (D + s - t), gain[n], form);
    // an endpoint beyond its limit is the limit: another neighbour's palette again
    if ((n / 3 == 2 && c0 == 127) || (n % 3 == 0 && c1 == -127)) error[n] = INFINITY;
    smallest = fminf(smallest, error[n]);
    most = fmaxf(most, gain[n]);
  }
  // Distance of either evaluation from the exact value, with H, S, G the sums of h, h r^2, h |r| <= (H D + S / D) / 2 (all h >= 0), u = 2^-24:
  //   reference  a difference from an entry is off by 889 * 2 u for the entry and u |r| for its own rounding, at residuals of up to |r| + 7;
  //              products and sums (two and eight deep) add 12 u of the error:  3556 u (G + 7 H) + 13 u (2 S + 98 H)
  //   here       the five sums are ten deep and r is rounded once: 2 (154 + 70 + 14) u G and (1960 + 1960 + 490) u H, their combination
  //              140 u G + 980 u H;  a listed weight's x is off by 2 u D, the sums of gains are eighteen deep:
  //              2 (D + 2) (2 u D H_listed + 18 u gain)
  // `slack` is their sum, rounded up.  All of it is relative: sums of moments that are not zero but below 2^-100 are left to the other way, as the
  // reference's products, 889^2 times smaller than the ones here, would lose to underflow (2^-149 each, 2^-125 of sixteen in these units) what `slack`
  // (2^-9 of the sum of moments or more) does not hold.
  constexpr float u = 0x1p-24f;
  const float spread = fmaf(sum_h, D, sum_s * (7.f * inverse));   // 2 G at most
  const float slack = u * (2100.f * spread + 32000.f * sum_h + 28.f * sum_s + (D + 2.f) * fmaf(5.f * D, listed_h, 40.f * most));
  const float limit = smallest + 2.f * slack;
  if (int(signs) < 0 || !(limit < INFINITY) || (sum_h > 0.f && sum_h < 0x1p-100f)) return false;    // (a moment below zero, or sums that are not numbers)
  unsigned contenders = 0;
#pragma unroll
  for (int n = 0; n < 9; ++n) contenders |= error[n] <= limit ? 1u << n : 0u;
  int out = __ffs(contenders) - 1;
  if (contenders & (contenders - 1)) {
    float best = INFINITY;
    out = -1;
#pragma unroll 1
    for (unsigned left = contenders; left; left &= left - 1) {
      const int n = __ffs(left) - 1;
      const float *row = palette_row(lut, c0 + n / 3 - 1, c1 + n % 3 - 1);
      const float err = exact_error(b, palette_half<WIDE>(row, 0), palette_half<WIDE>(row, 1));
      if (err < best) {
        best = err;
        out = n;
      }
    }
    if (out < 0) return false;
  }
  e.e0 = c0 + out / 3 - 1;
  e.e1 = c1 + out % 3 - 1;
  {
    const float seven_e0 = 7.f * float(e.e0), inverse_e = __frcp_rn(7.f * float(e.e0 - e.e1));
    float worst = 0.f;
    unsigned indices[2] = {kNoIndices, kNoIndices};
#pragma unroll
    for (int j = 0; j < 16; ++j) {
      const Place p = place_of(b.v(j), seven_e0, inverse_e);
      worst = fmaxf(worst, p.off);
      indices[j >> 3] += p.word << (3 * (j & 7));
    }
    if (!(worst < clear_of_tie(inverse_e))) settle_ties(b, palette_row(lut, e.e0, e.e1), seven_e0, inverse_e, indices);
    e.bits = selectors_of((unsigned long long)indices[0] | ((unsigned long long)indices[1] << 24));
  }
  return true;
}

// Whether a table is the software palette where the endpoints are apart (the others are only ever read).  Each of CTAS CTAs looks at its share, a
// row of the table a thread and step, and leaves a byte, 1 or 0, in the
// first CTAS bytes that every CTA of the encode kernel behind it is going to write, which reads them before it writes there: the verdict
// belongs to the call, without a word of its own that calls on two streams would share.
//
// The encode kernel starts beside it and finds its first rows' largest magnitudes before it waits.  A call that cannot use the answer pays 1.0 us for the launch
// and about two for what the wait is longer than that search: under the texture palette 2048 x 1024 takes 23.1 us without a verdict and
// 26.1 with, 2048 x 2048 43.4 and 46.4, 4096 x 4096 155.9 and 156.5 (28.5, 49.4 and 160.8 with a verdict of 128 CTAs in front of the whole encode kernel).
// 32 CTAs, 16 where a CTA's first step writes fewer bytes: 16, 32 and 64 take 26.3, 26.1 and 26.1 there.
constexpr int kPaletteRows = 255 * 255, kVerdicts = 32, kFewVerdicts = 16, kVerdictThreads = 1024;
template <int CTAS, bool WIDE>
__global__ void __launch_bounds__(kVerdictThreads) palette_verdict_kernel(const float *__restrict__ lut, uint8_t *__restrict__ blocks, int ctas, size_t cta_bytes,
                                                                          int shares, int share_bytes) {
  grid_launch_dependents();      // the encode kernel finds its first rows' largest magnitudes meanwhile
  constexpr int kEach = (kPaletteRows + CTAS * kVerdictThreads - 1) / (CTAS * kVerdictThreads);
  float4 entries[kEach][2];
  int left[kEach], right[kEach];
#pragma unroll
  for (int i = 0; i < kEach; ++i) {                     // all loads in flight together
    const int row = (i * CTAS + int(blockIdx.x)) * kVerdictThreads + int(threadIdx.x);
    right[i] = row / 255 - 127;
    left[i] = row < kPaletteRows ? row % 255 - 127 : -128;
    if (left[i] - right[i] >= kApart - 2) {
      entries[i][0] = palette_half<WIDE>(lut + size_t(row) * 8, 0);
      entries[i][1] = palette_half<WIDE>(lut + size_t(row) * 8, 1);
    }
  }
  bool same = true;
#pragma unroll
  for (int i = 0; i < kEach; ++i) {
    if (left[i] - right[i] < kApart - 2) continue;
    const float4 lo = entries[i][0], hi = entries[i][1];
    const float entry[8] = {lo.x, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w, lo.y};   // by interpolation index
    const float step = float(right[i] - left[i]);
    float expected = float(7 * left[i]);                  // 889 times the entry, a whole number
#pragma unroll
    for (int g = 0; g < 8; ++g) {
      same &= fabsf(__fmaf_rn(entry[g], 889.f, -expected)) <= 889.f * kEntryError;
      expected += step;
    }
  }
  same = __syncthreads_and(same);
  for (int i = threadIdx.x; i < ctas * shares; i += kVerdictThreads)
    blocks[size_t(i / shares) * cta_bytes + size_t(i % shares) * share_bytes + blockIdx.x] = same ? 1 : 0;
}

// From here on the verdict pays: 2048 x 1024 takes 23.2 us without it and 16.6 with; 300 x 4096, half the size, 20.6 and 20.7.
constexpr size_t kSpacedWeights = size_t(1) << 21;
constexpr int kEncodeWave = 148 * 4;   // blocks of threads resident at once (registers)

// A group of GROUP lanes encodes one row after another (rows group, group + groups, ...): the row's largest magnitude
// first, then one 16-weight block per lane and step.  With gridDim.y > 1 that many groups share a row: each finds the
// largest magnitude for itself (the row comes from L2) and takes every gridDim.y-th step.
// SPACED: palette_verdict_kernel ran in front and left `verdicts` bytes (every CTA has as many to write, or more).
template <int GROUP, bool WIDE, bool SPACED>
__global__ void __launch_bounds__(kEncodeThreads, 4) encode_kernel(const float *__restrict__ weight, const float *__restrict__ hdiag,
                                                                const float *__restrict__ lut, unsigned long long *blocks,
                                                                float *__restrict__ scales, int M, int K, int verdicts) {
  __shared__ Coefficients coef;
  __shared__ float peak[kEncodeThreads / 32];
  __shared__ float4 list[SPACED ? 16 : 1][kEncodeThreads];
  // (in shared memory: lanes read different entries)
  if (threadIdx.x < sizeof(Coefficients) / 4) reinterpret_cast<float *>(&coef)[threadIdx.x] = reinterpret_cast<const float *>(&kCoefficients)[threadIdx.x];
  __syncthreads();
  const int bpr = K / 16;
  const int in_group = threadIdx.x % GROUP, group = threadIdx.x / GROUP;
  constexpr int kGroups = kEncodeThreads / GROUP;
  bool spaced = false;
  for (int row0 = blockIdx.x * kGroups; row0 < M; row0 += gridDim.x * kGroups) {
    const int row = row0 + group;
    const bool live = row < M;
    const float4 *w4 = reinterpret_cast<const float4 *>(weight + size_t(live ? row : 0) * K);
    // scale_m = max(|W[m, :]|, 1e-12)
    float m = 0.f;
    if (live) {
#pragma unroll 8
      for (int i = in_group; i < bpr * 4; i += GROUP) {
        const float4 w = w4[i];
        m = max3_abs(max3_abs(m, w.x, w.y), w.z, w.w);
      }
    }
    for (int d = 16; d; d >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, d));
    if (GROUP > 32) {
      if ((threadIdx.x & 31) == 0) peak[threadIdx.x >> 5] = m;
      __syncthreads();
#pragma unroll
      for (int i = 0; i < GROUP / 32; ++i) m = fmaxf(m, peak[group * (GROUP / 32) + i]);
      __syncthreads();
    }
    if (SPACED && row0 == int(blockIdx.x) * kGroups) {
      const unsigned long long *verdict = blocks + size_t(row0) * bpr + blockIdx.y * GROUP;
      grid_dependency_wait();
      // (one barrier for all: read before one writes blocks there)
      spaced = __syncthreads_and(int(threadIdx.x) >= verdicts / 8 || __ldcg(verdict + threadIdx.x) == 0x0101010101010101ull);
    }
    const float scale = fmaxf(m, 1e-12f), reciprocal = __frcp_rn(scale);
    const bool normal = scale >= 0x1p-40f && scale <= 0x1p60f;
    if (!live) continue;
    if (in_group == 0 && blockIdx.y == 0) scales[row] = scale;

    for (int kb = blockIdx.y * GROUP + in_group; kb < bpr; kb += gridDim.y * GROUP) {
      Block b;
      float4 w[4];
      bool rough = !normal;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        w[j] = w4[kb * 4 + j];
        const float4 g = reinterpret_cast<const float4 *>(hdiag)[kb * 4 + j];
        b.h2[2 * j] = pack2(g.x, g.y);
        b.h2[2 * j + 1] = pack2(g.z, g.w);
        // (no weight of the row is above the scale, so the quotients need no clamp)
        const auto quotient = [&](float value) {
          rough |= !(fabsf(value) >= scale * 0x1p-60f || value == 0.f);   // (true for a weight that is not a number)
          return divide_by_scale(value, scale, reciprocal);
        };
        const float a0 = quotient(w[j].x), a1 = quotient(w[j].y), a2 = quotient(w[j].z), a3 = quotient(w[j].w);
        b.v2[2 * j] = pack2(a0, a1);
        b.v2[2 * j + 1] = pack2(a2, a3);
      }
      if (rough) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const auto quotient = [&](float value) { return __fdiv_rn(value, scale); };
          b.v2[2 * j] = pack2(quotient(w[j].x), quotient(w[j].y));
          b.v2[2 * j + 1] = pack2(quotient(w[j].z), quotient(w[j].w));
        }
      }
      b.find_extremes();
      Encoded e;
      const int rest = bpr - (kb - int(threadIdx.x & 31));   // blocks from the warp's first lane on (a warp has one row)
      const unsigned lanes = rest >= 32 ? 0xffffffffu : (1u << rest) - 1;
      if (!SPACED || !spaced || !encode_block_spaced<WIDE>(b, lut, coef, list, lanes, e)) e = encode_block<WIDE>(b, lut, coef);
      blocks[size_t(row) * bpr + kb] = (unsigned long long)(unsigned(e.e0) & 0xffu) | ((unsigned long long)(unsigned(e.e1) & 0xffu) << 8) | (e.bits << 16);
    }
  }
}

template <int GROUP>
static cudaError_t launch_encode_rows(const float *weight, const float *hdiag, const float *lut, int M, int K, uint8_t *blocks, float *scales, cudaStream_t stream) {
  const int per_cta = kEncodeThreads / GROUP, ctas = (M + per_cta - 1) / per_cta;
  // Rows alone fill the chip from about 600 blocks of threads on (four to an SM).  Beyond three times that the blocks take several each, beyond sixteen times
  // six times as many blocks share the rows.  One wave of blocks, three, six and a block a row, us -- 4096 x 4096 (6.9 waves) 75.8, 76.5, 78.3, 80.2, under the
  // texture palette 164, 157, 158, 159; 20000 x 4000 (33) 384, 387, 384, 425 and 830, 789, 763, 773; 34816 x 5120 (29) 738, 731, 727, 740 and
  // 1698, 1597, 1558, 1557.  Below one wave a row is shared, by as many groups as fit one wave and have a step each: 8 x 17408 84.6 -> 11.4 us, 100 x 11200 57.9 -> 16.6,
  // 300 x 11200 74.9 -> 44.3 (the kernel that spread single blocks over the chip took 29.2, 61.6 and 153.7).
  const int grid = std::min(ctas, (ctas > 16 * kEncodeWave ? 6 : 3) * kEncodeWave);
  const int steps = (K / 16 + GROUP - 1) / GROUP, most = std::max(1, std::min(kEncodeWave / grid, steps));
  const int rounds = (steps + most - 1) / most;   // steps of a group
  const int shares = (steps + rounds - 1) / rounds;
  // a palette may start at any float (a slice of a larger buffer): the wide loads are for tables on a 16-byte boundary
  const bool wide = !(reinterpret_cast<uintptr_t>(lut) & 15);
  const int fewest = std::min(K / 16 - (shares - 1) * GROUP, GROUP) * 8;   // bytes the first step of a CTA writes, at least
  const bool spaced = size_t(M) * K >= kSpacedWeights && fewest >= kFewVerdicts;
  const int verdicts = fewest >= kVerdicts ? kVerdicts : kFewVerdicts;
  if (spaced) {
    const size_t cta_bytes = size_t(per_cta) * K / 2;
    const auto verdict = verdicts == kVerdicts ? (wide ? palette_verdict_kernel<kVerdicts, true> : palette_verdict_kernel<kVerdicts, false>)
                                               : (wide ? palette_verdict_kernel<kFewVerdicts, true> : palette_verdict_kernel<kFewVerdicts, false>);
    verdict<<<verdicts, kVerdictThreads, 0, stream>>>(lut, blocks, grid, cta_bytes, shares, GROUP * 8);
    count_launch();
  }
  // four blocks of threads to an SM want 132 KB of its shared memory
  const auto kernel = spaced ? (wide ? encode_kernel<GROUP, true, true> : encode_kernel<GROUP, false, true>)
                             : (wide ? encode_kernel<GROUP, true, false> : encode_kernel<GROUP, false, false>);
  // early only behind the verdict, which is a plain launch: what the caller left on the stream has ended before either starts
  return launch_cluster(kernel, spaced, 1, dim3(grid, shares), dim3(kEncodeThreads), 0, stream, weight, hdiag, lut, reinterpret_cast<unsigned long long *>(blocks),
                        scales, M, K, verdicts);
}

int launch_encode(const float *weight, const float *hdiag, const float *lut, int M, int K, uint8_t *blocks, float *scales, cudaStream_t stream) {
  // lanes per row: the size that leaves the fewest lanes without a block in the last step of a row, the larger one when
  // equal (a row of 198 blocks is 2 steps of 128 lanes with 58 idle, 4 of 64 with 58 idle, 7 of 32 with 26 idle)
  const auto idle = [&](int group) { return (K / 16 + group - 1) / group * group - K / 16; };
  const auto rows = idle(128) <= idle(64) && idle(128) <= idle(32) ? launch_encode_rows<128> : idle(64) <= idle(32) ? launch_encode_rows<64> : launch_encode_rows<32>;
  TX_CUDA(rows(weight, hdiag, lut, M, K, blocks, scales, stream));
  count_launch();
  TX_CUDA(cudaGetLastError());
  return TX_OK;
}

}  // namespace tx

using namespace tx;

extern "C" int tx_encode(const float *weight, const float *hdiag, const float *lut, int M, int K, uint8_t *blocks_out, float *scales_out,
                         void *stream) {
  if (!weight || !hdiag || !lut || !blocks_out || !scales_out) return fail(TX_EINVAL, "tx_encode: null argument");
  if (M < 1 || K < 16 || K % 16) return fail(TX_EINVAL, "tx_encode: K must be a positive multiple of 16 (one BC4 block)");
  if ((reinterpret_cast<uintptr_t>(weight) | reinterpret_cast<uintptr_t>(hdiag) | reinterpret_cast<uintptr_t>(blocks_out)) & 15)
    return fail(TX_EINVAL, "tx_encode: weight, hdiag and blocks must be 16-byte aligned");
  return launch_encode(weight, hdiag, lut, M, K, blocks_out, scales_out, static_cast<cudaStream_t>(stream));
}
