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
// What bounds it: arithmetic -- ten palettes per block, eight entries each, sixteen weights.  The nine neighbours only
// need the distance to the nearest entry, not which entry it is, so they take packed subtractions (two weights per
// instruction) and three-input minima: ten instructions per weight and neighbour against the 45 of a search that
// carries the selector along.  Selectors are found twice per block (start and winner).  A group of lanes owns a row, so the
// row's scale is found and used by the same threads and the row is read from HBM once.
// 4096 x 4096: 679.6 us before (search with selectors for all ten palettes, coefficient tables in local memory,
// a launch of its own for the scales), 159.8 us a call now.
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
__device__ __forceinline__ float min8_abs(const float (&d)[8]) {
  return fminf(min3_abs(min3_abs(min3_abs(d[0], d[1], d[2]), d[3], d[4]), d[5], d[6]), fabsf(d[7]));
}

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

__device__ __forceinline__ int clamp127(int e) { return min(max(e, -127), 127); }

// value / scale, rounded to nearest: the residual correction of a quotient that is off by at most one unit in the last
// place is the correctly rounded quotient when the reciprocal is correctly rounded (Markstein 1990, "Computation of
// elementary functions on the IBM RISC System/6000 processor"); the product with the reciprocal can be off by two, so
// it takes a first correction too.  The last residual has to be exact: it is a multiple of 2^-46 times the quotient's
// and the scale's power of two, which is representable while the two exponents add up to -103 or more.  `normal` keeps
// the scale at 2^-40 or more, and weights below 2^-60 of the scale take the division.
__device__ __forceinline__ float divide_by_scale(float value, float scale, float reciprocal, bool normal) {
  if (!normal || !(fabsf(value) >= scale * 0x1p-60f || value == 0.f)) return __fdiv_rn(value, scale);
  float q = __fmul_rn(value, reciprocal);
  q = __fmaf_rn(__fmaf_rn(-q, scale, value), reciprocal, q);
  return __fmaf_rn(__fmaf_rn(-q, scale, value), reciprocal, q);
}

constexpr int kEncodeThreads = 128;
constexpr int kEncodeWave = 148 * 4;   // blocks of threads resident at once (registers)

// A group of GROUP lanes encodes one row after another (rows group, group + groups, ...): the row's largest magnitude
// first, then one 16-weight block per lane and step.  With gridDim.y > 1 that many groups share a row: each finds the
// largest magnitude for itself (the row comes from L2) and takes every gridDim.y-th step.
template <int GROUP, bool WIDE>
__global__ void __launch_bounds__(kEncodeThreads) encode_kernel(const float *__restrict__ weight, const float *__restrict__ hdiag,
                                                                const float *__restrict__ lut, unsigned long long *__restrict__ blocks,
                                                                float *__restrict__ scales, int M, int K) {
  // selector coefficients: value = a*u + b*z + c (encoder.py:53-70); the fractions are Python doubles rounded to fp32
  __shared__ float coef_a[2][8], coef_b[2][8], coef_c[2][8];
  __shared__ float peak[kEncodeThreads / 32];
  if (threadIdx.x < 16) {
    const int high = threadIdx.x < 8, s = threadIdx.x & 7, n = high ? 7 : 5;
    const int g = s == 0 ? 0 : (s == 1 ? n : s - 1);
    const bool fixed = !high && s >= 6;                  // selectors 6 and 7 of the low mode are -1 and +1
    coef_a[high][s] = fixed ? 0.f : float(double(n - g) / n);
    coef_b[high][s] = fixed ? 0.f : float(double(g) / n);
    coef_c[high][s] = fixed ? (s == 6 ? -1.f : 1.f) : 0.f;
  }
  __syncthreads();
  const int bpr = K / 16;
  const int in_group = threadIdx.x % GROUP, group = threadIdx.x / GROUP;
  constexpr int kGroups = kEncodeThreads / GROUP;
  for (int row0 = blockIdx.x * kGroups; row0 < M; row0 += gridDim.x * kGroups) {
    const int row = row0 + group;
    const bool live = row < M;
    const float4 *w4 = reinterpret_cast<const float4 *>(weight + size_t(live ? row : 0) * K);
    // scale_m = max(|W[m, :]|, 1e-12)
    float m = 0.f;
    if (live) {
#pragma unroll 4
      for (int i = in_group; i < bpr * 4; i += GROUP) {
        const float4 w = w4[i];
        m = fmaxf(fmaxf(m, fmaxf(fabsf(w.x), fabsf(w.y))), fmaxf(fabsf(w.z), fabsf(w.w)));
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
    const float scale = fmaxf(m, 1e-12f), reciprocal = __frcp_rn(scale);
    const bool normal = scale >= 0x1p-40f && scale <= 0x1p60f;
    if (!live) continue;
    if (in_group == 0 && blockIdx.y == 0) scales[row] = scale;

    for (int kb = blockIdx.y * GROUP + in_group; kb < bpr; kb += gridDim.y * GROUP) {
      unsigned long long v2[8], h2[8];
      float vmax = -INFINITY, vmin = INFINITY;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float4 w = w4[kb * 4 + j], g = reinterpret_cast<const float4 *>(hdiag)[kb * 4 + j];
        const float v[4] = {fminf(fmaxf(divide_by_scale(w.x, scale, reciprocal, normal), -1.f), 1.f),
                            fminf(fmaxf(divide_by_scale(w.y, scale, reciprocal, normal), -1.f), 1.f),
                            fminf(fmaxf(divide_by_scale(w.z, scale, reciprocal, normal), -1.f), 1.f),
                            fminf(fmaxf(divide_by_scale(w.w, scale, reciprocal, normal), -1.f), 1.f)};
        vmax = fmaxf(fmaxf(vmax, fmaxf(v[0], v[1])), fmaxf(v[2], v[3]));
        vmin = fminf(fminf(vmin, fminf(v[0], v[1])), fminf(v[2], v[3]));
        v2[2 * j] = pack2(v[0], v[1]);
        v2[2 * j + 1] = pack2(v[2], v[3]);
        h2[2 * j] = pack2(g.x, g.y);
        h2[2 * j + 1] = pack2(g.z, g.w);
      }
      const int e0 = clamp127(int(rintf(__fmul_rn(vmax, 127.f)))), e1 = clamp127(int(rintf(__fmul_rn(vmin, 127.f))));
      const auto palette_row = [&](int q0, int q1) { return lut + (size_t(q1 + 127) * 255 + (q0 + 127)) * 8; };
      unsigned long long start_bits = 0;
      float saa, sbb, sab, say, sby;
      {
        // weighted 2x2 normal equations on the start's selectors (encoder.py:72-84)
        const float4 p_lo = palette_half<WIDE>(palette_row(e0, e1), 0), p_hi = palette_half<WIDE>(palette_row(e0, e1), 1);
        const float p[8] = {p_lo.x, p_lo.y, p_lo.z, p_lo.w, p_hi.x, p_hi.y, p_hi.z, p_hi.w};
        const int high = e0 > e1;
        float taa[16], tbb[16], tab[16], tay[16], tby[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const float v = j & 1 ? hi2(v2[j / 2]) : lo2(v2[j / 2]), h = j & 1 ? hi2(h2[j / 2]) : lo2(h2[j / 2]);
          const int sel = nearest_selector(v, p);
          start_bits |= (unsigned long long)sel << (3 * j);
          const float a = coef_a[high][sel], b = coef_b[high][sel];
          const float target = high ? __fsub_rn(v, 0.f) : __fsub_rn(v, coef_c[0][sel]);
          const float ha = __fmul_rn(h, a), hb = __fmul_rn(h, b);
          taa[j] = __fmul_rn(ha, a);
          tbb[j] = __fmul_rn(hb, b);
          tab[j] = __fmul_rn(ha, b);
          tay[j] = __fmul_rn(ha, target);
          tby[j] = __fmul_rn(hb, target);
        }
        saa = sum16(taa); sbb = sum16(tbb); sab = sum16(tab); say = sum16(tay); sby = sum16(tby);
      }
      const float det = __fsub_rn(__fmul_rn(saa, sbb), __fmul_rn(sab, sab));
      const bool keep = fabsf(det) < 1e-12f;
      const float safe = fmaxf(det, 1e-12f);
      float u = fminf(fmaxf(__fdiv_rn(__fsub_rn(__fmul_rn(say, sbb), __fmul_rn(sby, sab)), safe), -1.f), 1.f);
      float z = fminf(fmaxf(__fdiv_rn(__fsub_rn(__fmul_rn(sby, saa), __fmul_rn(say, sab)), safe), -1.f), 1.f);
      if (keep) {
        u = __fdiv_rn(float(e0), 127.f);
        z = __fdiv_rn(float(e1), 127.f);
      }
      const int c0 = int(rintf(__fmul_rn(u, 127.f))), c1 = int(rintf(__fmul_rn(z, 127.f)));

      // the nine integer neighbours, delta0 outer, delta1 inner; strict "<" keeps the first best (encoder.py:88-101).
      // The next neighbour's palette is requested before this one's errors are computed.
      float best = INFINITY;
      int out = -1;
      const float *first = palette_row(clamp127(c0 - 1), clamp127(c1 - 1));
      float4 p_lo = palette_half<WIDE>(first, 0), p_hi = palette_half<WIDE>(first, 1);
#pragma unroll 1
      for (int n = 0; n < 9; ++n) {
        const int next = min(n + 1, 8);
        const float *ahead = palette_row(clamp127(c0 + next / 3 - 1), clamp127(c1 + next % 3 - 1));
        const float4 next_lo = palette_half<WIDE>(ahead, 0), next_hi = palette_half<WIDE>(ahead, 1);
        unsigned long long d2[8];
        nearest_distances(v2, p_lo, p_hi, d2);
        // (scalar products and sums: with packed multiplies and adds, .rn on both, 4 blocks of 5.6 million came out one
        // neighbour off the reference's, as a fused multiply-add would have it)
        float te[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const float d = j & 1 ? hi2(d2[j / 2]) : lo2(d2[j / 2]), h = j & 1 ? hi2(h2[j / 2]) : lo2(h2[j / 2]);
          te[j] = __fmul_rn(h, __fmul_rn(d, d));
        }
        const float err = sum16(te);
        if (err < best) {
          best = err;
          out = n;
        }
        p_lo = next_lo;
        p_hi = next_hi;
      }
      int out0 = e0, out1 = e1;
      unsigned long long bits = start_bits;
      if (out >= 0) {                                   // (no neighbour wins only when the errors are not numbers)
        out0 = clamp127(c0 + out / 3 - 1);
        out1 = clamp127(c1 + out % 3 - 1);
        const float4 q_lo = palette_half<WIDE>(palette_row(out0, out1), 0), q_hi = palette_half<WIDE>(palette_row(out0, out1), 1);
        const float p[8] = {q_lo.x, q_lo.y, q_lo.z, q_lo.w, q_hi.x, q_hi.y, q_hi.z, q_hi.w};
        bits = 0;
#pragma unroll
        for (int j = 0; j < 16; ++j) bits |= (unsigned long long)nearest_selector(j & 1 ? hi2(v2[j / 2]) : lo2(v2[j / 2]), p) << (3 * j);
      }
      blocks[size_t(row) * bpr + kb] = (unsigned long long)(unsigned(out0) & 0xffu) | ((unsigned long long)(unsigned(out1) & 0xffu) << 8) | (bits << 16);
    }
  }
}

template <int GROUP>
static void launch_encode_rows(const float *weight, const float *hdiag, const float *lut, int M, int K, uint8_t *blocks, float *scales, cudaStream_t stream) {
  const int per_cta = kEncodeThreads / GROUP;
  const int grid = int(std::min<size_t>((size_t(M) + per_cta - 1) / per_cta, size_t(1) << 20));
  // Rows alone fill the chip from about 600 blocks of threads on (four to an SM).  Below that a row is shared, by as many
  // groups as fit one wave and have a step each: 8 x 17408 84.6 -> 11.4 us, 100 x 11200 57.9 -> 16.6, 300 x 11200 74.9 -> 44.3
  // (the kernel that spread single blocks over the chip took 29.2, 61.6 and 153.7).
  const int steps = (K / 16 + GROUP - 1) / GROUP, shares = std::max(1, std::min(kEncodeWave / grid, steps));
  const int rounds = (steps + shares - 1) / shares;   // steps of a group
  const dim3 blocks_of_threads(grid, (steps + rounds - 1) / rounds);
  // a palette may start at any float (a slice of a larger buffer): the wide loads are for tables on a 16-byte boundary
  const auto kernel = reinterpret_cast<uintptr_t>(lut) & 15 ? encode_kernel<GROUP, false> : encode_kernel<GROUP, true>;
  kernel<<<blocks_of_threads, kEncodeThreads, 0, stream>>>(weight, hdiag, lut, reinterpret_cast<unsigned long long *>(blocks), scales, M, K);
}

int launch_encode(const float *weight, const float *hdiag, const float *lut, int M, int K, uint8_t *blocks, float *scales, cudaStream_t stream) {
  // lanes per row: the size that leaves the fewest lanes without a block in the last step of a row, the larger one when
  // equal (a row of 198 blocks is 2 steps of 128 lanes with 58 idle, 4 of 64 with 58 idle, 7 of 32 with 26 idle)
  const auto idle = [&](int group) { return (K / 16 + group - 1) / group * group - K / 16; };
  if (idle(128) <= idle(64) && idle(128) <= idle(32)) launch_encode_rows<128>(weight, hdiag, lut, M, K, blocks, scales, stream);
  else if (idle(64) <= idle(32)) launch_encode_rows<64>(weight, hdiag, lut, M, K, blocks, scales, stream);
  else launch_encode_rows<32>(weight, hdiag, lut, M, K, blocks, scales, stream);
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
