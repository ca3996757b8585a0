// Prefill GEMM for tokens >= prefill_threshold: Y[T, M] = X[T, K] * Wq[M, K]^T on the 5th-generation
// tensor cores (tcgen05.mma, accumulators in TMEM).
//
// Reference counterpart: the five CUTLASS 2.x tiles whose B iterator gathers BC4 texels
// (texelator/cuda/cutlass_texture_mainloop.cu:61-249, _t1/_t2/_t3/_smalln.cu; sm_80 mma.sync,
// two-stage register-staged pipeline).  B200 design, one CTA per MT*128 output rows x BN tokens:
//
//   pre-pass   one small kernel rescales the activations per token by an exact power of two and stores
//              them as fp16 (the decode GEMV's staging) in the chunk-major order of the B operand;
//   (threads below: one CTA an SM; the small form of the narrow tiles has eight producer warps)
//   warps 0-15 producers: 128-bit loads of the tiled BC4 payload, decode in registers exactly like the decode GEMV
//              (masked index fields + HFMA2 -> exact numerators n * 2^-16, n = 7*e0 + g*(e1-e0), as fp16) and
//              tcgen05.st of the A stage into TMEM: the payload's lane order is the 16x256b fragment order, so
//              nothing is shuffled and shared memory holds the activations alone;
//   warp 16    one lane issues the TMA load of the staged X tile (128 columns) per stage
//              through a 3-D tensor map whose rows are 512 contiguous bytes (no multicast);
//   warp 17    allocates TMEM and issues eight tcgen05.mma kind::f16 (A from TMEM, M=128 or a pair's 256, N=BN, K=16)
//              per stage, committing to the stage's "empty" barrier;
//   warps 0-15 epilogue: tcgen05.ld of the fp32 accumulators, * scale_m * 2^s * 65536/889, + bias, one bf16
//              rounding, store.
//
// Numerics are those of the decode GEMV: products of exact integers and exactly rescaled activations,
// fp32 accumulation, weights never rounded to bf16 (the reference rounds bf16(pal*scale); the outputs
// differ by that rounding only, rel-RMS about 1e-3).
//
// Output rows are the MMA M (TMEM lanes) and tokens the MMA N (TMEM columns), so every weight tile
// is decoded once per CTA for all BN tokens.  K is consumed in the same 16-column steps and the
// same order by every tile candidate, so candidates are bitwise identical to each other (the
// reference's admission rule, texelator/autotune.py:160-168).
//
// Every mbarrier wait is bounded: when a wait runs out, the thread records a code in a device status
// word, raises a CTA-wide abort flag, the roles leave their loops, outstanding TMA copies are waited
// for (bounded again), TMEM is freed and the CTA returns.
#include <cuda.h>

#include <map>
#include <mutex>
#include <tuple>

#include "tx_common.cuh"
#include "tx_decode.cuh"

namespace tx {

constexpr int kMmaM = 128;               // rows of a CTA's accumulator (TMEM lanes)
// Eight producer warps a group: warp w reaches the TMEM lanes of quarter w & 3 only, holds one of that quarter's two 16-row
// tiles and decodes whole 128-column units of it.  Two groups take alternate pipeline stages;
// a CTA of one group (tiles up to 128 tokens) is small enough for two on an SM, which then set up, fill their pipelines and store at different
// times (two_an_sm).
constexpr int kLook = 2;                        // units of its row a producer warp keeps in flight as register loads
constexpr unsigned kSpinLimit = 1u << 22;
constexpr unsigned kDrainLimit = 1u << 20;      // polls per stage for copies in flight after an abort
constexpr int kBK = 128;                        // columns per pipeline stage: one unit of the payload
constexpr int kChunks = kBK / 8;                // 16-byte K chunks of the activation tile per stage
constexpr int kAColumns = kBK / 2;              // TMEM columns of one A stage (two fp16 per 32-bit column)

// One tile shape: CTAS x 128 output rows x BN tokens.  The accumulator takes BN columns of every CTA's TMEM, the ring of
// decoded A stages the columns behind it; shared memory holds the activations alone, and with CTAS = 2 each CTA keeps
// half of the tokens (the tensor cores of a pair read both halves).
template <int CTAS, int BN, int GROUPS = 2> struct TileConfig {
  static constexpr int producers = 8 * GROUPS;
  static constexpr int threads = (producers + 2) * 32;        // producer/epilogue warps + TMA warp + MMA warp
  static constexpr int tmem_columns = GROUPS == 2 ? 512 : 256;
  static constexpr int rows = CTAS * kMmaM;
  static constexpr int tokens = BN / CTAS;                    // tokens this CTA stages
  static constexpr int b_lbo = tokens * 16;
  static constexpr int b_stage = kChunks * b_lbo;
  static constexpr int fixed = 1024 /*alignment*/ + 256 /*barriers*/;
  static constexpr int fit_smem = (220 * 1024 - fixed) / b_stage, fit_tmem = (tmem_columns - BN) / kAColumns;
  static constexpr int fit = fit_smem < fit_tmem ? fit_smem : fit_tmem;
  static constexpr int stages = fit > 6 ? 6 : fit;
  static constexpr size_t smem = fixed + size_t(stages) * b_stage;
  static_assert(stages >= 2, "tile does not fit two pipeline stages");
  static_assert(BN + stages * kAColumns <= tmem_columns, "accumulator and A stages must fit TMEM");
  static_assert(tokens % 32 == 0 && BN % 32 == 0 && BN <= 256, "the activation box is made of 32-token runs; N is at most 256");
  static_assert(stages * b_stage >= BN * kMmaM * (CTAS == 1 ? 4 : 2), "the output tile, or its fp32 sums, are staged where the activations were");
};

struct PrefillParams {
  const uint4 *tiles;
  const uint8_t *flags;
  const float *scales;
  const __nv_bfloat16 *bias;
  const float *xmul;   // per-token multiplier 2^s * 65536/889 of the staged activations
  __nv_bfloat16 *y;
  int *status;
  int M, K, KI, MT, T;
  int palette;
  int half_io;   // bias and y are fp16 (the staged activations are fp16 either way)
  float *partial;   // gridDim.z > 1: K is cut into gridDim.z ranges of units and the scaled fp32 sums go to partial[range][T][M]; null: the ranges
                    // of a tile are a cluster that adds them in shared memory
};

// ---- PTX wrappers -------------------------------------------------------------------------------
__device__ __forceinline__ void mbar_init(unsigned bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
// Arrival on the barrier at this shared-memory offset of the CTA `rank` of the cluster.  No cluster scope: it hands over
// TMEM stores (complete since tcgen05.wait::st) and TMA copies that the tensor core reads, nothing that a thread of the
// other CTA loads.  A release at cluster scope waits for all of the thread's loads in flight; with it in a relay thread, and
// an acquire to match, 5120x17408 with 4096 tokens took 874 us (now 680; 34816x5120 1357, now 1225).
__device__ __forceinline__ void mbar_arrive_at(unsigned bar, unsigned rank) {
  asm volatile(
      "{\n\t.reg .b32 remote;\n\t"
      "mapa.shared::cluster.u32 remote, %0, %1;\n\t"
      "mbarrier.arrive.shared::cluster.b64 _, [remote];\n\t}" ::"r"(bar), "r"(rank) : "memory");
}
__device__ __forceinline__ void mbar_arrive(unsigned bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(unsigned bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(unsigned bar, unsigned parity) {
  unsigned done;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(done) : "r"(bar), "r"(parity) : "memory");
  return done != 0;
}
// Bounded wait; returns false (after recording `code`) when the limit is reached or the CTA aborted.
__device__ __forceinline__ bool mbar_wait(unsigned bar, unsigned parity, volatile int *abort_flag, int *status, int code) {
  for (unsigned spin = 0; spin < kSpinLimit; ++spin) {
    if (mbar_try_wait(bar, parity)) return true;
    if (*abort_flag) return false;
  }
  atomicCAS(status, 0, code);
  *abort_flag = 1;
  return false;
}
__device__ __forceinline__ void tma_load_3d(unsigned dst, const CUtensorMap *map, unsigned bar, int c0, int c1, int c2) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];"
      ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2) : "memory");
}
// one lane of a converged warp; the compiler keeps what it guards on the uniform datapath, which tcgen05.mma wants
__device__ __forceinline__ bool elect_one() {
  unsigned elected;
  asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(elected));
  return elected != 0;
}
// D[tmem] (+)= A[tmem] * B[smem]: M = CTAS * 128, fp16 operands, fp32 accumulation
template <int CTAS>
__device__ __forceinline__ void umma_f16(unsigned tmem_d, unsigned tmem_a, unsigned long long bdesc, unsigned idesc, unsigned accumulate) {
  if (CTAS == 1)
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
  else
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
// arrives at the barrier (of both CTAs of a pair) when the MMAs issued so far are complete
template <int CTAS>
__device__ __forceinline__ void umma_commit(unsigned bar) {
  if (CTAS == 1)
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
  else
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                 ::"r"(bar), "h"((unsigned short)3) : "memory");
}
// Sixteen TMEM lanes x 32 columns in the fragment order of mma.sync: registers 4j, 4j+1 of lane (g, t) are columns
// 8j + 2t, 8j + 2t + 1 of TMEM lane g, registers 4j+2, 4j+3 those of lane g + 8.
__device__ __forceinline__ void tmem_store_fragments(unsigned taddr, const unsigned (&q)[8], const unsigned (&r)[8]) {
  asm volatile(
      "tcgen05.st.sync.aligned.16x256b.x4.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
      ::"r"(taddr), "r"(q[0]), "r"(q[1]), "r"(r[0]), "r"(r[1]), "r"(q[2]), "r"(q[3]), "r"(r[2]), "r"(r[3]),
        "r"(q[4]), "r"(q[5]), "r"(r[4]), "r"(r[5]), "r"(q[6]), "r"(q[7]), "r"(r[6]), "r"(r[7]) : "memory");
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_load32(unsigned taddr, unsigned (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr) : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
// K-major, no-swizzle shared-memory matrix descriptor: 8-row groups `sbo` bytes apart, 16-byte K chunks
// `lbo` bytes apart (canonical layout ((8,m),(8,2)):((16B,SBO),(2B,LBO)) for 16-bit elements).
__device__ __forceinline__ unsigned long long smem_desc(unsigned addr, unsigned lbo, unsigned sbo) {
  return (unsigned long long)((addr >> 4) & 0x3FFF) | ((unsigned long long)((lbo >> 4) & 0x3FFF) << 16) |
         ((unsigned long long)((sbo >> 4) & 0x3FFF) << 32) | (1ull << 46);
}

// Sums of 32 tokens (a register each) of a lane's row, scaled and rounded, to out[token * kMmaM].  Eight at a time and step by step, two to a
// conversion: with all steps of one token behind one another a chunk took 1250 cycles of sixteen warps.
template <bool HALF>
__device__ __forceinline__ void round_to(uint16_t *out, const unsigned (&v)[32], float row_scale, float bias, float token_scale) {
#pragma unroll
  for (int j0 = 0; j0 < 32; j0 += 8) {
    float value[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) value[j] = __shfl_sync(0xffffffffu, token_scale, j0 + j);
#pragma unroll
    for (int j = 0; j < 8; ++j) value[j] = fmaf(__uint_as_float(v[j0 + j]), row_scale * value[j], bias);
#pragma unroll
    for (int j = 0; j < 8; j += 2) {
      unsigned pair;
      if (HALF) {
        const __half2 h = __floats2half2_rn(value[j], value[j + 1]);
        pair = *reinterpret_cast<const unsigned *>(&h);
      } else {
        const __nv_bfloat162 h = __floats2bfloat162_rn(value[j], value[j + 1]);
        pair = *reinterpret_cast<const unsigned *>(&h);
      }
      out[(j0 + j) * kMmaM] = uint16_t(pair);
      out[(j0 + j + 1) * kMmaM] = uint16_t(pair >> 16);
    }
  }
}
// the same for a K range: fp32, to dst[token * M], of the first `last` tokens
__device__ __forceinline__ void scale_to(float *dst, int M, const unsigned (&v)[32], float row_scale, float token_scale, int last) {
#pragma unroll
  for (int j0 = 0; j0 < 32; j0 += 8) {
    float value[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) value[j] = __uint_as_float(v[j0 + j]) * (row_scale * __shfl_sync(0xffffffffu, token_scale, j0 + j));
#pragma unroll
    for (int j = 0; j < 8; ++j)
      if (j0 + j < last) dst[size_t(j0 + j) * M] = value[j];
  }
}

// Activation staging for the GEMM: per token an exact power-of-two rescale to fp16 (the decode GEMV's
// arithmetic), stored chunk-major -- out[(chunk * padded_tokens + token) * 8 .. +8], padded_tokens a
// multiple of 32 -- which is the K-major core-matrix order of the B operand.  A TMA box then copies
// runs of 32 tokens x 16 bytes = 512 contiguous bytes; with the row-major layout every 16-byte piece
// was a TMA row of its own and the load, not the tensor pipe, set the pace of the wide tiles.
//
// A CTA stages `per_cta` tokens (1, 2 or 4: as many as leave every SM a CTA) in one trip to global memory: the rows wait in
// shared memory while the magnitude scan finishes, then are converted and written out with neighbouring lanes on
// neighbouring tokens.  Rows that do not fit are read again instead.
//
// Order of K.  A producer lane (g, t) holds whole 16-column blocks, and TMEM wants from it four K elements of every
// 16-element MMA step, so the K elements are numbered the way the lanes hold them: element 4t + i of step j of a
// 64-column half unit is column 16t + 4j + i.  The activations are written in that order here.
constexpr int kStageThreads = 512;
constexpr size_t kStageSmem = 200 * 1024;
static size_t stage_row_bytes(int K) { return size_t(K) * 2 + 16; }   // + 16: rows start on different banks
__global__ void __launch_bounds__(kStageThreads) stage_activations_kernel(const __nv_bfloat16 *__restrict__ x, __half *__restrict__ out,
                                                                          float *__restrict__ xmul, int K, int KP, int tokens,
                                                                          int padded_tokens, int per_cta, int rows_fit, int half_in) {
  extern __shared__ __align__(16) uint8_t rows_smem[];
  __shared__ unsigned warp_max[kStageThreads / 32];
  grid_dependency_wait();        // the scratch may still be read by an earlier call's tile kernel, and x be on its way
  grid_launch_dependents();      // the tile kernel may set up (barriers, TMEM, first weight loads) while this one runs
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int chunks = K / 8, padded = KP / 8, row_bytes = K * 2 + 16;
  const int first = blockIdx.x * per_cta, per_token = kStageThreads / per_cta;   // threads that read one row
  {
    const int j = threadIdx.x / per_token, tok = first + j;
    unsigned m = 0;
    if (tok < tokens && (rows_fit || !half_in)) {
      const uint4 *src = reinterpret_cast<const uint4 *>(x + size_t(tok) * K);
      uint4 *row = reinterpret_cast<uint4 *>(rows_smem + size_t(j) * row_bytes);
#pragma unroll 8
      for (int i = threadIdx.x % per_token; i < chunks; i += per_token) {
        const uint4 v = __ldcg(src + i);
        if (rows_fit) row[i] = v;
        if (!half_in) m = max(m, chunk_absmax(v));
      }
    }
    m = __reduce_max_sync(0xffffffffu, m);
    if (lane == 0) warp_max[warp] = m;
  }
  __syncthreads();
  const int j = threadIdx.x % per_cta, tok = first + j;
  const int warps = per_token / 32;
  unsigned m = 0;
  for (int w = 0; w < warps; ++w) m = max(m, warp_max[j * warps + w]);
  float mult, inverse;
  token_scaling(m, mult, inverse);
  if (half_in) inverse = 1.f;   // fp16 activations (x then points to fp16) are the operand as they are
  if (int(threadIdx.x) < per_cta && tok < tokens) xmul[tok] = inverse * kNumeratorScale;
  uint4 *dst = reinterpret_cast<uint4 *>(out);
  const uint8_t *row = rows_smem + size_t(j) * row_bytes;
  const __nv_bfloat16 *again = x + size_t(tok < tokens ? tok : 0) * K;
  const auto four = [&](int column) {
    return rows_fit ? *reinterpret_cast<const uint2 *>(row + size_t(column) * 2) : __ldcg(reinterpret_cast<const uint2 *>(again + column));
  };
#pragma unroll 4
  for (int chunk = threadIdx.x / per_cta; chunk < padded; chunk += per_token) {
    // chunk 2j + c of a half unit: columns 16(2c) + 4j .. + 3 and 16(2c + 1) + 4j .. + 3
    const int column = (chunk >> 3) * 64 + (chunk & 1) * 32 + ((chunk >> 1) & 3) * 4;
    uint4 v = make_uint4(0, 0, 0, 0);
    if (tok < tokens) {
      if (column < K) {
        const uint2 low = four(column);
        v.x = low.x;
        v.y = low.y;
      }
      if (column + 16 < K) {
        const uint2 high = four(column + 16);
        v.z = high.x;
        v.w = high.y;
      }
      if (!half_in) v = convert_chunk(v, mult);
    }
    dst[size_t(chunk) * padded_tokens + tok] = v;
  }
}

// Few tokens with long rows: a cluster a row (stage_split_row)
__global__ void __launch_bounds__(kSplitThreads) stage_split_kernel(const __nv_bfloat16 *__restrict__ x, __half *__restrict__ out, float *__restrict__ xmul, int K,
                                                                    int padded_tokens, int half_in) {
  grid_dependency_wait();        // the scratch may still be read by an earlier call's tile kernel, and x be on its way
  grid_launch_dependents();
  const uint4 *row = reinterpret_cast<const uint4 *>(x + size_t(blockIdx.y) * K);
  stage_split_row(reinterpret_cast<uint4 *>(out), xmul, K, padded_tokens, half_in != 0, [&](int i) { return __ldcg(row + i); });
}

template <int CTAS, int BN, bool GENERIC, int GROUPS>
__global__ void __launch_bounds__(TileConfig<CTAS, BN, GROUPS>::threads, GROUPS == 2 ? 1 : 2)
prefill_umma_kernel(const PrefillParams p, const __grid_constant__ CUtensorMap x_map) {
  using Cfg = TileConfig<CTAS, BN, GROUPS>;
  constexpr int kProducerWarps = Cfg::producers, kGroups = GROUPS, kTmaWarp = kProducerWarps, kMmaWarp = kProducerWarps + 1;
  constexpr int S = Cfg::stages;
  extern __shared__ uint8_t smem_raw[];
  const unsigned sbase = unsigned(__cvta_generic_to_shared(smem_raw));
  const unsigned b_s = (sbase + 1023) & ~1023u;          // activation stages, then barriers + small state (256 bytes)
  const unsigned bars_s = b_s + S * Cfg::b_stage;
  uint8_t *bars_g = smem_raw + (bars_s - sbase);
  const unsigned full = bars_s, empty = bars_s + 8 * S, accum = bars_s + 16 * S;
  volatile int *abort_flag = reinterpret_cast<volatile int *>(bars_g + 200);
  unsigned *tmem_slot = reinterpret_cast<unsigned *>(bars_g + 208);

  const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const unsigned rank = CTAS == 2 ? blockIdx.x & 1 : 0;  // the pair is cut from blockIdx.x; rank 0 issues its MMAs
  // Launched with programmatic stream serialisation behind the staging kernel: everything up to the first read
  // of the staged activations (the TMA lane) or of the token multipliers (the epilogue) touches only the
  // immutable payload and this CTA's own memory and may run while the staging kernel is still at work.
  grid_launch_dependents();
  // this CTA's range of 128-column units (the whole row unless the launch cuts K); one unit is one pipeline stage
  const int u0 = int(blockIdx.z) * p.KI / int(gridDim.z), u1 = (int(blockIdx.z) + 1) * p.KI / int(gridDim.z);
  const int KT = u1 - u0;
  const int row0 = blockIdx.x * kMmaM, tok0 = blockIdx.y * BN;
  const bool merge = CTAS == 1 && GROUPS == 2 && gridDim.z > 1 && p.partial == nullptr;

  if (tid == 0) {
    for (int s = 0; s < S; ++s) {
      // the producer warps and the TMA lane of a stage.  A pair counts on its issuing CTA: both CTAs' producers arrive there
      // themselves, for the other CTA's TMA lane a relay does, and the other CTA's barrier takes its copy alone.
      mbar_init(full + 8 * s, CTAS == 1 ? kProducerWarps / kGroups + 1 : rank == 0 ? CTAS * (kProducerWarps / kGroups + 1) : 1);
      mbar_init(empty + 8 * s, 1);
    }
    mbar_init(accum, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == kMmaWarp) {
    if (CTAS == 1) {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(bars_s + 208), "r"(unsigned(Cfg::tmem_columns)) : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    } else {
      asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(bars_s + 208), "r"(unsigned(Cfg::tmem_columns)) : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
  }
  // The producers' first loads leave before the barrier: set-up takes 940 cycles, a load from HBM as long.
  const int quarter = warp & 3, pair = (warp >> 2) & 1, group = warp >> 3;
  const int rt = blockIdx.x * (kMmaM / 16) + quarter * 2 + pair;
  // (row tiles past the end of the matrix decode tile 0 again: their accumulator rows are never stored)
  const uint4 *src = p.tiles + size_t(rt < p.MT ? rt : 0) * p.KI * 64 + lane;
  const uint8_t *flags = p.flags + size_t(rt < p.MT ? rt : 0) * p.KI;
  uint4 pend[kLook][2];
  unsigned flag[kLook];
  auto fetch = [&](int slot, int unit) {
    if (unit < u1) {
      pend[slot][0] = ldg_stream(src + size_t(unit) * 64);
      pend[slot][1] = ldg_stream(src + size_t(unit) * 64 + 32);
      if (GENERIC) flag[slot] = flags[unit];
    }
  };
  if (warp < kProducerWarps) {
#pragma unroll
    for (int slot = 0; slot < kLook; ++slot) fetch(slot, u0 + group + slot * kGroups);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (CTAS == 2) cluster_sync();                         // the other CTA's barriers exist
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const unsigned tmem_base = *tmem_slot;

  if (warp < kProducerWarps) {
    // ---------------- producers: BC4 -> fp16 A stage in TMEM ----------------
    const unsigned a_lane = tmem_base + (unsigned(quarter * 32 + pair * 16) << 16) + BN;
    int s = group % S;
    unsigned parity = 1;                                 // of the stage's previous release; a fresh barrier passes
    bool ok = true;
    for (int base = u0 + group; base < u1 && ok; base += kLook * kGroups) {
#pragma unroll
      for (int slot = 0; slot < kLook; ++slot) {
        const int unit = base + slot * kGroups;
        if (unit >= u1 || !ok) break;                    // warp-uniform
        const uint4 q = pend[slot][0], r = pend[slot][1];   // duos of rows g and g + 8
        const bool low = GENERIC && flag[slot];          // warp-uniform: the unit's flag
        fetch(slot, unit + kLook * kGroups);
        // Decode before waiting for the stage: a warp takes a few hundred cycles over a unit, and the time from a
        // stage's release to its next use is what sets the pace.
        unsigned a[2][2][8];                             // [block column][row g / g + 8]: exact numerators n * 2^-16 as fp16x2
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const uint4 duo = h == 0 ? q : r;
          if (GENERIC && p.palette == TX_PALETTE_HARDWARE) {   // uniform
            const DuoConstants c = duo_constants<true>(duo.w);
            decode_duo_first<true>(duo, c, a[0][h]);
            decode_duo_second<true>(duo, c, a[1][h]);
          } else {
            const DuoConstants c = duo_constants<false>(duo.w);
            decode_duo_first(duo, c, a[0][h]);
            decode_duo_second(duo, c, a[1][h]);
          }
          if (low) {
            if (duo_block_is_low(duo, 0)) decode_block_low(duo, 0, a[0][h], p.palette);
            if (duo_block_is_low(duo, 1)) decode_block_low(duo, 1, a[1][h], p.palette);
          }
        }
        ok = __all_sync(0xffffffffu, mbar_wait(empty + 8 * s, parity, abort_flag, p.status, 1));
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        tmem_store_fragments(a_lane + unsigned(s * kAColumns), a[0][0], a[0][1]);
        tmem_store_fragments(a_lane + unsigned(s * kAColumns + kAColumns / 2), a[1][0], a[1][1]);
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) {
          if (CTAS == 1 || rank == 0) mbar_arrive(full + 8 * s);
          else mbar_arrive_at(full + 8 * s, 0);
        }
        s += kGroups;
        if (s >= S) {
          s -= S;
          parity ^= 1;
        }
      }
    }
  } else if (warp == kTmaWarp) {
    // ---------------- TMA: this CTA's tokens of the staged X tile, 128 columns per stage ----------------
    if (lane == 0) {
      grid_dependency_wait();              // the staged activations are complete
      int issued = 0, s = 0;
      unsigned parity = 1;
      for (int kt = 0; kt < KT; ++kt) {
        if (!mbar_wait(empty + 8 * s, parity, abort_flag, p.status, 2)) break;
        mbar_expect_tx(full + 8 * s, Cfg::b_stage);
        tma_load_3d(b_s + s * Cfg::b_stage, &x_map, full + 8 * s, 0, (tok0 + int(rank) * Cfg::tokens) / 32, (u0 + kt) * kChunks);
        issued = kt + 1;
        if (++s == S) {
          s = 0;
          parity ^= 1;
        }
      }
      if (*abort_flag) {
        // give copies that were issued but never consumed time (bounded) to land before the CTA exits; the wait ends early
        // where a stage's producers arrived too, and is a delay where they left before it
        for (int kt = issued > S ? issued - S : 0; kt < issued; ++kt)
          for (unsigned spin = 0; spin < kDrainLimit && !mbar_try_wait(full + 8 * (kt % S), (kt / S) & 1); ++spin) {}
      }
    }
  } else if (rank == 0) {
    // ---------------- MMA issue ----------------
    // One instruction stream feeds the tensor core, and what it spends on a stage beyond the MMAs' own time leaves the core
    // idle.  A single lane in a divergent branch, with two barriers a stage and descriptors built on the spot, spent
    // 1240 cycles on a stage whatever the tile (a 256-token stage is 1024 cycles of MMA): hence a converged warp with
    // one elected lane, one barrier a stage and descriptors that only need an addition.
    // D = f32 (bits 4-5 = 1), A = B = f16 (format 0), both K-major, N at bit 17, M at bit 24
    constexpr unsigned idesc = (1u << 4) | (unsigned(BN >> 3) << 17) | (unsigned(Cfg::rows >> 4) << 24);
    const unsigned long long bdesc = smem_desc(b_s, Cfg::b_lbo, 128);
    const unsigned tmem_d = __shfl_sync(0xffffffffu, tmem_base, 0);
    int s = 0;
    unsigned parity = 0;
    bool ok = true;
    for (int kt = 0; kt < KT; ++kt) {
      ok = __all_sync(0xffffffffu, mbar_wait(full + 8 * s, parity, abort_flag, p.status, 3));
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      if (elect_one()) {
        const unsigned long long stage_desc = bdesc + unsigned(s * (Cfg::b_stage >> 4));
        const unsigned stage_a = tmem_d + unsigned(BN + s * kAColumns);
#pragma unroll
        for (int j = 0; j < kBK / 16; ++j)
          umma_f16<CTAS>(tmem_d, stage_a + unsigned(j * 8), stage_desc + unsigned(j * 2 * (Cfg::b_lbo >> 4)), idesc, j ? 1u : unsigned(kt != 0));
        umma_commit<CTAS>(empty + 8 * s);  // frees the stage when these MMAs have read it
      }
      __syncwarp();
      if (++s == S) {
        s = 0;
        parity ^= 1;
      }
    }
    if (ok && elect_one()) umma_commit<CTAS>(accum);   // accumulators complete
    __syncwarp();
  } else if (lane == 0) {
    // ---------------- second CTA of a pair: tell the issuing CTA when this one's activations of a stage are there ----------------
    int s = 0;
    unsigned parity = 0;
    for (int kt = 0; kt < KT; ++kt) {
      if (!mbar_wait(full + 8 * s, parity, abort_flag, p.status, 3)) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      mbar_arrive_at(full + 8 * s, 0);
      if (++s == S) {
        s = 0;
        parity ^= 1;
      }
    }
  }

  // ---------------- epilogue: TMEM -> registers -> y ----------------
  if (warp < kProducerWarps) {
    grid_dependency_wait();                // xmul comes from the staging kernel
    // What the sums are multiplied with is fetched before they are waited for: behind the wait the three loads came one after another, 2500 of
    // 26000 cycles with sixteen stages of 256 tokens and of 9000 with six of 64.
    const int row = row0 + quarter * 32 + lane;
    const float row_scale = row < p.M ? p.scales[row] : 0.f;
    const float bias = (row < p.M && p.bias)
                           ? (p.half_io ? __half2float(reinterpret_cast<const __half *>(p.bias)[row]) : __bfloat162float(p.bias[row]))
                           : 0.f;
    constexpr int kParts = kProducerWarps / 4, kMost = (BN / 32 + kParts - 1) / kParts;   // the warps of one lane quarter share its BN/32 accumulator chunks
    float token_scale[kMost];
#pragma unroll
    for (int i = 0; i < kMost; ++i) {
      const int tok = tok0 + ((warp >> 2) + i * kParts) * 32 + lane;
      token_scale[i] = tok < p.T ? __ldcg(p.xmul + tok) : 0.f;
    }
    const bool ready = __all_sync(0xffffffffu, mbar_wait(accum, 0, abort_flag, p.status, 5));
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (ready && merge) {
      float *sums = reinterpret_cast<float *>(smem_raw + (b_s - sbase));        // [BN][128 rows], where the activations were
#pragma unroll
      for (int i = 0; i < kMost; ++i) {
        const int c = (warp >> 2) + i * kParts;
        if (c >= BN / 32) break;
        unsigned v[32];
        tmem_load32(tmem_base + (unsigned(quarter * 32) << 16) + unsigned(c * 32), v);
        scale_to(sums + c * 32 * kMmaM + quarter * 32 + lane, kMmaM, v, row_scale, token_scale[i], 32);
      }
    } else if (GROUPS == 2 && ready && gridDim.z > 1) {                        // (two_an_sm: the small form has one range)
#pragma unroll
      for (int i = 0; i < kMost; ++i) {
        const int c = (warp >> 2) + i * kParts;
        if (c >= BN / 32) break;
        float *dst = p.partial + (size_t(blockIdx.z) * p.T + tok0 + c * 32) * p.M + row;
        unsigned v[32];
        tmem_load32(tmem_base + (unsigned(quarter * 32) << 16) + unsigned(c * 32), v);
        scale_to(dst, p.M, v, row_scale, token_scale[i], row < p.M ? p.T - tok0 - c * 32 : 0);
      }
    } else if (ready) {
      // A lane holds one output row, so stores from here would be 64-byte pieces; the tile goes through shared memory (the
      // activation stages are free now) and leaves as runs of 256 bytes.
      uint16_t *out = reinterpret_cast<uint16_t *>(smem_raw + (b_s - sbase));   // [BN][128 rows]
#pragma unroll
      for (int i = 0; i < kMost; ++i) {
        const int c = (warp >> 2) + i * kParts;
        if (c >= BN / 32) break;
        unsigned v[32];
        tmem_load32(tmem_base + (unsigned(quarter * 32) << 16) + unsigned(c * 32), v);
        uint16_t *to = out + c * 32 * kMmaM + quarter * 32 + lane;
        if (p.half_io) round_to<true>(to, v, row_scale, bias, token_scale[i]);   // (uniform)
        else round_to<false>(to, v, row_scale, bias, token_scale[i]);
      }
    }
    asm volatile("bar.sync 1, %0;" ::"n"(kProducerWarps * 32) : "memory");
    if (ready && gridDim.z == 1) {
      const uint8_t *out = smem_raw + (b_s - sbase);
      const int rows = min(kMmaM, p.M - row0), last = min(BN, p.T - tok0);
      __nv_bfloat16 *dst = p.y + size_t(tok0) * p.M + row0;
      if (p.M % 8 == 0) {                  // rows of y are 16-byte aligned
        for (int i = tid; i < last * (kMmaM / 8); i += kProducerWarps * 32) {
          const int tok = i / (kMmaM / 8), part = i % (kMmaM / 8);
          if (part * 8 < rows)
            *reinterpret_cast<uint4 *>(dst + size_t(tok) * p.M + part * 8) = *reinterpret_cast<const uint4 *>(out + (tok * kMmaM + part * 8) * 2);
        }
      } else {
        for (int i = tid; i < last * kMmaM; i += kProducerWarps * 32) {
          const int tok = i / kMmaM, r = i % kMmaM;
          if (r < rows) dst[size_t(tok) * p.M + r] = reinterpret_cast<const __nv_bfloat16 *>(out)[i];
        }
      }
    }
  }
  if (merge) {
    // The ranges of this tile, in order, bias, one rounding: launch_combine's sums to the bit, without its launch and without [ranges][T][M] floats
    // through global memory.  A CTA takes every gridDim.z-th token, a warp a token, a lane four rows (a row of sums is one conflict-free read).
    __syncwarp();                          // (the cluster barrier wants whole warps, and the roles end in single lanes)
    cluster_sync();
    const bool whole = !*abort_flag;       // (an abort is reported; what this CTA would add is not there)
    if (warp < kProducerWarps && whole) {
      const int row = row0 + lane * 4, rows = min(4, p.M - row), last = min(BN, p.T - tok0), ranges = int(gridDim.z);
      const bool wide = p.M % 4 == 0;      // rows of y are 8-byte aligned
      float bias[4] = {};
      if (p.bias) {
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (i < rows) bias[i] = p.half_io ? __half2float(reinterpret_cast<const __half *>(p.bias)[row + i]) : __bfloat162float(p.bias[row + i]);
      }
      for (int tok = int(blockIdx.z) + ranges * warp; tok < last; tok += ranges * kProducerWarps) {
        const unsigned at = b_s + unsigned((tok * kMmaM + lane * 4) * 4);
        float sum[4] = {};
        for (int r = 0; r < ranges; ++r) {
          float4 part;
          asm volatile("{\n\t.reg .b32 remote;\n\tmapa.shared::cluster.u32 remote, %4, %5;\n\tld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [remote];\n\t}"
                       : "=f"(part.x), "=f"(part.y), "=f"(part.z), "=f"(part.w) : "r"(at), "r"(r) : "memory");
          sum[0] += part.x;
          sum[1] += part.y;
          sum[2] += part.z;
          sum[3] += part.w;
        }
        uint16_t out[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          if (p.bias) sum[i] += bias[i];
          out[i] = p.half_io ? __half_as_ushort(__float2half_rn(sum[i])) : __bfloat16_as_ushort(__float2bfloat16(sum[i]));
        }
        uint16_t *dst = reinterpret_cast<uint16_t *>(p.y) + size_t(tok0 + tok) * p.M + row;
        if (wide) {
          if (rows == 4) *reinterpret_cast<uint2 *>(dst) = make_uint2(out[0] | (unsigned(out[1]) << 16), out[2] | (unsigned(out[3]) << 16));
        } else {
#pragma unroll
          for (int i = 0; i < 4; ++i)
            if (i < rows) dst[i] = out[i];
        }
      }
    }
    __syncwarp();
    cluster_sync();                        // no CTA leaves while another reads its sums
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (CTAS == 2) cluster_sync();           // neither CTA leaves while the other's tensor core or barriers may still reach it
  if (warp == kMmaWarp) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (CTAS == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(unsigned(Cfg::tmem_columns)) : "memory");
    else asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(unsigned(Cfg::tmem_columns)) : "memory");
  }
}

// ---- host side ------------------------------------------------------------------------------------
using EncodeTiled = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                 const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                 CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiled encode_tiled_entry() {
  static EncodeTiled entry = [] {
    void *fn = nullptr;
    cudaDriverEntryPointQueryResult query;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &query) != cudaSuccess ||
        query != cudaDriverEntryPointSuccess)
      fn = nullptr;
    return reinterpret_cast<EncodeTiled>(fn);
  }();
  return entry;
}

// Tile candidates behind the reference's backend ids 5..9 (texelator/autotune.py:16-22):
//   5: 128 rows x 256 tokens (baseline)   6: 256 x 256 (a pair of CTAs)   7: 128 x 128   8: 128 x 64   9: 128 x 192
// (192 tokens: 5120-row matrices at 512+ tokens launch 120 CTAs instead of 80 or 160 on the 148 SMs)
// Tall tiles re-read the activations less often (tensor-bound prompts); narrow ones suit short prompts
// where the weight stream is the bound.
bool prefill_tile_eligible(const Handle *h, int backend, int tokens) {
  return backend >= 5 && backend <= 9 && tokens >= 1 && h->K % 16 == 0 && encode_tiled_entry() != nullptr;
}

// Short prompts on matrices with few rows leave most SMs without a CTA (5120 rows = 40 CTAs of 128 rows): K is
// then cut into ranges, one CTA per (row block, token block, range), whose fp32 sums are added in the order of the ranges.  The
// number of ranges depends on the matrix and the token count only -- never on the tile -- so that all tiles keep
// adding in the same order and stay bitwise identical to each other (the autotuner's admission rule).
static int prefill_k_ranges(const Handle *h, int tokens, const Workspace *ws) {
  const int blocks = ((h->M + 127) / 128) * ((tokens + 127) / 128);
  int ranges = std::min(std::min(ws->sm_count / std::max(blocks, 1), 8), h->KI / 4);
  while (ranges > 1 && size_t(ranges) * tokens * h->M > ws->partial_floats) --ranges;
  return std::max(ranges, 1);
}

// Whether a tile of at most 128 tokens runs as two small CTAs an SM (half the producers, registers and TMEM each).  A CTA alone on its SM spends
// 3 to 4 us before and after its stages with the tensor core and the memory idle, and 272 CTAs on 148 SMs cost as much as 296; two on an SM fill
// each other's gaps.  They lose where rounding the grid up to two an SM costs a wave and the rows are long enough to show it.  One / two an SM, us a
// call from HBM, waves of one an SM before the figures -- 64 tokens: 24576x1024 2: 11.9 / 9.6; 22016x2048 2: 16.3 / 14.2; 34816x5120 2: 32.8 / 30.3;
// 57344x8192 4: 85.9 / 79.6.  With the 128-token tile: 22016x2048 2: 20.1 / 17.5, 3: 29.1 / 27.1, 7: 65.0 / 59.8; 19200x4096 3: 43.0 / 44.9,
// 7: 106.4 / 101.0; 28672x8192 4: 100.3 / 92.8, 5: 141.6 / 144.1; 24576x1024 8: 52.0 / 38.6; 5120x17408 9: 492 / 563.
//
// The generic instance spends longer on a unit than the gaps last, so it gains on short rows and where there are many waves.  Under the texture palette, 64
// tokens: 22016x2048 2: 21.1 / 21.4, 34816x5120 2: 44.8 / 47.3, 34816x8192 2: 66.6 / 71.6, 57344x3072 4: 53.7 / 52.7, 57344x8192 4: 123.7 / 127.0; with the
// 128-token tile: 22016x2048 7: 77.7 / 73.1, 22016x3072 7: 107.9 / 106.3, 5120x17408 2: 147.8 / 158.0, 22016x17408 7: 557 / 581.
static bool two_an_sm(long ctas, int ranges, int units, int sm_count, bool generic) {
  const long one = (ctas + sm_count - 1) / sm_count, two = (ctas + 2 * sm_count - 1) / (2 * sm_count);
  if (ranges != 1 || one < 2) return false;
  if (units <= 16) return true;
  if (generic) return units <= 32 && one >= 4 && (2 * two <= one || one >= 7);
  return 2 * two <= one || (one >= 7 && units <= 64);
}

// The tile of handles without a tuned backend (ids 0..4; 5..9 name one): all tiles give the same bits, so only time decides.
// A wave of CTAs takes its 128-column stages at the pace of the MMAs or, below 128 tokens, of the producers, plus
// what a CTA spends before and after them (TMEM, first loads, epilogue).  Measured on 5120x17408 with 512 tokens
// (136 stages): 0.30, 0.35, 0.50 and 0.67 us a stage for 64, 128, 192 and 256 tokens and about 4 us a CTA; the tile with
// the smallest sum over the waves wins, the wider one on a tie (it reads the activations less often).  The sums are those of one CTA an SM also where
// two_an_sm would take two: the line then lies a little late for short rows (24576x1024 with 700 tokens: 128-token tile 38.6, 192 tokens 42.5 us).
// The pair tile (id 6) is left out: against the 256-token tile it measured between 6 % less and 13 % more for 512 to 4096 tokens, by the
// GPU's power state more than by shape, and never less below that.
//
// Up to eight tokens (a threshold below the default of 16) the decode kernel keeps the call: it pays one group of MMA columns
// there, and two from nine on.  Decode kernel against the 64-token tile, us a call from HBM with one, eight, nine and fifteen
// tokens: 256x2048 2.7 / 5.9, 3.8 / 6.0, 4.5 / 6.0, 5.0 / 6.3; 2560x2048 3.4 / 6.1, 4.5 / 6.1, 5.3 / 6.2, 5.7 / 6.4; 5120x5120 6.2 / 9.3, 9.3 / 9.6,
// 11.1 / 9.6, 11.8 / 10.2; 22016x2048 8.1 / 13.4, 12.7 / 13.4, 14.8 / 13.5, 17.0 / 13.5; 34816x5120 22.6 / 28.6, 29.0 / 28.7, 35.1 / 28.9, 38.7 / 29.4.
// From nine tokens on the tile is the faster one but on matrices of few rows.
//
// Distance from 64 bits, tile against decode kernel, which adds a row in sixteen shorter chains: on Gaussian activations
// both end at the output's rounding (fp16, 11008x2048, 160 tokens: 2.0759e-4 and 2.0757e-4 of the result; bf16 equal to
// five digits).  Where the sum cancels to a 500th of its terms the one chain shows: 1.5e-6 against 4.5e-7 of the
// terms' norm.  A caller who wants the shorter chains for prompts raises the handle's threshold.
constexpr int kStreamedTokens = 8;
int prefill_choose_backend(const Handle *h, int tokens) {
  if (tokens <= kStreamedTokens) return 0;
  const Workspace *ws = workspace_for(h->device);
  if (!ws) return 5;
  const struct { int backend, bn, stage; } tiles[4] = {{5, 256, 67}, {9, 192, 50}, {7, 128, 35}, {8, 64, 30}};   // stage: 10 ns
  const int ranges = prefill_k_ranges(h, tokens, ws), stages = (h->KI + ranges - 1) / ranges;
  const long blocks = long((h->M + 127) / 128) * ranges;
  long best = 0;
  int pick = 5;
  for (const auto &tile : tiles) {
    const long waves = (blocks * ((tokens + tile.bn - 1) / tile.bn) + ws->sm_count - 1) / ws->sm_count;
    const long cost = waves * (400 + long(stages) * tile.stage);
    if (best == 0 || cost < best) {
      best = cost;
      pick = tile.backend;
    }
  }
  return pick;
}

// the lean instances decode high-mode blocks of the software palette and nothing else
static bool takes_generic(const Handle *h) { return h->has_low_mode || h->palette == TX_PALETTE_HARDWARE; }

// What a tile's instance is asked for once per device: its shared memory, and how many clusters of 2 to 8 K ranges are resident at once.
struct TileSetup {
  bool ready = false;
  int clusters[9] = {-1, -1, -1, -1, -1, -1, -1, -1, -1};   // -1: not asked yet
};

template <int CTAS, int BN, typename Kernel>
static int resident_clusters(Kernel kernel, int ranges, int sm_count) {
  cudaLaunchConfig_t config{};
  cudaLaunchAttribute attribute{};
  config.gridDim = dim3(unsigned(sm_count / ranges), 1, unsigned(ranges));
  config.blockDim = dim3(TileConfig<CTAS, BN>::threads);
  config.dynamicSmemBytes = TileConfig<CTAS, BN>::smem;
  attribute.id = cudaLaunchAttributeClusterDimension;
  attribute.val.clusterDim.x = attribute.val.clusterDim.y = 1;
  attribute.val.clusterDim.z = unsigned(ranges);
  config.attrs = &attribute;
  config.numAttrs = 1;
  int found = 0;
  if (cudaOccupancyMaxActiveClusters(&found, kernel, &config) == cudaSuccess) return found;
  cudaGetLastError();
  return 0;
}

// One launch of the tile over `n` staged tokens (of `padded_tokens` in the buffer), and where K is cut the sum of its ranges: inside the launch, by clusters, where all of them are
// resident at once (a cluster waits for as many free SMs of one GPC as it has CTAs), else by a combine behind it.  By clusters / by a combine, us a
// call from HBM with 16, 64 and 128 tokens on the 64-token tile: 256x2048 6.3, 6.9, 7.3 / 7.7, 7.9, 8.9; 5120x5120 10.2, 12.6, 21.7 / 12.1, 14.0,
// 22.7; 5120x17408 19.8, 24.4, 42.5 / 22.7, 26.8, 46.5; 8192x28672 39.5, 44.5, 84.6 / 44.1, 48.4, 88.3.  No shape was slower.
template <int CTAS, int BN, int GROUPS>
static int launch_staged_groups(const Handle *h, const Workspace *ws, const __half *staged, int padded_tokens, const float *xmul, __nv_bfloat16 *y, int n, cudaStream_t stream, bool half_io) {
  using Cfg = TileConfig<CTAS, BN, GROUPS>;
  const bool generic = takes_generic(h);
  const auto kernel = generic ? prefill_umma_kernel<CTAS, BN, true, GROUPS> : prefill_umma_kernel<CTAS, BN, false, GROUPS>;
  const int ranges = prefill_k_ranges(h, n, ws);
  dim3 grid((h->M + Cfg::rows - 1) / Cfg::rows * CTAS, (n + BN - 1) / BN, ranges);
  bool merge = CTAS == 1 && GROUPS == 2 && ranges > 1;
  static std::mutex guard;
  static std::map<std::pair<int, bool>, TileSetup> configured;
  {
    std::lock_guard<std::mutex> lock(guard);
    TileSetup &setup = configured[{h->device, generic}];
    if (!setup.ready) {
      TX_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(Cfg::smem)));
      setup.ready = true;
    }
    if (merge) {
      int &clusters = setup.clusters[ranges];        // (at most 8 ranges)
      if (clusters < 0) clusters = resident_clusters<CTAS, BN>(kernel, ranges, ws->sm_count);
      merge = int(grid.x * grid.y) <= clusters;
    }
  }
  const int KP = h->KI * 128;
  // staged X viewed as [KP/8 chunks][padded_tokens/32][32 tokens x 8 elements]: a box is one run of
  // 512 contiguous bytes per 32 tokens and chunk and lands as core-matrix columns
  CUtensorMap map;
  cuuint64_t dims[3] = {256, cuuint64_t(padded_prompt(n) / 32), cuuint64_t(KP / 8)};
  cuuint64_t strides[2] = {512, cuuint64_t(padded_tokens) * 16};
  cuuint32_t box[3] = {256, cuuint32_t(Cfg::tokens / 32), cuuint32_t(kChunks)};
  cuuint32_t elem[3] = {1, 1, 1};
  CUresult cr = encode_tiled_entry()(&map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<__half *>(staged), dims, strides, box, elem,
                                     CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                                     CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (cr != CUDA_SUCCESS) return fail(TX_ECUDA, "cuTensorMapEncodeTiled failed with code " + std::to_string(int(cr)));
  PrefillParams p{};
  p.tiles = reinterpret_cast<const uint4 *>(h->tiles);
  p.flags = h->unit_flags;
  p.scales = h->scales;
  p.bias = h->bias;
  p.xmul = xmul;
  p.y = y;
  p.status = ws->status;
  p.M = h->M;
  p.K = h->K;
  p.KI = h->KI;
  p.MT = h->MT;
  p.T = n;
  p.palette = h->palette;
  p.half_io = half_io ? 1 : 0;
  p.partial = merge ? nullptr : ws->partial;
  TX_CUDA(launch_pdl_cluster(kernel, merge ? dim3(1, 1, ranges) : dim3(CTAS), grid, dim3(Cfg::threads), Cfg::smem, stream, p, map));
  count_launch();
  if (ranges > 1 && !merge) return launch_combine(ws->partial, ranges, h->bias, y, n, h->M, half_io, ws->sm_count, stream);
  return TX_OK;
}

template <int CTAS, int BN>
static int launch_staged_tile(const Handle *h, const Workspace *ws, const __half *staged, int padded_tokens, const float *xmul, __nv_bfloat16 *y, int n, cudaStream_t stream, bool half_io) {
  constexpr bool small = CTAS == 1 && BN <= 128;
  if (small && two_an_sm(long(h->M + kMmaM - 1) / kMmaM * ((n + BN - 1) / BN), prefill_k_ranges(h, n, ws), h->KI, ws->sm_count, takes_generic(h)))
    return launch_staged_groups<CTAS, BN, small ? 1 : 2>(h, ws, staged, padded_tokens, xmul, y, n, stream, half_io);
  return launch_staged_groups<CTAS, BN, 2>(h, ws, staged, padded_tokens, xmul, y, n, stream, half_io);
}

// A call goes in chunks of as many tokens as the per-device scratch holds in staged form, also where the activations come staged and need no scratch:
// the number of K ranges, and so the order of the sums, follows from a chunk's tokens.
static int chunk_tokens(const Handle *h, const Workspace *ws) {
  return int(std::min<size_t>(ws->xprep_halfs / (size_t(h->KI) * 128), 65536)) & ~31;   // staged tokens are padded to 32
}

template <int CTAS, int BN>
static int launch_tile(const Handle *h, const __nv_bfloat16 *x, __nv_bfloat16 *y, int tokens, cudaStream_t stream, bool half_io) {
  Workspace *ws = workspace_for(h->device);
  if (!ws) return TX_ECUDA;
  static std::mutex guard;
  static std::map<int, bool> configured;
  {
    std::lock_guard<std::mutex> lock(guard);
    if (!configured[h->device]) {
      TX_CUDA(cudaFuncSetAttribute(stage_activations_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kStageSmem)));
      configured[h->device] = true;
    }
  }
  // Activations are staged once as fp16 after an exact per-token power-of-two rescale (the decode GEMV's
  // arithmetic), in chunks of tokens that fit the per-device scratch.
  const int KP = h->KI * 128, capacity = chunk_tokens(h, ws);
  if (capacity < 32) return fail(TX_EINVAL, "K is too large for the prefill activation scratch");
  for (int t0 = 0; t0 < tokens; t0 += capacity) {
    const int n = std::min(capacity, tokens - t0);
    const int padded_tokens = padded_prompt(n);
    const int shares = h->K >= kSplitColumns && n <= ws->sm_count ? staging_shares(h->K, n, ws->sm_count) : 1;
    int per_cta = 4;
    while (per_cta > 1 && (padded_tokens / per_cta < ws->sm_count * 3 / 4 || per_cta * stage_row_bytes(h->K) > kStageSmem)) per_cta /= 2;
    const bool rows_fit = per_cta * stage_row_bytes(h->K) <= kStageSmem;
    if (shares > 1)
      TX_CUDA(launch_pdl_cluster(stage_split_kernel, shares, dim3(shares, n), dim3(kSplitThreads), 0, stream, x + size_t(t0) * h->K, ws->xprep, ws->xmul, h->K,
                                 padded_tokens, half_io ? 1 : 0));
    else
      TX_CUDA(launch_pdl(stage_activations_kernel, dim3(padded_tokens / per_cta), dim3(kStageThreads), rows_fit ? per_cta * stage_row_bytes(h->K) : 0,
                       stream, x + size_t(t0) * h->K, ws->xprep, ws->xmul, h->K, KP, n, padded_tokens, per_cta, rows_fit ? 1 : 0, half_io ? 1 : 0));
    count_launch();
    const int rc = launch_staged_tile<CTAS, BN>(h, ws, ws->xprep, padded_tokens, ws->xmul, y + size_t(t0) * h->M, n, stream, half_io);
    if (rc != TX_OK) return rc;
  }
  TX_CUDA(cudaGetLastError());
  return TX_OK;
}

// `half_io`: x, y and the handle's bias are fp16 (the reference multiplies fp16(pal*scale) with cuBLAS there,
// texelator_cuda.cu:996-1046; this kernel multiplies the exact numerators and scales in the epilogue)
int launch_prefill_tile(const Handle *h, int backend, const __nv_bfloat16 *x, __nv_bfloat16 *y, int tokens, cudaStream_t stream,
                        bool half_io) {
  switch (backend) {
    case 5: return launch_tile<1, 256>(h, x, y, tokens, stream, half_io);
    case 6: return launch_tile<2, 256>(h, x, y, tokens, stream, half_io);
    case 7: return launch_tile<1, 128>(h, x, y, tokens, stream, half_io);
    case 8: return launch_tile<1, 64>(h, x, y, tokens, stream, half_io);
    case 9: return launch_tile<1, 192>(h, x, y, tokens, stream, half_io);
    default: return fail(TX_EINVAL, "backend is not a tensor-core tile candidate");
  }
}

// The same for activations that the kernel in front wrote in staged form (bf16 in and out), in a buffer of the caller's.
int launch_prefill_staged(const Handle *h, int backend, const uint8_t *staged, __nv_bfloat16 *y, int tokens, cudaStream_t stream) {
  Workspace *ws = workspace_for(h->device);
  if (!ws) return TX_ECUDA;
  const int capacity = chunk_tokens(h, ws), padded = padded_prompt(tokens);
  if (capacity < 32) return fail(TX_EINVAL, "K is too large for the prefill activation scratch");
  for (int t0 = 0; t0 < tokens; t0 += capacity) {
    const int n = std::min(capacity, tokens - t0);
    const __half *x = reinterpret_cast<const __half *>(staged) + size_t(t0) * 8;   // (a chunk of eight columns is a run of tokens)
    const float *xmul = reinterpret_cast<const float *>(staged + staged_prompt_multipliers(h->K, tokens)) + t0;
    __nv_bfloat16 *out = y + size_t(t0) * h->M;
    int rc;
    switch (backend) {
      case 5: rc = launch_staged_tile<1, 256>(h, ws, x, padded, xmul, out, n, stream, false); break;
      case 6: rc = launch_staged_tile<2, 256>(h, ws, x, padded, xmul, out, n, stream, false); break;
      case 7: rc = launch_staged_tile<1, 128>(h, ws, x, padded, xmul, out, n, stream, false); break;
      case 8: rc = launch_staged_tile<1, 64>(h, ws, x, padded, xmul, out, n, stream, false); break;
      case 9: rc = launch_staged_tile<1, 192>(h, ws, x, padded, xmul, out, n, stream, false); break;
      default: return fail(TX_EINVAL, "backend is not a tensor-core tile candidate");
    }
    if (rc != TX_OK) return rc;
  }
  TX_CUDA(cudaGetLastError());
  return TX_OK;
}

template <int CTAS, int BN>
static int tile_info(int64_t out[9]) {
  using Cfg = TileConfig<CTAS, BN>;
  cudaFuncAttributes attributes{};
  TX_CUDA(cudaFuncGetAttributes(&attributes, prefill_umma_kernel<CTAS, BN, false, 2>));
  TX_CUDA(cudaFuncSetAttribute(prefill_umma_kernel<CTAS, BN, false, 2>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(Cfg::smem)));
  int active = 0;
  TX_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&active, prefill_umma_kernel<CTAS, BN, false, 2>, Cfg::threads, Cfg::smem));
  out[0] = attributes.numRegs;
  out[1] = int64_t(attributes.sharedSizeBytes);
  out[2] = int64_t(attributes.localSizeBytes);
  out[3] = attributes.maxThreadsPerBlock;
  out[4] = int64_t(Cfg::smem);
  out[5] = Cfg::rows;   // output rows per tile
  out[6] = BN;          // tokens per tile
  out[7] = kBK;         // columns per pipeline stage
  out[8] = active;
  return TX_OK;
}

int prefill_kernel_info(int backend, int64_t out[9]) {
  switch (backend) {
    case 5: return tile_info<1, 256>(out);
    case 6: return tile_info<2, 256>(out);
    case 7: return tile_info<1, 128>(out);
    case 8: return tile_info<1, 64>(out);
    case 9: return tile_info<1, 192>(out);
    default: return fail(TX_EINVAL, "backend is not a tensor-core tile candidate");
  }
}

}  // namespace tx
