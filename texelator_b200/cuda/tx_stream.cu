// Decode linear for up to sixteen tokens: one launch from the activations as they are to rounded outputs.
// (reference: texelator_bc4_kernel / texelator_bc4_bf16_kernel, texelator/cuda/texelator_cuda.cu:77-199)
//
// The walk over the payload is gemv_tile_kernel's (tx_gemv.cu): 128-bit loads of 1 KiB units, decode in registers,
// mma.sync with the tokens as MMA columns.  What differs is how a row is cut.  A row's units fall into eight or sixteen
// runs, by K and whether there is one token; a warp multiplies one run of one 16-row tile after another and
// always the same run, so
//
//   * a CTA of a cluster of C needs 1/C of the activations and stages them itself: one warp per (token, run), an exact
//     power-of-two rescale per run, no scan of the whole row, no launch in front, no scratch in global memory;
//   * warps meet once, at the end: every run's 16 x tokens sums go to the CTA of the cluster that finishes the tile
//     (distributed shared memory), one cluster barrier, then the runs are added in order and rounded once.  There is no
//     barrier per tile and no combine launch;
//   * the order of the sums does not depend on the rows of the matrix, the cluster size or the look-ahead, so row shards
//     reassemble bit for bit.
//
// What bounds it: instruction issue.  With the weights in L2 a call takes as long as with the weights in HBM; one token of
// 34816 x 5120 is 154 warp instructions a unit, all counted, on 3.7 warps a scheduler that issue in 58 % of the cycles.  What comes
// before the first unit (index arithmetic on kernel parameters alone, no division) and after the last one counts on small
// matrices.  us a call (a graph over copies larger than L2, look-ahead 3), the row walk with its pre-pass and combine
// launches / this kernel, for one, eight and fifteen bf16 tokens:
//
//   34816 x 5120   24.3 / 22.4   31.2 / 29.3   55.2 / 38.3        2048 x 11008   8.3 / 6.8   14.1 / 8.8   23.1 / 11.7
//   5120 x 17408   16.8 / 16.1   24.8 / 18.9   38.9 / 24.3        512 x 5120     3.5 / 3.6    9.2 / 4.8   15.4 / 6.0
//   22016 x 2048    9.2 / 8.1    13.3 / 12.6   23.0 / 17.1        256 x 2048     2.6 / 2.7    7.7 / 3.8   12.8 / 4.9
//   one fp16 token on the texture palette, 5120 x 17408: 30.7 / 20.5
//
// The only waits are CTA and cluster barriers.
#include <algorithm>
#include <map>
#include <mutex>
#include <tuple>

#include "tx_common.cuh"
#include "tx_decode.cuh"

namespace tx {

constexpr int kStreamThreads = 256;
constexpr int kStreamWarps = kStreamThreads / 32;
constexpr int kStreamTokens = 16;
constexpr int kHeldChunks = 4;              // 16-byte pieces of a run a lane keeps while it looks for the largest magnitude
constexpr int kStreamHalf = 1, kStreamSwiglu = 2, kStreamStrided = 4;   // flags in StreamParams::mode

struct StreamParams {
  const uint4 *tiles;
  const uint8_t *flags;
  const float *scales;
  const void *bias;
  const void *x;       // [T, K] bf16 or fp16
  void *y;             // [T, M], or [T, M / 2] behind SwiGLU
  int M, K, KI, T;
  int tile_begin, tile_count; // row tiles of this launch
  int clusters, tiles_each;   // cluster c takes tiles c, c + clusters, ...: tiles_each of them, one more below tile_count % clusters
  int chain_shift, cluster_shift;   // log2 of the runs of a row and of the CTAs of a cluster
  int mode;
};

__device__ __forceinline__ unsigned map_to_rank(unsigned addr, unsigned rank) {
  unsigned r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
// the lanes with `take` load 32 bytes; the others keep what they have (their MMA columns are never stored)
__device__ __forceinline__ void lds256_if(bool take, unsigned addr, uint4 &a, uint4 &b) {
  asm volatile(
      "{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %8, 0;\n\t"
      "@q ld.shared.v4.b32 {%0, %1, %2, %3}, [%9];\n\t"
      "@q ld.shared.v4.b32 {%4, %5, %6, %7}, [%9 + 16];\n\t}"
      : "+r"(a.x), "+r"(a.y), "+r"(a.z), "+r"(a.w), "+r"(b.x), "+r"(b.y), "+r"(b.z), "+r"(b.w) : "r"(unsigned(take)), "r"(addr));
}
__device__ __forceinline__ void store_shared(unsigned addr, float v) { asm volatile("st.shared.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory"); }
__device__ __forceinline__ void store_remote(unsigned addr, float v) {
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}

// The units of run c: first, first + step, ...  Runs are consecutive units, or (strided, one token) every eighth one.
struct Runs {
  int KI, shift;
  bool strided;
  __host__ __device__ __forceinline__ int first(int c) const { return strided ? c : (c * KI) >> shift; }
  __host__ __device__ __forceinline__ int length(int c) const {
    return strided ? (KI - c + (1 << shift) - 1) >> shift : ((c + 1) * KI >> shift) - (c * KI >> shift);
  }
  __host__ __device__ __forceinline__ int step() const { return strided ? 1 << shift : 1; }
  __host__ __device__ __forceinline__ int longest() const { return (KI + (1 << shift) - 1) >> shift; }
};
// place of a row in a token's sixteen sums: every other pair of tokens is turned by eight, so that the stores of a warp's
// fragments meet a bank twice and not four times
__device__ __forceinline__ int partial_row(int row, int tok) { return row ^ ((tok & 2) << 2); }

__host__ __device__ __forceinline__ int stream_head_bytes(int tokens, int chains) { return (tokens * chains * 4 + 127) & ~127; }
__host__ __device__ __forceinline__ int stream_part_bytes(int tiles_of_cluster, int cluster_shift, int tokens, int chains) {
  const int owned = (tiles_of_cluster + (1 << cluster_shift) - 1) >> cluster_shift;   // tiles a CTA finishes
  return (owned * chains * tokens * 64 + 127) & ~127;
}

// MODE: 0 software palette, 1 texture palette, + 2 where the payload has low-mode blocks.  (One instance for both palettes with such
// blocks chose at run time: 34816 x 5120, nine weights of ten zero, one token, 69.7 us, 61.2 with an instance each.)
template <int LOOKAHEAD, int NT, int MODE>
__global__ void __launch_bounds__(kStreamThreads, 2) cluster_gemv_tile_kernel(const StreamParams p) {
  extern __shared__ __align__(16) uint8_t smem_raw[];
  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int g = lane >> 2, t = lane & 3;
  const int KI = p.KI, T = p.T, NS = p.chain_shift, NC = 1 << NS;
  const int CS = p.cluster_shift, C = 1 << CS, rank = int(blockIdx.x) & (C - 1);   // clusters lie along x
  const int ns = NS - CS, n = 1 << ns;                     // runs of this CTA (up to eight)
  const int clusters = p.clusters, cluster = int(blockIdx.x) >> CS;
  const int tiles_here = p.tiles_each + (cluster < p.tile_count - p.tiles_each * clusters ? 1 : 0);
  const int chain = rank * n + (warp & (n - 1));
  const Runs runs{KI, NS, (p.mode & kStreamStrided) != 0};
  const int len = runs.length(chain), unit_step = runs.step(), run_bytes = runs.longest() * 256;
  const int tile_step = kStreamWarps >> ns, first_tile = warp >> ns;

  // shared memory: exponents [T][NC], partial tiles of the tiles finished here, activations
  int *exps_g = reinterpret_cast<int *>(smem_raw);
  const int head = stream_head_bytes(T, NC);
  float *part_g = reinterpret_cast<float *>(smem_raw + head);
  const int part_bytes = stream_part_bytes(p.tiles_each + (p.tile_count > p.tiles_each * clusters ? 1 : 0), CS, T, NC);
  uint8_t *xs_g = smem_raw + head + part_bytes;
  const unsigned sbase = unsigned(__cvta_generic_to_shared(smem_raw));
  const unsigned part_s = sbase + head, xs_s = part_s + part_bytes;
  const unsigned xs_stride = unsigned(n * run_bytes) + 16;   // + 16: tokens start on different banks

  // -- first weight loads, before anything else
  const int tiles_of_warp = first_tile < tiles_here ? (tiles_here - first_tile + tile_step - 1) >> (3 - ns) : 0;
  int left = tiles_of_warp * len, run_left = len;          // units still to fetch, of them in this run
  unsigned unext = (unsigned(p.tile_begin + cluster) + unsigned(first_tile) * unsigned(clusters)) * unsigned(KI) + unsigned(runs.first(chain));
  const unsigned wrap_step = unsigned(tile_step) * unsigned(clusters) * unsigned(KI) - unsigned(len - 1) * unsigned(unit_step);
  const uint4 *const base = p.tiles + lane;
  uint4 pend[LOOKAHEAD][2];
  unsigned pflag[LOOKAHEAD];
  auto prefetch = [&](int slot) {
    if (left > 0) {
      const uint4 *src = base + size_t(unext) * 64;
      pend[slot][0] = ldg_stream(src);
      pend[slot][1] = ldg_stream(src + 32);
      if (MODE >= 2) pflag[slot] = p.flags[unext];
    }
    --left;
    const bool wrap = --run_left == 0;
    unext += wrap ? wrap_step : unsigned(unit_step);
    run_left = wrap ? len : run_left;
  };
#pragma unroll
  for (int i = 0; i < LOOKAHEAD; ++i) prefetch(i);
  if (C > 1) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");   // waited for before the first remote store
  grid_launch_dependents();
  grid_dependency_wait();

  // -- activations: one warp per (token, run), fp16 after an exact power-of-two rescale of the run
  const int chunks_of_row = p.K / 8;
  const bool half_io = p.mode & kStreamHalf;
  for (int task = warp; task < T * n; task += kStreamWarps) {
    const int tok = task >> ns, c = rank * n + (task & (n - 1));
    const int count = runs.length(c) * 16, first = runs.first(c);
    const uint4 *src = static_cast<const uint4 *>(p.x) + size_t(tok) * chunks_of_row;
    uint4 *dst = reinterpret_cast<uint4 *>(xs_g + size_t(tok) * xs_stride + (c - rank * n) * run_bytes);
    const auto fetch = [&](int i) {                       // 16-byte piece i of the run
      const int at = (first + (i >> 4) * unit_step) * 16 + (i & 15);
      return i < count && at < chunks_of_row ? __ldcg(src + at) : make_uint4(0, 0, 0, 0);   // L2: another kernel wrote these moments ago
    };
    uint4 held[kHeldChunks];
    unsigned m = 0;
#pragma unroll
    for (int j = 0; j < kHeldChunks; ++j) held[j] = fetch(lane + j * 32);
    // what a lane does not keep waits in shared memory as it came: no trip to L2 for it a second time
#pragma unroll 1
    for (int i0 = kHeldChunks * 32; i0 < count; i0 += kHeldChunks * 32) {
      uint4 more[kHeldChunks];
#pragma unroll
      for (int j = 0; j < kHeldChunks; ++j) more[j] = fetch(i0 + lane + j * 32);
#pragma unroll
      for (int j = 0; j < kHeldChunks; ++j) {
        const int i = i0 + lane + j * 32;
        if (i < count) dst[i] = more[j];
        m = max(m, chunk_absmax(more[j]));
      }
    }
    int exponent = 0;
    float mult = 1.f;
    if (!half_io) {                                       // (fp16 activations are the operand as they are)
#pragma unroll
      for (int j = 0; j < kHeldChunks; ++j) m = max(m, chunk_absmax(held[j]));
      m = __reduce_max_sync(0xffffffffu, m);
      float inverse;
      token_scaling(m, mult, inverse);
      exponent = __float_as_int(inverse) >> 23;
      if (m == 0) exponent = 0;                           // a run of zeros: any scale fits, the smallest never sets the token's
    }
#pragma unroll
    for (int j = 0; j < kHeldChunks; ++j) {
      const int i = lane + j * 32;
      if (i < count) dst[i] = half_io ? held[j] : convert_chunk(held[j], mult);
    }
    if (!half_io)
#pragma unroll 1
      for (int i = lane + kHeldChunks * 32; i < count; i += 32) dst[i] = convert_chunk(dst[i], mult);
    if (lane == 0) exps_g[tok * NC + c] = exponent;
  }
  __syncthreads();
  if (C > 1) {
    asm volatile("barrier.cluster.wait.aligned;" ::: "memory");   // every CTA of the cluster runs
    // this CTA's exponents to the others
    for (int j = tid; j < T * NC; j += kStreamThreads) {
      const int peer = (j >> ns) & (C - 1), at = (j >> NS) * NC + rank * n + (j & (n - 1));
      if (peer != rank) store_remote(map_to_rank(sbase + unsigned(at) * 4, unsigned(peer)), __int_as_float(exps_g[at]));
    }
  }

  // -- this thread's first output: its constants are fetched while the weights stream
  const bool swiglu = p.mode & kStreamSwiglu;
  const int owned = tiles_here > rank ? (tiles_here - rank + C - 1) >> CS : 0;
  const int outputs = owned * T * 16;
  auto place = [&](int e, int &slot, int &tok, int &row) {   // output e: rows fastest, then tokens, then tiles
    const int r = e & 15, rest = e >> 4;
    slot = T == 1 ? rest : rest / T;
    tok = T == 1 ? 0 : rest - slot * T;
    row = (p.tile_begin + cluster + ((slot << CS) + rank) * clusters) * 16 + r;
  };
  auto bias_of = [&](int row) {
    if (!p.bias) return 0.f;
    return half_io ? __half2float(static_cast<const __half *>(p.bias)[row]) : __bfloat162float(static_cast<const __nv_bfloat16 *>(p.bias)[row]);
  };
  float scale0 = 0.f, bias0 = 0.f;
  if (tid < outputs) {
    int slot, tok, row;
    place(tid, slot, tok, row);
    if (row < p.M) {
      scale0 = p.scales[row];
      bias0 = bias_of(row);
    }
  }

  // -- the weight stream
  if (first_tile < tiles_here && len > 0) {
    unsigned xs_lane[NT];
    const bool live_token = g < T;
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
      const bool ok = nt * 8 + g < T;      // lanes whose token does not exist read another's: their MMA columns are never stored
      xs_lane[nt] = xs_s + (ok ? unsigned(nt * 8 + g) * xs_stride : 0u) + t * 32 + unsigned((chain - rank * n) * run_bytes);
    }
    float acc[NT][4], acc2[NT][4];         // two chains halve the MMA latency chain
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
      for (int q = 0; q < 4; ++q) acc[nt][q] = acc2[nt][q] = 0.f;
    uint4 bsolo[2] = {make_uint4(0, 0, 0, 0), make_uint4(0, 0, 0, 0)};
    int tile = first_tile, todo = len;
    unsigned xoff = 0;
    bool more = true;
    while (more) {
#pragma unroll
      for (int slot = 0; slot < LOOKAHEAD; ++slot) {
        const uint4 q = pend[slot][0], r = pend[slot][1];   // duos of rows g and g + 8
        const unsigned flag = pflag[slot];
        constexpr bool texture = MODE & 1;
        constexpr int palette = texture ? TX_PALETTE_HARDWARE : TX_PALETTE_SOFTWARE;
        const DuoConstants cq = duo_constants<texture>(q.w), cr = duo_constants<texture>(r.w);
#pragma unroll
        for (int sub = 0; sub < 2; ++sub) {
          unsigned aq[8], ar[8];
          if (sub == 0) { decode_duo_first<texture>(q, cq, aq); decode_duo_first<texture>(r, cr, ar); }
          else { decode_duo_second<texture>(q, cq, aq); decode_duo_second<texture>(r, cr, ar); }
          if (MODE >= 2 && __any_sync(0xffffffffu, flag != 0)) {   // warp-uniform: redo the low-mode blocks
            if (duo_block_is_low(q, sub)) decode_block_low(q, sub, aq, palette);
            if (duo_block_is_low(r, sub)) decode_block_low(r, sub, ar, palette);
          }
#pragma unroll
          for (int nt = 0; nt < NT; ++nt) {
            uint4 b0, b1;
            const unsigned xa = xs_lane[nt] + xoff + sub * 128;
            if (NT == 1) {
              lds256_if(live_token, xa, bsolo[0], bsolo[1]);   // one token: four lanes of the warp touch shared memory
              b0 = bsolo[0];
              b1 = bsolo[1];
            } else {
              b0 = lds128(xa);
              b1 = lds128(xa + 16);
            }
            mma_f16(acc[nt], aq[0], ar[0], aq[1], ar[1], b0.x, b0.y);
            mma_f16(acc2[nt], aq[2], ar[2], aq[3], ar[3], b0.z, b0.w);
            mma_f16(acc[nt], aq[4], ar[4], aq[5], ar[5], b1.x, b1.y);
            mma_f16(acc2[nt], aq[6], ar[6], aq[7], ar[7], b1.z, b1.w);
          }
        }
        prefetch(slot);
        xoff += 256;
        if (--todo == 0) {
          // ---- a run of a tile is done: its sums go to the CTA that finishes the tile
          const unsigned offset = unsigned(((((tile >> CS) << NS) + chain) * T * 16 + partial_row(g, 2 * t)) * 4);
          const unsigned dst = C == 1 ? part_s + offset : map_to_rank(part_s, unsigned(tile & (C - 1))) + offset;
#pragma unroll
          for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              const int tok = nt * 8 + 2 * t + e;
              if (tok < T) {
                const float low = acc[nt][e] + acc2[nt][e], high = acc[nt][e + 2] + acc2[nt][e + 2];
                const unsigned at = dst + unsigned(tok) * 64, other = at ^ 32;   // row g and row g + 8
                if (C == 1) {
                  store_shared(at, low);
                  store_shared(other, high);
                } else {
                  store_remote(at, low);
                  store_remote(other, high);
                }
              }
              acc[nt][e] = acc2[nt][e] = acc[nt][e + 2] = acc2[nt][e + 2] = 0.f;
            }
          tile += tile_step;
          todo = len;
          xoff = 0;
          if (tile >= tiles_here) {
            more = false;
            break;
          }
        }
      }
    }
  }
  __syncwarp();
  if (C > 1) asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  else __syncthreads();

  const int existing = min(NC, KI);                        // (a strided row shorter than eight units has fewer runs)
  // -- runs in order, one rounding.  Every run has its own power-of-two scale: bring them to the token's largest
  //    (exact unless a run is 2^126 below it, which fp16 would have lost at the token's scale as well).
  for (int e = tid; e < outputs; e += kStreamThreads) {
    int slot, tok, row;
    place(e, slot, tok, row);
    const bool first = e == tid;
    if (row >= p.M || (swiglu && (e & 8))) continue;
    const int *exps = exps_g + tok * NC;
    float multiplier = kNumeratorScale;
    int top = 1;
    if (!half_io) {
#pragma unroll 8
      for (int c = 0; c < existing; ++c) top = max(top, exps[c]);
      multiplier *= __int_as_float(top << 23);
    }
    auto total = [&](int r) {
      const float *src = part_g + (size_t(slot) * NC * T + tok) * 16 + partial_row(r, tok);
      float sum = 0.f;
#pragma unroll 8
      for (int c = 0; c < existing; ++c) {
        const int biased = half_io ? 127 : max(exps[c] - top + 127, 0);
        sum = fmaf(src[c * T * 16], __int_as_float(biased << 23), sum);
      }
      return sum;
    };
    const float row_scale = first ? scale0 : p.scales[row], row_bias = first ? bias0 : bias_of(row);
    const float value = fmaf(total(e & 15), row_scale * multiplier, row_bias);
    if (swiglu) {
      // gate rows 0-7 of a tile, up rows 8-15; both rounded first, like the outputs of an unfused linear, then
      // combined with silu_mul's arithmetic
      const float up_value = fmaf(total((e & 15) + 8), p.scales[row + 8] * multiplier, bias_of(row + 8));
      const float gate = __bfloat162float(__float2bfloat16(value)), up = __bfloat162float(__float2bfloat16(up_value));
      static_cast<__nv_bfloat16 *>(p.y)[size_t(tok) * (p.M / 2) + (row >> 4) * 8 + (row & 7)] = __float2bfloat16(gate / (1.f + __expf(-gate)) * up);
    } else if (half_io) {
      static_cast<__half *>(p.y)[size_t(tok) * p.M + row] = __float2half_rn(value);
    } else {
      static_cast<__nv_bfloat16 *>(p.y)[size_t(tok) * p.M + row] = __float2bfloat16(value);
    }
  }
}

// ------------------------------------------------------------------------------------------
// Host launcher
// ------------------------------------------------------------------------------------------
using StreamKernel = void (*)(const StreamParams);

template <int NT, int MODE>
static StreamKernel pick_lookahead(int lookahead) {
  // (one unit in flight on two CTAs an SM is too few: 5120 x 17408 with one token 22.3 us, 18.7 with two)
  switch (lookahead) {
    case 1: case 2: return cluster_gemv_tile_kernel<2, NT, MODE>;
    case 3: return cluster_gemv_tile_kernel<3, NT, MODE>;
    case 4: return cluster_gemv_tile_kernel<4, NT, MODE>;
    case 6: return cluster_gemv_tile_kernel<6, NT, MODE>;
    default: return cluster_gemv_tile_kernel<8, NT, MODE>;
  }
}
template <int NT>
static StreamKernel pick_mode(const Handle *h) {
  const bool texture = h->palette == TX_PALETTE_HARDWARE;
  if (h->has_low_mode) return texture ? pick_lookahead<NT, 3>(h->lookahead) : pick_lookahead<NT, 2>(h->lookahead);
  return texture ? pick_lookahead<NT, 1>(h->lookahead) : pick_lookahead<NT, 0>(h->lookahead);
}

constexpr int kStreamSmem[3] = {0, 200 * 1024, 112 * 1024};   // dynamic shared memory of a CTA that has an SM to itself, and of two

// Runs of a row, from K and from whether there is one bf16 token.  One: eight strided runs, the order in which rows were
// added up before this kernel, so a decoded token keeps its bits.  Otherwise: eight or sixteen runs of consecutive units,
// two to eight each in the usual range, few enough that a warp keeps one run.
static Runs stream_runs(int KI, int tokens, bool half_io) {
  if (tokens == 1 && !half_io) return Runs{KI, 3, true};
  return Runs{KI, KI >= 64 ? 4 : KI >= 8 ? 3 : KI >= 4 ? 2 : KI >= 2 ? 1 : 0, false};
}

struct StreamPlan {
  int cluster_shift, clusters, chain_shift;
  int smem;
  int slab;   // row tiles of a launch
};

// resident clusters of `cluster` CTAs, `per_sm` CTAs to an SM; looked up once per (device, kernel, cluster, per_sm)
static int resident_clusters(int device, StreamKernel kernel, int cluster, int per_sm, int sm_count) {
  static std::mutex guard;
  static std::map<std::tuple<int, const void *, int>, int> cache;
  const auto key = std::make_tuple(device, reinterpret_cast<const void *>(kernel), cluster * 4 + per_sm);
  std::lock_guard<std::mutex> lock(guard);
  const auto hit = cache.find(key);
  if (hit != cache.end()) return hit->second;
  int found = 0;
  if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kStreamSmem[1]) == cudaSuccess &&
      cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared) == cudaSuccess) {
    cudaLaunchConfig_t config{};
    config.gridDim = dim3(unsigned(sm_count * 2 / cluster * cluster));
    config.blockDim = dim3(kStreamThreads);
    config.dynamicSmemBytes = kStreamSmem[per_sm];
    cudaLaunchAttribute attribute{};
    attribute.id = cudaLaunchAttributeClusterDimension;
    attribute.val.clusterDim.x = unsigned(cluster);
    attribute.val.clusterDim.y = attribute.val.clusterDim.z = 1;
    config.attrs = &attribute;
    config.numAttrs = 1;
    if (cudaOccupancyMaxActiveClusters(&found, kernel, &config) != cudaSuccess) found = 0;   // (the error is read below)
  }
  if (cudaGetLastError() == cudaSuccess) cache[key] = found;   // (a failed query may succeed next time)
  return found;
}

// Cluster size and number of launches.  The estimate, in us: a warp takes 0.35 us a unit (0.55 beyond eight tokens, where it
// issues twice the MMAs) with sixteen warps on an SM and two thirds of that with eight, half of it counted by the warp with most
// units and half by the average; 0.35 us for each (token, run) a warp stages and the bytes staged by all CTAs at 8 TB/s, both
// smaller in a larger cluster; what a cluster costs at its barriers, in SMs that no whole cluster fits and, for four and
// eight, in an early start lost (launch_stream); 2.5 us a launch.  The constants are fitted to 34 shapes of 200 x 256 to
// 57344 x 8192 with 1, 2, 3, 5, 8, 12 and 15 tokens, each timed with clusters of 1, 2, 4 and 8 in a graph of 30 calls over three
// matrices: the pick is 0.4 % slower than the best of the four on average, 10 % at worst.  us a call, by cluster:
//
//   256 x 2048     one token 2.6, 2.7, 3.3, 3.5      eight tokens 7.0, 4.8, 4.2, 3.9
//   512 x 5120     one token 3.5, 3.4, 4.1, 4.2      eight tokens 8.4, 5.8, 5.2, 4.6
//   2048 x 11008   one token 7.9, 5.6, 6.5, 6.2      eight tokens (too large), 12.4, 9.5, 7.9
//   34816 x 5120   one token 21.1, 22.2, 23.9, 25.9  eight tokens 36.3, 27.6, 27.5, 28.7
//
// One bf16 token never takes clusters of more than two: its eight runs are fixed, so a warp's longest run stays as long while
// warps idle, and the early start is worth 0.5 us (512 x 5120 with four CTAs 4.1 us, 3.4 with two).
static bool plan_stream(const Handle *h, StreamKernel kernel, int tokens, bool half_io, int sm_count, StreamPlan &best) {
  const Runs runs = stream_runs(h->KI, tokens, half_io);
  const int NS = runs.shift, NC = 1 << NS;
  const double step = tokens <= 8 ? 0.35 : 0.55, cluster_cost[4] = {0.0, 0.35, 1.1, 1.1};
  double best_cost = 0;
  for (int slabs = 1; slabs <= h->MT; slabs *= 2) {
    const int tiles = (h->MT + slabs - 1) / slabs;
    for (int CS = 0; CS <= 3 && CS <= NS; ++CS) {
      const int C = 1 << CS, n = NC >> CS;
      if (n > kStreamWarps) continue;
      if (runs.strided && CS > 1 && best_cost != 0) break;
      const int units = n * runs.longest(), fixed = stream_head_bytes(tokens, NC) + tokens * (units * 256 + 16);
      for (int per_sm = 2; per_sm >= 1; --per_sm) {
        const int clusters = std::min(tiles, resident_clusters(h->device, kernel, C, per_sm, sm_count));
        if (clusters < 1) continue;
        const int per_cluster = (tiles + clusters - 1) / clusters;
        const int smem = fixed + stream_part_bytes(per_cluster, CS, tokens, NC);
        if (smem > kStreamSmem[per_sm]) continue;
        const double longest = double((per_cluster * n + kStreamWarps - 1) / kStreamWarps) * runs.longest();
        const double average = double(tiles) * h->KI / (double(clusters) * C * kStreamWarps);
        const double stream = (per_sm == 2 ? step : step * 0.67) * 0.5 * (longest + average);
        const double staging = 0.35 * ((tokens * n + kStreamWarps - 1) / kStreamWarps) + double(clusters) * C * tokens * units * 256 / 8e6;
        const double cost = slabs * (stream + staging + cluster_cost[CS] + 2.5);
        if (best_cost == 0 || cost < best_cost) {
          best_cost = cost;
          best = StreamPlan{CS, clusters, NS, smem, tiles};
        }
        break;
      }
    }
    if (best_cost != 0 && slabs >= 4) break;
  }
  return best_cost != 0;
}

// Tokens of one pass over the weights (0: the rows are too long for the kernel).  Rows that are too many for one launch's
// shared memory go in slabs of row tiles.
int stream_tokens(const Handle *h, int tokens, bool half_io) {
  if (h->KI > 1024) return 0;
  tokens = std::min(tokens, kStreamTokens);
  const Runs runs = stream_runs(h->KI, tokens, half_io);
  const int NC = 1 << runs.shift, C = NC < 8 ? NC : 8, n = NC / C;
  const auto smem = [&](int t) { return stream_head_bytes(t, NC) + t * (runs.longest() * n * 256 + 16) + 2 * NC * t * 64; };
  while (smem(tokens) > kStreamSmem[1]) --tokens;
  return tokens;
}

int launch_stream(const Handle *h, const void *x, void *y, int tokens, bool half_io, bool swiglu, cudaStream_t stream) {
  Workspace *ws = workspace_for(h->device);
  if (!ws) return TX_ECUDA;
  const StreamKernel kernel = tokens <= 8 ? pick_mode<1>(h) : pick_mode<2>(h);
  StreamParams p{};
  p.tiles = reinterpret_cast<const uint4 *>(h->tiles);
  p.flags = h->unit_flags;
  p.scales = h->scales;
  p.bias = h->bias;
  p.x = x;
  p.y = y;
  p.M = h->M;
  p.K = h->K;
  p.KI = h->KI;
  p.T = tokens;
  p.mode = (stream_runs(h->KI, tokens, half_io).strided ? kStreamStrided : 0) | (half_io ? kStreamHalf : 0) | (swiglu ? kStreamSwiglu : 0);
  StreamPlan plan{};
  if (!plan_stream(h, kernel, tokens, half_io, ws->sm_count, plan)) return fail(TX_EUNSUPPORTED, "no thread-block cluster of the decode kernel fits this device");
  p.chain_shift = plan.chain_shift;
  p.cluster_shift = plan.cluster_shift;
  for (int begin = 0; begin < h->MT; begin += plan.slab) {
    p.tile_begin = begin;
    p.tile_count = std::min(plan.slab, h->MT - begin);
    p.clusters = std::min(plan.clusters, p.tile_count);
    p.tiles_each = p.tile_count / p.clusters;
    // Clusters of four and eight start when the launch in front has ended: while its blocks (or those of the launch before)
    // still hold registers, the whole clusters that would fit an empty chip do not, and the rest waits for a second wave
    // (5120 x 17408 with 16 tokens inside a decode step 39 us, 24 alone).  Clusters of four behind a slab of the same call start
    // early: its clusters leave whole places (57344 x 8192 with eight tokens 72.8 us, 71.7 so).
    TX_CUDA(launch_cluster(kernel, plan.cluster_shift <= (begin > 0 ? 2 : 1), 1 << plan.cluster_shift,
                           dim3(unsigned(p.clusters << plan.cluster_shift)), dim3(kStreamThreads), size_t(plan.smem), stream, p));
    count_launch();
  }
  TX_CUDA(cudaGetLastError());
  return TX_OK;
}

int gemv_kernel_info(int64_t out[9]) {
  cudaFuncAttributes attributes{};
  const StreamKernel kernel = cluster_gemv_tile_kernel<2, 1, 0>;
  TX_CUDA(cudaFuncGetAttributes(&attributes, kernel));
  TX_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kStreamSmem[1]));
  int active = 0;
  const size_t smem = stream_head_bytes(1, 8) + stream_part_bytes(1, 0, 1, 8) + 4096 * 2 + 16;   // one token, K = 4096, one row tile
  TX_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&active, kernel, kStreamThreads, smem));
  out[0] = attributes.numRegs;
  out[1] = int64_t(attributes.sharedSizeBytes);
  out[2] = int64_t(attributes.localSizeBytes);
  out[3] = attributes.maxThreadsPerBlock;
  out[4] = int64_t(smem);
  out[5] = 16;   // rows per unit
  out[6] = 8;    // tokens per mma tile
  out[7] = 128;  // columns per unit
  out[8] = active;
  return TX_OK;
}

}  // namespace tx
