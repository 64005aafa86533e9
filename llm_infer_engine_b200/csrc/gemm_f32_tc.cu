// True float32 matrix product on the tensor cores: C[M, N] = A[M, K] * W[N, K]^T for large weights of the 32-bit path.
//
// A float32 number from 2^-110 on is the exact sum of three bfloat16 numbers, x = x1 + x2 + x3: x rounded, what is left rounded, the
// rest. (Below, the third part falls under bfloat16's least number, 2^-133; what is lost is 2^-134 at most: products of numbers around
// 2^-110 / 2^-112 / 2^-116 have an error of 1.2e-7 / 1.9e-7 / 2.2e-6, where FMAs keep 2.1e-7.) A product of two bfloat16 numbers is
// exact in float32. Of the nine products of parts the six with a weight of 2^-16 or more are formed; the three left
// out are below 2^-25 of the product (parts that were cut off instead of rounded would leave out 3e-8 of one sign). w1 x1 has a
// sum of its own, G1; the other five share G2, which is 2^-8 of it, so that only G1 is subject to the accumulator's rounding.
//
// The accumulator cuts off what does not fit, towards zero. So it keeps 64 k at a time, then G1 + G2 joins a float32 sum in
// registers; and slices go in pairs: the products of the second one are SUBTRACTED from where the first one ended. With sums of
// one sign the accumulator goes up and comes back through the same range, and loses as much on the way back as on the way up: with
// v1 after the first slice and v2 after the second one, 2 v1 - v2 is free of it. Relative error against 64-bit sums (2-norm, 1e-7;
// without pairs, 128 k a slice; in brackets the packed FMAs of gemm_simt.cu), K of 1,024 / 2,048 / 8,192: normal numbers 1.1 / 1.2
// / 1.5 (1.3 / 1.3 / 1.5) (1.6 / 2.1 / 4.1), their magnitudes 0.55 / 0.56 / 0.66 (1.73 / 1.72 / 1.74, all of it bias) (0.60 / 0.67 /
// 1.01), 1 +- 0.01 0.45 / 0.47 / 0.57 (0.40 / 0.42 / 0.48) (0.55 / 0.61 / 0.88), equal numbers 0.25 / 0.25 / 1.2 (4.8 / 9.6 / 38).
// Uniform numbers that rise along K have 0.57 / 0.57 / 0.71 (0.54 / 0.59 / 0.74): the one kind seen above the FMAs, by 5 % with 1,024.
//
// One summation order for every shape. K is cut into slices of 128; n slices make four chains, chain j the slices
// [j n / 4, (j + 1) n / 4), in pairs from its first on (the last of an odd number has no partner); a chain's sum P_j adds the
// halves of its slices in order, and the result is (P_0 + P_1) + (P_2 + P_3). A row's result does not depend on which other rows
// share the launch, on the tile or on how the chains are shared among blocks.
//
// Sums that are not finite (an infinity or NaN among the inputs, whose parts are NaN, or an overflow, of a part too) are formed again by plain
// FMAs over K, a warp a sum, which give what IEEE arithmetic gives.
//
// A block makes 128 weight rows x NT tokens. The weights are the 128-row operand, in tensor memory; per 16 k five tcgen05.mma: w1
// by [x1 x2] into [G1 G2], then w1 x3, w2 x1, w2 x2, w3 x1 into G2. Sixteen warps in four groups, a group a stage of 32 k, read
// the weights as float32, a lane its row, a round of the groups ahead, split them and store the parts; the tokens' parts were
// made by a kernel in front and come by TMA, eight stages deep (NT = 16: the same warps split them); one lane issues the
// products, two stages a turn behind one barrier; eight warps empty one of two accumulators while the other fills, and keep the
// sums of finished chains in shared memory.
//
// What bounds it: the issue of the products, about 80 cycles each with 80 tokens, 56 with 16, of which the tensor cores work 48
// (80 tokens), and the weights' way through L1, a lane its row (301 x 16,384: tensor pipe 48 % of the active cycles, L1 80 %). With the
// weights' parts in shared memory it was its bandwidth. Products of 2,048 k (128 k a slice, no pairs; FMA): 301 x 16,384 158 us (151;
// 500), 301 x 2,048 x 8,192 k 75 (75; 279).
#include "tcgen05.cuh"

namespace llmie {
namespace {
using namespace tc;

constexpr int kMt = 128;                  // weight rows of a block
constexpr int kStageK = 32;              // 64 bytes of a part's row, 64-byte swizzle
constexpr int kPerSlice = 128 / kStageK;  // stages of a slice
constexpr int kSliceK = 128;
constexpr int kChains = 4;
constexpr uint32_t kNegateA = 1u << 13;   // of an instruction descriptor: the products' signs
constexpr int kSumWarps = 8, kSplitWarps = 16;
constexpr int kStages = 4;                // four warps split for each
static_assert(kSplitWarps == 4 * kStages && kStages == kPerSlice, "the stages of a slice go round four groups of warps");
constexpr int kTcThreads = 32 * (kSumWarps + kSplitWarps + 4);        // the last four: one issues products, one copies

template <int NT>
struct Shape {
  static constexpr bool kSplitsX = NT == 16;                 // else the tokens' parts come by TMA
  static constexpr int kXPart = NT * 64, kXStage = 3 * kXPart;        // bytes of one part of a stage, of all
  static constexpr int kXTurns = kSplitsX ? 2 : 4;           // two stages each: copies run further ahead, they take a turn's time
  static constexpr int kSmem = kXTurns * 2 * kXStage + 2 * NT * kMt * 4 + 1024;
  static constexpr int kAccCols = 2 * NT, kWCol = 2 * kAccCols;       // tensor memory: two accumulators, then the weights' parts
  static constexpr int kWStageCols = 3 * kStageK / 2, kTmemCols = NT == 16 ? 256 : 512;
  static_assert(kWCol + kStages * kWStageCols <= kTmemCols, "");
  static constexpr int kCols = NT / 2;                       // of a sum warp
};

// Byte offset of piece `piece` (16 bytes) of row `row` in 64-byte rows with the 64-byte swizzle, and its operand descriptor.
__device__ __forceinline__ uint32_t swizzle64_offset(int row, int piece) {
  return (uint32_t)row * 64u + (uint32_t)((piece ^ ((row >> 1) & 3)) << 4);
}
__device__ __forceinline__ uint64_t operand_desc(uint32_t smem_addr) {
  return (uint64_t)((smem_addr >> 4) & 0x3FFF) | (uint64_t)1 << 16 | (uint64_t)(512 >> 4) << 32 | (uint64_t)1 << 46 |
         (uint64_t)4 << 61;
}

struct TcShared {
  uint64_t ready[4], empty[kStages], x_empty[4], acc_full[2], drained;       // ready: all that a turn of two stages needs
  uint32_t tmem;
  int abort, copied;                        // copied: turns whose tokens' parts have been asked for
};

// 8 neighbouring floats; WIDE: from a 32-byte aligned address. No condition around it, and the registers are named as read too:
// a value that is merged with another, or moved, waits for its load.
template <bool WIDE>
__device__ __forceinline__ void load_8(const float* p, float (&v)[8]) {
  if (WIDE) {
    asm volatile("ld.global.L1::no_allocate.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "+f"(v[0]), "+f"(v[1]), "+f"(v[2]), "+f"(v[3]), "+f"(v[4]), "+f"(v[5]), "+f"(v[6]), "+f"(v[7]) : "l"(p));
  } else {
#pragma unroll
    for (int e = 0; e < 8; ++e) asm volatile("ld.global.f32 %0, [%1];" : "+f"(v[e]) : "l"(p + e));
  }
}

__device__ __forceinline__ unsigned pack_rn(float a, float b) {
  unsigned v;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(v) : "f"(b), "f"(a));
  return v;
}
// The three parts of 8 floats, 16 bytes each.
__device__ __forceinline__ void split_8(const float (&v)[8], uint4 (&parts)[3]) {
  unsigned h[3][4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float a = v[2 * i], b = v[2 * i + 1];
#pragma unroll
    for (int part = 0; part < 3; ++part) {
      h[part][i] = pack_rn(a, b);
      if (part < 2) {
        a -= __uint_as_float(h[part][i] << 16);
        b -= __uint_as_float(h[part][i] & 0xffff0000u);
      }
    }
  }
#pragma unroll
  for (int part = 0; part < 3; ++part) parts[part] = make_uint4(h[part][0], h[part][1], h[part][2], h[part][3]);
}
__device__ __forceinline__ void split_store(const float (&v)[8], unsigned char* dst, int part_bytes) {
  uint4 parts[3];
  split_8(v, parts);
#pragma unroll
  for (int part = 0; part < 3; ++part) *reinterpret_cast<uint4*>(dst + part * part_bytes) = parts[part];
}

// parts[p][t][k]: part p of A[t][k], K a multiple of 8.
template <bool WIDE>
__global__ void __launch_bounds__(256) split_rows_kernel(const float* A, __nv_bfloat16* __restrict__ out, int M, int K, int lda) {
  pdl_launch_dependents();
  pdl_wait();
  const int per_row = K >> 3;
  const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
  if (i >= (long long)M * per_row) return;
  const int t = (int)(i / per_row), k = (int)(i - (long long)t * per_row) << 3;
  float v[8] = {};
  uint4 parts[3];
  load_8<WIDE>(A + (size_t)t * lda + k, v);
  split_8(v, parts);
#pragma unroll
  for (int p = 0; p < 3; ++p) *reinterpret_cast<uint4*>(out + ((size_t)p * M + t) * K + k) = parts[p];
}

__device__ __forceinline__ bool is_finite(float v) { return fabsf(v) <= 3.402823466e38f; }

template <bool VEC>
__device__ __forceinline__ float4 load_4(const float* p) {
  return VEC ? *reinterpret_cast<const float4*>(p) : make_float4(p[0], p[1], p[2], p[3]);
}
__device__ __forceinline__ float dot_4(const float4& x, const float4& w, float s) {
  return fmaf(x.w, w.w, fmaf(x.z, w.z, fmaf(x.y, w.y, fmaf(x.x, w.x, s))));
}

// Sums that are not finite are formed again by FMAs: a warp a sum, lane l the k of 4 l to 4 l + 3 of every 128, in turn; then the lanes'
// sums in pairs. R weight rows at a time.
template <int R, bool VEC>
__device__ __forceinline__ void warp_dots(const float* x, const float* const (&w)[R], int K, float (&s)[R]) {
#pragma unroll
  for (int r = 0; r < R; ++r) s[r] = 0.f;
#pragma unroll 2
  for (int k = 4 * (threadIdx.x & 31); k < K; k += 128) {
    const float4 a = load_4<VEC>(x + k);
#pragma unroll
    for (int r = 0; r < R; ++r) s[r] = dot_4(a, load_4<VEC>(w[r] + k), s[r]);
  }
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int o = 16; o; o >>= 1) s[r] += __shfl_xor_sync(0xffffffffu, s[r], o);
}
// Those of the n results out[i * out_step] of rows x + i * x_step and this lane's weight row (w of lane 0) that are not finite; whole warps.
template <int R, bool VEC>
__device__ __forceinline__ void plain_sums(const float* x, size_t x_step, const float* w, int ldw, float* out, size_t out_step, int n,
                                           bool there, int K) {
  const int lane = threadIdx.x & 31;
#pragma unroll 1
  for (int i = 0; i < n; ++i, x += x_step, out += out_step) {
    unsigned again = __ballot_sync(0xffffffffu, there && !is_finite(*out));
    if (!again) continue;
    bool nan = false;                     // then so are all results of this row, and they are already
#pragma unroll 2
    for (int k = 4 * lane; k < K; k += 128) {
      const float4 v = load_4<VEC>(x + k);
      nan = nan || v.x != v.x || v.y != v.y || v.z != v.z || v.w != v.w;
    }
    if (__any_sync(0xffffffffu, nan)) continue;
#pragma unroll 1
    while (again) {
      const float* rows[R];
      float s[R];
      int at[R];
#pragma unroll
      for (int r = 0; r < R; ++r) {
        at[r] = again ? __ffs(again) - 1 : at[0];
        again &= again - 1;
        rows[r] = w + (size_t)at[r] * ldw;
      }
      warp_dots<R, VEC>(x, rows, K, s);
#pragma unroll
      for (int r = 0; r < R; ++r)
        if (lane == at[r]) *out = s[r];
    }
  }
}

// N consecutive columns of 32 lanes, N a multiple of 8; tmem_ld_wait() before they are used.
__device__ __forceinline__ void tmem_ld_32x8(uint32_t taddr, uint32_t* r) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr));
}
// run (+)= times (G1 + G2), 16 columns at a time.
template <int C0, int N>
__device__ __forceinline__ void sum_columns(uint32_t g1, int to_g2, float (&run)[N], bool fresh, float times) {
  constexpr int n = N - C0 < 16 ? N - C0 : 16;
  uint32_t a[n], b[n];
#pragma unroll
  for (int c = 0; c < n; c += 8) tmem_ld_32x8(g1 + C0 + c, a + c);
#pragma unroll
  for (int c = 0; c < n; c += 8) tmem_ld_32x8(g1 + to_g2 + C0 + c, b + c);
  tmem_ld_wait();
#pragma unroll
  for (int c = 0; c < n; ++c) {
    const float v = __uint_as_float(a[c]) + __uint_as_float(b[c]);
    run[C0 + c] = fmaf(times, v, fresh ? 0.f : run[C0 + c]);
  }
  if constexpr (C0 + n < N) sum_columns<C0 + n, N>(g1, to_g2, run, fresh, times);
}

__device__ __forceinline__ void tmem_st_32x4(uint32_t taddr, const uint4& v) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};" ::"r"(taddr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w)
               : "memory");
}
// D[tmem] (+)= A[tmem] * B[smem]; one thread issues.
__device__ __forceinline__ void mma_bf16_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}

// LIMIT: polls before a wait gives up, a constant as in attention_latent_tc.cu.
template <int NT, bool WIDE, unsigned LIMIT>
__global__ void __launch_bounds__(kTcThreads, 1)
gemm_f32_tc_kernel(const __grid_constant__ CUtensorMap map_x, const float* A, const float* W, float* C, int M, int N, int K, int lda,
                   int ldw, int ldc, int split, int w_written, int* __restrict__ status) {
  using S = Shape<NT>;
  extern __shared__ __align__(1024) unsigned char tc_smem[];
  __shared__ TcShared sh;
  unsigned char* x_stages = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(tc_smem) + 1023) & ~(uintptr_t)1023);
  float* hold = reinterpret_cast<float*>(x_stages + S::kXTurns * 2 * S::kXStage);        // [2][NT][kMt]: sums of finished chains
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int rank = blockIdx.x % split;
  const int tiles_m = (M + NT - 1) / NT, tile = blockIdx.x / split;
  const int m0 = (tile % tiles_m) * NT, n0 = (tile / tiles_m) * kMt;
  const int slices = K / kSliceK;
  const int chain0 = rank * (kChains / split);
  const int slice0 = chain0 * slices / kChains, slice1 = (chain0 + kChains / split) * slices / kChains;
  const int n_stages = kPerSlice * (slice1 - slice0), n_turns = n_stages / 2;
  volatile int* abort = &sh.abort;

  if (tid == 0) {
    for (int i = 0; i < 4; ++i) {         // eight splitting warps, the tokens' copy, the sum warps
      mbar_init(&sh.ready[i], 8 + (S::kSplitsX ? 0 : 1) + kSumWarps);
      mbar_init(&sh.empty[i], 1);
      mbar_init(&sh.x_empty[i], 1);
    }
    for (int i = 0; i < 2; ++i) mbar_init(&sh.acc_full[i], 1);
    mbar_init(&sh.drained, 1);
    sh.abort = sh.copied = 0;
    fence_mbar_init();
  }
  if (warp == kSumWarps + kSplitWarps) {
    tmem_alloc(&sh.tmem, S::kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = sh.tmem;

  if (warp < kSumWarps) {
    // ---------------------------------------------------------------- sums: half of the tokens each four warps
    if (S::kSplitsX) asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
    else asm volatile("setmaxnreg.inc.sync.aligned.u32 104;");
    pdl_wait();
    const int quarter = warp & 3, col0 = (warp >> 2) * S::kCols, row = quarter * 32 + lane;
    const uint32_t acc = tmem + ((uint32_t)(quarter * 32) << 16) + col0;
    const bool row_there = n0 + row < N;
    float* h = hold + (size_t)col0 * kMt + row;
    float* out = C + (size_t)(m0 + col0) * ldc + n0 + row;
    const int n_cols = min(S::kCols, M - m0 - col0);       // of the result
    float run[S::kCols] = {};
    int chain = 0, chain_end = (chain0 + 1) * slices / kChains;
    bool fresh = true, second = false, ok = true;
    if (lane < 2) mbar_arrive(&sh.ready[lane]);           // both accumulators are free
#pragma unroll 1
    for (int turn = 0; turn < n_turns; ++turn) {
      const int ab = turn & 1, slice = slice0 + (turn >> 1);
      ok = __all_sync(0xffffffffu, mbar_wait(&sh.acc_full[ab], (turn >> 1) & 1, abort, LIMIT));
      if (!ok) {
        if (!*abort) { *abort = 1; atomicExch(status, kStatusTimeoutMma); }
        break;
      }
      tc_fence_after_sync();
      sum_columns<0, S::kCols>(acc + ab * S::kAccCols, NT, run, fresh, second ? -1.f : slice + 1 < chain_end ? 2.f : 1.f);
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&sh.ready[(turn + 2) & 3]);
      fresh = ab && slice + 1 == chain_end;
      second = second != (ab != 0) && !fresh;
      if (fresh) {                        // the chain is done: ((P_0 + P_1) + (P_2 + P_3)) as far as this block has them
        if (chain & 1) {
          const float* from = h + (chain == 3 ? NT * kMt : 0);
#pragma unroll
          for (int c = 0; c < S::kCols; ++c) run[c] = from[c * kMt] + run[c];
        }
        if (chain == 3) {
#pragma unroll
          for (int c = 0; c < S::kCols; ++c) run[c] = h[c * kMt] + run[c];
        }
        if (chain < kChains / split - 1 || split > 1) {       // (the last one of a cluster's block: for the others to read)
          float* to = h + (chain == 2 ? NT * kMt : 0);
#pragma unroll
          for (int c = 0; c < S::kCols; ++c) to[c * kMt] = run[c];
        }
        ++chain;
        chain_end = (chain0 + chain + 1) * slices / kChains;
      }
    }
    if (!ok) {                            // (the plain sums below then replace these)
#pragma unroll
      for (int c = 0; c < S::kCols; ++c) h[c * kMt] = run[c] = __int_as_float(0x7fc00000);
    }
    if (split == 1) {
      bool finite = true;
#pragma unroll
      for (int c = 0; c < S::kCols; ++c) {
        if (row_there && c < n_cols) {
          out[(size_t)c * ldc] = run[c];
          finite = finite && is_finite(run[c]);
        }
      }
      if (!__all_sync(0xffffffffu, finite))
        plain_sums<NT == 16 ? 1 : 4, WIDE>(A + (size_t)(m0 + col0) * lda, lda, W + (size_t)(n0 + quarter * 32) * ldw, ldw, out, ldc, n_cols, row_there, K);
    } else {                              // each block of the cluster finishes its share of the tokens
      cluster_sync_all();
      const int first = rank * 2 + (warp >> 2), step = 2 * split;
      float* out = C + (size_t)(m0 + first) * ldc + n0 + row;
      bool finite = true;
      const int n = (min(NT, M - m0) - first + step - 1) / step;
      for (int i = 0; row_there && i < n; ++i) {
        const uint32_t a = smem_u32(hold + (size_t)(first + i * step) * kMt + row);
        float v;
        if (split == 2)
          v = ld_cluster_f32(map_to_block(a, 0)) + ld_cluster_f32(map_to_block(a, 1));
        else
          v = (ld_cluster_f32(map_to_block(a, 0)) + ld_cluster_f32(map_to_block(a, 1))) +
              (ld_cluster_f32(map_to_block(a, 2)) + ld_cluster_f32(map_to_block(a, 3)));
        out[(size_t)i * step * ldc] = v;
        finite = finite && is_finite(v);
      }
      if (!__all_sync(0xffffffffu, finite))
        plain_sums<1, WIDE>(A + (size_t)(m0 + first) * lda, (size_t)step * lda, W + (size_t)(n0 + quarter * 32) * ldw, ldw, out,
                         (size_t)step * ldc, n, row_there, K);
      cluster_sync_all();                 // nobody leaves while its sums are read
    }
  } else if (warp < kSumWarps + kSplitWarps) {
    // ---------------------------------------------------------------- float32 in, parts out
    if (S::kSplitsX) asm volatile("setmaxnreg.inc.sync.aligned.u32 88;");
    else asm volatile("setmaxnreg.dec.sync.aligned.u32 64;");
    // a thread a weight row (a lane of the tensor memory) and 32 k of a stage
    const int group = (warp - kSumWarps) >> 2, quarter = warp & 3;
    const uint32_t to = tmem + ((uint32_t)(quarter * 32) << 16) + S::kWCol + group * S::kWStageCols;
    // the row behind the last is the last one again, the stage behind the last one too: nobody reads what becomes of them
    const float* w_src = W + (size_t)min(n0 + quarter * 32 + lane, N - 1) * ldw + slice0 * kSliceK;
    float w[4][8] = {}, x[8] = {};
    if (w_written) pdl_wait();
#pragma unroll
    for (int i = 0; i < 4; ++i) load_8<WIDE>(w_src + group * kStageK + 8 * i, w[i]);
    // (up to 16 tokens: 64 threads of the group a piece of 8)
    const int gt = tid & 127, r = gt >> 2;
    const float* a_src = A + (size_t)min(m0 + r, M - 1) * lda + slice0 * kSliceK + (gt & 3) * 8;
    unsigned char* x_to = x_stages + group * S::kXStage + swizzle64_offset(r, gt & 3);
    if (S::kSplitsX) {
      pdl_wait();
      load_8<WIDE>(a_src + group * kStageK, x);
    }
    uint64_t* empty = &sh.empty[group];
    uint32_t parity = 1;                    // a fresh barrier counts as released
    for (int s = group; s < n_stages; s += kStages, parity ^= 1) {
      const bool ok = __all_sync(0xffffffffu, mbar_wait(empty, parity, abort, LIMIT));
      if (!ok) {
        if (!*abort) { *abort = 1; atomicExch(status, kStatusTimeoutEmpty); }
        break;
      }
      tc_fence_after_sync();
      const int next = min(s + kStages, n_stages - 1) * kStageK;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        uint4 parts[3];
        split_8(w[i], parts);
        load_8<WIDE>(w_src + next + 8 * i, w[i]);
#pragma unroll
        for (int p = 0; p < 3; ++p) tmem_st_32x4(to + p * (kStageK / 2) + 4 * i, parts[p]);
      }
      if (S::kSplitsX) {
        if (r < NT) split_store(x, x_to, S::kXPart);
        load_8<WIDE>(a_src + next, x);
      }
      tmem_st_wait();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&sh.ready[(s >> 1) & 3]);
    }
  } else {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
    if (warp == kSumWarps + kSplitWarps) {
      // -------------------------------------------------------------- products
      // The whole warp walks the stages, so that addresses and descriptors are the warp's and not a thread's; one lane issues.
      constexpr uint32_t d2 = make_instr_desc_bf16(kMt, 2 * NT, 0, 0), d1 = make_instr_desc_bf16(kMt, NT, 0, 0);
      const bool leader = elect_one();
      const uint64_t first_x = operand_desc(smem_u32(x_stages));
      constexpr uint64_t kXNext = S::kXPart / 16;
      constexpr uint32_t kWNext = kStageK / 2;
      int chain = chain0, chain_end = (chain0 + 1) * slices / kChains;
      uint32_t second = 0;                             // a pair's second slice: its products are subtracted from the first one's sums
      bool ok = mbar_wait(&sh.ready[0], 0, abort, LIMIT);
      for (int turn = 0; ok && turn < n_turns; ++turn) {
        const int ws = turn & 1, xs = S::kSplitsX ? ws : turn & 3;
        const uint32_t g1 = tmem + ws * S::kAccCols, g2 = g1 + NT, minus = second * kNegateA;
        if (S::kSplitsX) fence_proxy_async_smem();     // these parts were written through the generic proxy
        tc_fence_after_sync();
        auto products = [&](int e, int kk) {           // 32 bytes of a token's row: 2 in a descriptor's units; 8 columns
          const uint32_t w1 = tmem + S::kWCol + (2 * ws + e) * S::kWStageCols + 8 * kk, w2 = w1 + kWNext, w3 = w2 + kWNext;
          const uint64_t x1 = first_x + (2 * xs + e) * (S::kXStage / 16) + 2 * kk, x2 = x1 + kXNext, x3 = x2 + kXNext;
          mma_bf16_ts(g1, w1, x1, d2 | minus, e > 0 || kk > 0 ? 1u : second);
          mma_bf16_ts(g2, w1, x3, d1 | minus, 1u);
          mma_bf16_ts(g2, w2, x1, d1 | minus, 1u);
          mma_bf16_ts(g2, w2, x2, d1 | minus, 1u);
          mma_bf16_ts(g2, w3, x1, d1 | minus, 1u);
        };
        if (leader) {
          products(0, 0);
          products(0, 1);
          mma_commit(&sh.empty[2 * ws]);
          products(1, 0);
        }
        __syncwarp();
        // the wait for the next turn stands in front of this one's last products: they are worked on meanwhile
        if (turn + 1 < n_turns) ok = mbar_wait(&sh.ready[(turn + 1) & 3], ((turn + 1) >> 2) & 1, abort, LIMIT);
        if (leader) {
          products(1, 1);
          mma_commit(&sh.empty[2 * ws + 1]);
          if (!S::kSplitsX) mma_commit(&sh.x_empty[xs]);
          mma_commit(&sh.acc_full[ws]);
        }
        __syncwarp();
        if (ws) {
          second ^= 1;
          if (slice0 + (turn >> 1) + 1 == chain_end) {
            second = 0;
            chain_end = (++chain + 1) * slices / kChains;
          }
        }
      }
      if (!ok && leader && !*abort) { *abort = 1; atomicExch(status, kStatusTimeoutFull); }
      __syncwarp();
    } else if (warp == kSumWarps + kSplitWarps + 1 && !S::kSplitsX) {
      // -------------------------------------------------------------- the tokens' parts
      if (elect_one()) {
        tma_prefetch_desc(&map_x);
        pdl_wait();
        int turn = 0;
        for (; turn < n_turns; ++turn) {
          const int xs = turn & 3;
          if (!mbar_wait(&sh.x_empty[xs], ((turn >> 2) & 1) ^ 1, abort, LIMIT)) {
            if (!*abort) { *abort = 1; atomicExch(status, kStatusTimeoutEmpty); }
            break;
          }
          mbar_arrive_expect_tx(&sh.ready[xs], 2 * S::kXStage);
#pragma unroll
          for (int e = 0; e < 2; ++e)
#pragma unroll
            for (int p = 0; p < 3; ++p)
              tma_load_2d(x_stages + (2 * xs + e) * S::kXStage + p * S::kXPart, &map_x,
                          slice0 * kSliceK + (2 * turn + e) * kStageK, p * M + m0, &sh.ready[xs]);
        }
        sh.copied = turn;
      }
      __syncwarp();
    }
  }
  if (split > 1 && warp >= kSumWarps) {
    cluster_sync_all();
    cluster_sync_all();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  if (*abort) {
    // whichever role gave up: copies and products still in flight end, or have had the time to, before the block gives its memory up
    // (a turn's barrier is also short of the splitting warps that gave up: its copies then have the whole of the wait)
    if (tid == 0) {
      for (int turn = max(0, sh.copied - 4); turn < sh.copied; ++turn)
        for (unsigned spin = 0; spin < (1u << 14) && !mbar_test(&sh.ready[turn & 3], (turn >> 2) & 1); ++spin) __nanosleep(64);
    }
    if (warp == kSumWarps + kSplitWarps && elect_one()) {       // the lane that issued the products
      mma_commit(&sh.drained);
      for (unsigned spin = 0; spin < (1u << 16) && !mbar_test(&sh.drained, 0); ++spin) __nanosleep(64);
    }
    __syncthreads();
  }
  if (warp == kSumWarps + kSplitWarps) tmem_dealloc(tmem, S::kTmemCols);
}

// ------------------------------------------------------------------------------------------ up to 16 tokens
// What bounds it: large weights, their way from memory; small ones, the chain of products on one another (40 of a turn share G2) behind the
// loads. Microseconds one after another, weights from memory, FMA from shared memory (gemm_simt.cu) / this, 1, 4, 8 and 16 tokens:
//
//   128 x 1,024 k     2.5 / 2.9    3.3 / 2.9    4.9 / 3.8    8.3 / 4.8       2,048 x 8,192 k    16.4 / 18.0    23.5 / 18.8    36 / 20    50 / 26
//   512 x 2,048 k     3.9 / 4.3    5.5 / 4.0    9.4 / 5.9    14.1 / 7.5      16,384 x 2,048 k   27.5 / 31.8    32.4 / 32.7    43 / 33    64 / 35
//   2,048 x 2,048 k   5.9 / 6.7    7.8 / 6.7    11 / 7.6     15.5 / 8.8      32,000 x 2,048 k   46.6 / 51.0    52.8 / 52.8    74 / 54    120 / 65
//   3,072 x 2,048 k   7.8 / 8.1    10.0 / 8.7   15 / 10.1    20.3 / 12.9     16,384 x 8,192 k   92 / 105       104 / 108      142 / 108  226 / 108
//
// So one token (two, of large weights) takes up to 20 % longer than by FMAs; the choice of kernel looks at the weight alone, or a row's
// bits would depend on its step.
//
// The same sums by mma.sync, which rounds as tcgen05.mma does, whatever the order of the k inside a product (tests compare the
// bits): weights go from memory into registers and are split there, so nothing stands between a load and the next one. A block
// makes 16 weight rows; its warps take slices in turn, and a slice's sums meet in shared memory, where they are added in the
// order of the chains. A lane's 16 bytes of a row are four neighbouring k of the sixteen of a product.

__device__ __forceinline__ void few_mma(float (&c)[4], const unsigned (&a)[4], unsigned b0, unsigned b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
template <bool VEC>
__device__ __forceinline__ float4 few_load_w(const float* p) {
  float4 v;
  if (VEC) {
    asm volatile("ld.global.L1::no_allocate.L2::256B.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
  } else {
    asm volatile("ld.global.f32 %0, [%4];\n\tld.global.f32 %1, [%4 + 4];\n\tld.global.f32 %2, [%4 + 8];\n\tld.global.f32 %3, [%4 + 12];"
                 : "=&f"(v.x), "=&f"(v.y), "=&f"(v.z), "=&f"(v.w) : "l"(p));
  }
  return v;
}
// The parts of four neighbours, each part as two packed pairs.
__device__ __forceinline__ void split_4(const float4& v, unsigned (&h)[3][2]) {
  float e[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int part = 0; part < 3; ++part) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      h[part][i] = pack_rn(e[2 * i], e[2 * i + 1]);
      if (part < 2) {
        e[2 * i] -= __uint_as_float(h[part][i] << 16);
        e[2 * i + 1] -= __uint_as_float(h[part][i] & 0xffff0000u);
      }
    }
  }
}

// What a warp takes at a time: 64 k of each slice of a pair, or the two halves of a slice that has no partner; as many items as
// slices. Halves are counted over all slices: the item is half `a` = few_item >> 1 and half a + 1 + (few_item & 1).
__device__ __forceinline__ int few_item(int item, int slices) {
  int chain = 0;
  while (item >= (chain + 1) * slices / kChains) ++chain;
  const int c0 = chain * slices / kChains, n = (chain + 1) * slices / kChains - c0, at = item - c0;
  return at + 1 == n && (n & 1) ? 4 * item : 4 * item - 2 * (at & 1) + 1;
}

// T8: eights of tokens, a block's tile has 16 weight rows; 0: up to four tokens and a tile of 8 weight rows. A product's rows are then
// the 8 of one item over the 8 of the next one, its columns the tokens of the one beside those of the other, and two quarters of its
// result are used: two items a warp at a time, where the chain of a product on the one before it is what there is to wait for.
// VEC: rows on 16 bytes.
//
// Shared memory is kept small because the weights come through what it leaves of L1: with the tokens staged there, or their parts, 8,192 x
// 4,096 k took 36 us instead of 32.
template <int T8, bool VEC, int WARPS>
__global__ void __launch_bounds__(WARPS * 32, 16 / WARPS)
gemm_f32_few_rows_kernel(const float* A, const float* W, float* __restrict__ C, int M, int N, int K, int lda, int ldw, int ldc,
                         int w_written, int buffers) {
  constexpr bool PAIR = T8 == 0;
  constexpr int kX = PAIR ? 1 : T8, kRows = PAIR ? 8 : 16;
  constexpr int kHalf = kSliceK / 2;
  extern __shared__ __align__(16) float few_smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int tiles = (N + kRows - 1) / kRows, slices = K / kSliceK, turns = PAIR ? (slices + 1) / 2 : slices;
  // sums: [halves of slices][rows 8 to 15][odd tokens][pairs of tokens][8 rows]: a warp's stores are neighbours
  constexpr int kPairs = PAIR ? 2 : 4 * T8, kOut = 2 * kPairs * kRows;
  const int buffer = 2 * slices * kOut;
  const float *w_lo, *w_hi;               // of the turn that is loaded
  int lo_b, hi_b;                         // from where an item's first half ends to its second one
  // the items of a turn: one, or two (after an odd number of them the last one twice)
  auto item_lo = [&](int turn) { return few_item(PAIR ? 2 * turn : turn, slices); };
  auto item_hi = [&](int turn) { return few_item(min(2 * turn + 1, slices - 1), slices); };
  auto point = [&](int tile, int f_lo, int f_hi) {
    const float* w = W + 4 * t;
    w_lo = w + (size_t)min(tile * kRows + g, N - 1) * ldw + (f_lo >> 1) * kHalf;
    w_hi = w + (size_t)min(tile * kRows + g + (PAIR ? 0 : 8), N - 1) * ldw + (f_hi >> 1) * kHalf;
    lo_b = (f_lo & 1) * kHalf;
    hi_b = (f_hi & 1) * kHalf;
  };
  float4 lo[8], hi[8];                    // a turn of this warp: eight products' worth of k
  auto load = [&](int j) {
    lo[j] = few_load_w<VEC>(w_lo + 16 * j + (j < 4 ? 0 : lo_b));
    hi[j] = few_load_w<VEC>(w_hi + 16 * j + (j < 4 ? 0 : hi_b));
  };
  const int first = min(warp, turns - 1);
  const int first_lo = item_lo(first), first_hi = PAIR ? item_hi(first) : first_lo;
  point(blockIdx.x, first_lo, first_hi);
  if (w_written) pdl_wait();
  if (warp < turns) {
#pragma unroll
    for (int j = 0; j < 8; ++j) load(j);
  }
  pdl_wait();
  int which = 0;                          // buffer of this tile's sums
#pragma unroll 1
  for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    float* sums = few_smem + which * buffer;
    int f_lo = first_lo, f_hi = first_hi;
#pragma unroll 1
    for (int turn = warp; turn < turns; turn += WARPS) {
      float g1[kX][4], g2[kX][4];
      // the next turn of this tile, or this warp's first of the block's next tile
      const bool more = turn + WARPS < turns;
      const int next_lo = more ? item_lo(turn + WARPS) : first_lo;
      const int next_hi = !PAIR ? next_lo : more ? item_hi(turn + WARPS) : first_hi;
      point(more ? tile : min(tile + (int)gridDim.x, tiles - 1), next_lo, next_hi);
      const unsigned minus = (unsigned)(PAIR && g >= 4 ? f_hi : f_lo) << 31;
      auto store = [&](bool second) {
        const int u_lo = (f_lo >> 1) + (second ? 1 + (f_lo & 1) : 0), u_hi = (f_hi >> 1) + (second ? 1 + (f_hi & 1) : 0);
        if (PAIR) {
          float* to = sums + (t < 2 ? u_lo : u_hi) * kOut + (t & 1) * 8 + g;
          to[0] = t < 2 ? g1[0][0] + g2[0][0] : g1[0][2] + g2[0][2];
          to[kPairs * 8] = t < 2 ? g1[0][1] + g2[0][1] : g1[0][3] + g2[0][3];
        } else {
#pragma unroll
          for (int i = 0; i < kX; ++i) {
            float* to = sums + u_lo * kOut + (4 * i + t) * 8 + g;
#pragma unroll
            for (int e = 0; e < 4; ++e) to[e * kPairs * 8] = g1[i][e] + g2[i][e];
          }
        }
      };
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        if (j == 4) store(false);
        if (j % 4 == 0) {
#pragma unroll
          for (int i = 0; i < kX; ++i)
#pragma unroll
            for (int e = 0; e < 4; ++e)
              if (j == 0 || !((e < 2 ? f_lo : f_hi) & 1)) g1[i][e] = g2[i][e] = 0.f;
        }
        unsigned a[2][3][2];
        split_4(lo[j], a[0]);
        split_4(hi[j], a[1]);
        load(j);
        unsigned w[3][4];
#pragma unroll
        for (int p = 0; p < 3; ++p) {
          w[p][0] = a[0][p][0];
          w[p][1] = a[1][p][0];
          w[p][2] = a[0][p][1];
          w[p][3] = a[1][p][1];
        }
#pragma unroll
        for (int i = 0; i < kX; ++i) {
          const int f = PAIR && g >= 4 ? f_hi : f_lo, token = min(PAIR ? g & 3 : g + 8 * i, M - 1);
          float4 v = load_4<VEC>(A + (size_t)token * lda + ((f >> 1) + (j < 4 ? 0 : f & 1)) * kHalf + 16 * j + 4 * t);
          if (j >= 4) {                   // subtracted from the pair's first slice
            v.x = __uint_as_float(__float_as_uint(v.x) ^ minus);
            v.y = __uint_as_float(__float_as_uint(v.y) ^ minus);
            v.z = __uint_as_float(__float_as_uint(v.z) ^ minus);
            v.w = __uint_as_float(__float_as_uint(v.w) ^ minus);
          }
          unsigned x[3][2];
          split_4(v, x);
          few_mma(g1[i], w[0], x[0][0], x[0][1]);
          few_mma(g2[i], w[0], x[1][0], x[1][1]);
          few_mma(g2[i], w[0], x[2][0], x[2][1]);
          few_mma(g2[i], w[1], x[0][0], x[0][1]);
          few_mma(g2[i], w[1], x[1][0], x[1][1]);
          few_mma(g2[i], w[2], x[0][0], x[0][1]);
        }
      }
      store(true);
      f_lo = next_lo;
      f_hi = next_hi;
    }
    __syncthreads();
    if (warp * 32 < kOut) {
      // the four chains side by side; they differ by a slice at most
      const float* from[kChains];
      int n[kChains];
      float P[kChains];
#pragma unroll
      for (int c = 0; c < kChains; ++c) {
        const int c0 = c * slices / kChains;
        n[c] = (c + 1) * slices / kChains - c0;
        from[c] = sums + 2 * c0 * kOut + min((int)threadIdx.x, kOut - 1);
        P[c] = 0.f;
      }
      const int most = (slices + kChains - 1) / kChains;
#pragma unroll 2
      for (int k = 0; k < most; ++k) {
#pragma unroll
        for (int c = 0; c < kChains; ++c) {
          if (k < n[c]) {
            const float times = k & 1 ? -1.f : k + 1 < n[c] ? 2.f : 1.f;
            P[c] = fmaf(times, from[c][(2 * k + 1) * kOut], fmaf(times, from[c][2 * k * kOut], P[c]));
          }
        }
      }
      float v = (P[0] + P[1]) + (P[2] + P[3]);
      const int part = (int)threadIdx.x / (8 * kPairs);
      const int row = tile * kRows + (threadIdx.x & 7) + (part >> 1) * 8, token = 2 * ((threadIdx.x >> 3) % kPairs) + (part & 1);
      const bool there = (int)threadIdx.x < kOut && row < N && token < M;
      for (unsigned again = __ballot_sync(0xffffffffu, there && !is_finite(v)); again; again &= again - 1) {
        const int at = __ffs(again) - 1;
        const float* w_row[1] = {W + (size_t)__shfl_sync(0xffffffffu, row, at) * ldw};
        float dot[1];
        warp_dots<1, VEC>(A + (size_t)__shfl_sync(0xffffffffu, token, at) * lda, w_row, K, dot);
        if (lane == at) v = dot[0];
      }
      if (there) C[(size_t)token * ldc + row] = v;
    }
    if (buffers == 2) which ^= 1;
    else if (tile + (int)gridDim.x < tiles) __syncthreads();      // else the next tile's sums would meet this one's readers
  }
}

constexpr int kFewSmem = 200 * 1024;      // of a block that has an SM to itself; two of half of it
constexpr int kFewSecond = 40 * 1024;     // up to here a block has two buffers of sums
constexpr int few_out(int t8) { return t8 ? 128 * t8 : 32; }
size_t few_sums(int K, int t8) { return (size_t)(K / kSliceK) * 2 * few_out(t8) * 4; }

template <int T8, bool VEC, int WARPS>
int launch_few(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldw, int ldc, int w_written,
               cudaStream_t stream) {
  constexpr int kLimit = kFewSmem / (16 / WARPS);
  constexpr int kRows = T8 ? 16 : 8;
  const int tiles = (N + kRows - 1) / kRows, slots = 148 * (16 / WARPS);
  const size_t sums = few_sums(K, T8);
  const int buffers = tiles > slots && 2 * sums <= kFewSecond ? 2 : 1;
  const size_t smem = buffers * sums;
  if (smem > kLimit) return LLMIE_ERR_UNSUPPORTED_SIZE;
  auto kernel = gemm_f32_few_rows_kernel<T8, VEC, WARPS>;
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kLimit);
  if (e != cudaSuccess) return (int)e;
  launch_k(kernel, dim3(tiles < slots ? tiles : slots), dim3(WARPS * 32), smem, stream, A, W, C, M, N, K, lda, ldw, ldc, w_written,
           buffers);
  LLMIE_LAUNCH_CHECK();
  return LLMIE_OK;
}

template <int NT, bool WIDE>
int launch_tc(const float* A, const float* W, float* C, void* parts, int M, int N, int K, int lda, int ldw, int ldc, int split,
              int w_written, bool no_wait, int* status, cudaStream_t stream) {
  using S = Shape<NT>;
  auto kernel = no_wait ? gemm_f32_tc_kernel<NT, WIDE, 0> : gemm_f32_tc_kernel<NT, WIDE, kSpinLimit>;
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, S::kSmem);
  if (e != cudaSuccess) return (int)e;
  const long long blocks = (long long)((M + NT - 1) / NT) * ((N + kMt - 1) / kMt) * split;
  if (blocks > 0x7fffffffLL) return LLMIE_ERR_UNSUPPORTED_SIZE;
  CUtensorMap map = {};
  if (!S::kSplitsX) {
    if (!parts) return LLMIE_ERR_BAD_ARG;
    EncodeTiledFn fn = encode_tiled_fn();
    if (!fn) return LLMIE_ERR_BAD_ARG;
    if (!aligned16(parts)) return LLMIE_ERR_ALIGNMENT;
    cuuint64_t dims[2] = {(cuuint64_t)K, 3 * (cuuint64_t)M}, pitch[1] = {(cuuint64_t)K * 2};
    cuuint32_t box[2] = {kStageK, NT}, one[2] = {1, 1};
    if (fn(&map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, parts, dims, pitch, box, one, CU_TENSOR_MAP_INTERLEAVE_NONE,
           CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return LLMIE_ERR_BAD_ARG;
    launch_k(split_rows_kernel<WIDE>, dim3((unsigned)(((long long)M * (K / 8) + 255) / 256)), dim3(256), 0, stream, A,
             (__nv_bfloat16*)parts, M, K, lda);
    LLMIE_LAUNCH_CHECK();
  }
  if (split > 1)
    launch_k_cluster(kernel, dim3((unsigned)blocks), dim3(kTcThreads), S::kSmem, stream, split, map, A, W, C, M, N, K, lda, ldw, ldc,
                     split, w_written, status);
  else
    launch_k(kernel, dim3((unsigned)blocks), dim3(kTcThreads), S::kSmem, stream, map, A, W, C, M, N, K, lda, ldw, ldc, split, w_written,
             status);
  LLMIE_LAUNCH_CHECK();
  return LLMIE_OK;
}

// One block an SM where there are no more, and turns enough for its warps; or where the sums of two leave too little (1 token, 4,096 x
// 12,288 k 45 us against 53; 4,096 x 8,192 k 35 against 32).
bool few_alone(int t8, int N, int K) {
  return (t8 ? N <= 148 * 16 : N <= 148 * 8 && K > 16 * kSliceK) || few_sums(K, t8) > 80 * 1024;
}
// Whether a product of few rows fits the kernel: its sums, whose number follows K.
bool few_takes(int t8, int K, bool alone) { return few_sums(K, t8) <= (alone ? kFewSmem : kFewSmem / 2); }
template <int T8>
int few_form(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldw, int ldc, int w_written,
             bool alone, cudaStream_t stream) {
  const bool vec = aligned16(A) && aligned16(W) && ((lda | ldw) & 3) == 0;
#define LLMIE_FEW(vec_, warps_) launch_few<T8, vec_, warps_>(A, W, C, M, N, K, lda, ldw, ldc, w_written, stream)
  if (alone) return vec ? LLMIE_FEW(true, 16) : LLMIE_FEW(false, 16);
  return vec ? LLMIE_FEW(true, 8) : LLMIE_FEW(false, 8);
#undef LLMIE_FEW
}

// 1 when the kernel takes a weight [N, K]. The answer depends on the weight alone: a row's bits are then the same in every step.
bool takes(int N, int K) { return N >= 128 && K >= 1024 && K % kSliceK == 0; }

// form: tokens a block (8: the kernel for up to 16 tokens, 4: its form for up to 4; 16, 64, 80) + 1000 * split (blocks of a tile: 1, 2, 4;
// of the kernel for few tokens 2: eight warps a block, 4: sixteen), for tests: every form gives the same bits. 0:
// chosen by size. + 10000: every wait gives up at once (for tests of that path; the sums are then made by plain FMAs). `parts`: 3 M K bfloat16 of scratch, not needed for 16 tokens a block.
int product(const float* A, const float* W, float* C, void* parts, int M, int N, int K, int lda, int ldw, int ldc, int form,
            int w_written, int* status, cudaStream_t stream) {
  if (M < 0 || N <= 0 || K <= 0 || lda < K || ldw < K || ldc < N || !status) return LLMIE_ERR_BAD_ARG;
  if (!takes(N, K)) return LLMIE_ERR_UNSUPPORTED_SIZE;
  if (M == 0) return LLMIE_OK;
  const bool no_wait = form >= 10000;
  form %= 10000;
  int nt = form % 1000, split = form / 1000;
  if (form == 0) {
    const long long rows = (N + kMt - 1) / kMt;
    // blocks of a tile: as many as fit the GPU at once, a block a SM (33 clusters of 4, 74 of 2)
    auto share = [&](int n) {
      const long long tiles = (M + n - 1) / n * rows;
      return tiles <= 33 ? 4 : tiles <= 74 ? 2 : 1;
    };
    if (M <= 16) {
      // microseconds, the kernel for few rows / 16 tokens a block: 8 rows, 8,192 x 4,096 k 35.7 / 35.3, 16,384 x 4,096 k 64 / 60,
      // 32,000 x 4,096 k 108 / 115; 16 rows, 3,072 x 1,024 k 8.0 / 9.5, x 2,048 k 12.8 / 12.9, x 4,096 k 23.0 / 19.5
      const int t8 = M <= 8 ? 1 : 2;
      const bool few = few_takes(t8, K, few_alone(t8, N, K)) &&
                       (M <= 4 || (M <= 8 ? !(K >= 4096 && N >= 8192 && N <= 148 * kMt) : N <= 148 * 16 || (N < 8192 && K <= 1024)));
      // two items at a time / one, 4 rows: 512 x 2,048 k 4.0 / 6.1, 2,048 x 2,048 k 6.7 / 7.5, 3,072 x 4,096 k 15.8 / 17.5,
      // 4,096 x 4,096 k 18.9 / 18.8, 8,192 x 8,192 k 62 / 61
      nt = M <= 4 && N <= 3072 && few_takes(0, K, few_alone(0, N, K)) ? 4 : few ? 8 : 16;
    } else {
      // a block's time does not follow its tokens (2,048 k: 35 us with 64, 37 with 80), so what counts is how many rounds of
      // blocks there are, and how many share a tile
      auto cost = [&](int n, int us) {
        const long long blocks = (M + n - 1) / n * rows * share(n);
        return (double)us * ((blocks + 147) / 148) / share(n);
      };
      nt = cost(64, 35) <= cost(80, 37) ? 64 : 80;
    }
    split = share(nt);
  }
  if (split != 1 && split != 2 && split != 4) return LLMIE_ERR_BAD_ARG;
  const bool wide = ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(W)) & 31) == 0 && ((lda | ldw) & 7) == 0;
  if (nt == 4 || nt == 8) {
    const int t8 = nt == 4 ? 0 : M <= 8 ? 1 : 2;
    const bool alone = form / 1000 > 1 ? split == 4 : few_alone(t8, N, K);
    if (M > (nt == 4 ? 4 : 16) || !few_takes(t8, K, alone)) return LLMIE_ERR_UNSUPPORTED_SIZE;
    return t8 == 0   ? few_form<0>(A, W, C, M, N, K, lda, ldw, ldc, w_written, alone, stream)
           : t8 == 1 ? few_form<1>(A, W, C, M, N, K, lda, ldw, ldc, w_written, alone, stream)
                     : few_form<2>(A, W, C, M, N, K, lda, ldw, ldc, w_written, alone, stream);
  }
#define LLMIE_TC(nt_)                                                                                     \
  case nt_:                                                                                               \
    return wide ? launch_tc<nt_, true>(A, W, C, parts, M, N, K, lda, ldw, ldc, split, w_written, no_wait, status, stream)      \
                : launch_tc<nt_, false>(A, W, C, parts, M, N, K, lda, ldw, ldc, split, w_written, no_wait, status, stream)
  switch (nt) {
    LLMIE_TC(16);
    LLMIE_TC(64);
    LLMIE_TC(80);
    default: return LLMIE_ERR_BAD_ARG;
  }
#undef LLMIE_TC
}

}  // namespace
}  // namespace llmie

using namespace llmie;

extern "C" int llmie_gemm_f32_tc_takes(int N, int K) { return takes(N, K) ? 1 : 0; }

extern "C" int llmie_gemm_f32_tc_form(const float* A, const float* W, float* C, void* parts, int M, int N, int K, int lda, int ldw,
                                      int ldc, int form, int* status, cudaStream_t stream) {
  return product(A, W, C, parts, M, N, K, lda, ldw, ldc, form, 1, status, stream);
}

// w_written: whether a kernel in front may have written W, which is then read behind the wait for it.
extern "C" int llmie_gemm_f32_tc(const float* A, const float* W, float* C, void* parts, int M, int N, int K, int lda, int ldw,
                                 int ldc, int w_written, int* status, cudaStream_t stream) {
  return product(A, W, C, parts, M, N, K, lda, ldw, ldc, 0, w_written, status, stream);
}
