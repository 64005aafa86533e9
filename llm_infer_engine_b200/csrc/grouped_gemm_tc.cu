// Many matrix products of one shape in one launch, C_g = A_g W_g^T, bfloat16 in and out, on the 5th-generation tensor cores
// (tcgen05.mma, float32 accumulators in tensor memory): what prompts give to the products of grouped_gemm.cu. Two forms:
//
//   batched   every group has the same M rows; group g reads columns [g * a_gcs, + K) of A and writes columns
//             [g * c_gcs, + N) of C (the heads of an attention layer, each with a matrix of its own)
//   routed    group g has rows [group_end[g - 1], group_end[g]) of A and C (the experts of a routed feed-forward, rows
//             sorted by expert); rows behind the last group's are neither read for a result nor written
//
// W is [groups][N (or 2 N), K]. With DUAL it is [gate rows | up rows] and the result is act(A gate^T) * (A up^T), both
// products rounded to bfloat16 first, as two launches would leave them; otherwise act(A W^T).
//
// One block per SM walks over the tiles (128 rows x BN weight rows; the row tiles of one slice of weights follow one another,
// so the slice comes from memory once). Warp 0 loads (TMA, 128-byte swizzle, a ring of stages of 64 k), warp 1 multiplies,
// warps 2 to 9 (to 17 with a gate) take the sums out of tensor memory, two tiles of sums in turn, while the next tile is multiplied. Every wait is
// bounded; one that gives up records a status, what the block has not finished becomes NaN (C may hold something else that
// looks like a result: the routed experts' second product writes over their gathered inputs), and the block waits for its copies
// and products, frees its tensor memory and returns.
//
// What bounds it: many rows, shared memory (a stage of 48 KB is written and read once for 512 cycles of products); few, the
// weights' way from memory; one short K (attention heads), the way of the results out of tensor memory, hence eight warps for
// it (four: 15.5 us where eight take 13.4) and stores of 64 bytes a row (a thread storing its own row: 17.5). With a gate, the
// activation of the tile that a block ends with: its divisions wait for one another, so sixteen warps (eight, silu: 16 experts of 2 x
// 2,048 x 2,048, 600 pairs 59 us where sixteen take 54; 8 of 2 x 1,408 x 4,096, 2,400 pairs 87 / 79).
//
// Measured, us, the vendor's grouped products with the activation (silu) by itself / this, gate and up with it + down: 16 experts of 2 x 2,048
// x 2,048 and 2,048 x 2,048, 600 pairs 71 + 39 / 53 + 27, 2,400 pairs 72 + 36 / 72 + 36, 5,331 pairs 114 + 54 / 97 + 49, 16,384 pairs 250 +
// 113 / 221 + 126; 8 of 2 x 1,408 x 4,096, 600 pairs 76 + 33 / 46 + 18, 5,331 pairs 114 + 56 / 117 + 62, 16,384 pairs 301 + 135 / 279 + 151;
// 128 of 2 x 768 x 2,048, 3,000 pairs 171 + 93 / 139 + 67; 32 of 2 x 1,024 x 2,880, 2,400 pairs 99 + 56 / 71 + 39, 5,331 pairs 95 + 50 / 99 +
// 54. So from some 500 rows an expert on the down product takes up to 13 % longer, both together up to 5 % (8 of 1,408 x 4,096 with 670
// rows each, 32 of 1,024 x 2,880 with 170: tiles of 128 rows that are two thirds full, rounds of blocks that are nearly empty). Heads, the
// mma.sync kernel / this: 32 of 256 x 64, 2,130 rows 22.8 / 13.4; of 64 x 256, 19.9 / 9.3.
#include "tcgen05.cuh"

namespace llmie {
using namespace tc;

namespace {

constexpr int kRows = 128, kK = 64;
constexpr int kRing = 192 * 1024;                 // bytes of the ring of stages
constexpr int kMostGroups = 1024;
template <bool DUAL> constexpr int kEpilogueWarps = DUAL ? 16 : 8;
template <bool DUAL> constexpr int kThreads = 64 + 32 * kEpilogueWarps<DUAL>;
constexpr int kStaged = 8 * 32 * 64;              // 32 rows x 32 columns of results for each epilogue warp, on their way to memory
constexpr int kSmem = kRing + kStaged + 1024 + 2 * (kMostGroups + 1) * 4;

struct Args {
  __nv_bfloat16* C;
  long long ldc, c_gcs;
  const int* group_end;
  int groups, M, N, K, a_gcs, act;
  int* status;
};

struct Shared {
  uint64_t full[8], empty[8], acc_full[2], acc_empty[2], drained;
  uint32_t tmem;
  int abort, loaded;       // loaded: stages that warp 0 has asked for
};

__device__ __forceinline__ void give_up(volatile int* abort, int* status, int code) {
  if (!*abort) { *abort = 1; atomicExch(status, code); }
}

// LIMIT: polls before a wait gives up, a constant as in attention_latent_tc.cu.
template <int BN, bool DUAL, unsigned LIMIT>
__global__ void __launch_bounds__(kThreads<DUAL>, 1)
grouped_tc_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w, const Args p) {
  constexpr int kStageBytes = (kRows + BN) * kK * 2;
  constexpr int kStages = kRing / kStageBytes;            // 4 at BN 256, 6 at 128, 8 at 64
  constexpr int kCols = DUAL ? BN / 2 : BN;               // columns of C a tile covers
  constexpr int kParts = kEpilogueWarps<DUAL> / 4, kChunk = DUAL ? 16 : 32, kPieces = kChunk / 8;
  extern __shared__ uint8_t smem_raw[];
  __shared__ Shared sh;
  uint8_t* ring = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  int* tile0 = reinterpret_cast<int*>(ring + kRing + kStaged);      // first tile of each group, groups + 1 of them
  int* row0 = tile0 + p.groups + 1;                       // first row of each group, groups + 1
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int k_tiles = (p.K + kK - 1) / kK, n_tiles = (p.N + kCols - 1) / kCols;

  pdl_launch_dependents();
  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&sh.full[s], 1);
      mbar_init(&sh.empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&sh.acc_full[b], 1);
      mbar_init(&sh.acc_empty[b], kEpilogueWarps<DUAL>);
    }
    mbar_init(&sh.drained, 1);
    sh.abort = sh.loaded = 0;
    fence_mbar_init();
    tma_prefetch_desc(&map_a);
    tma_prefetch_desc(&map_w);
  }
  if (warp == 1) {
    tmem_alloc(&sh.tmem, 2 * BN);
    tmem_relinquish();
  }
  pdl_wait();
  if (warp == 0) {                                        // where the groups' tiles and rows begin
    int before = 0;
    for (int e0 = 0; e0 < p.groups; e0 += 32) {
      const int e = e0 + lane;
      int rows = 0, first = 0;
      if (e < p.groups) {
        if (p.group_end) {
          first = e ? min(max(p.group_end[e - 1], 0), p.M) : 0;
          rows = max(min(p.group_end[e], p.M) - first, 0);
        } else {
          rows = p.M;
        }
        row0[e] = first;
      }
      const int tiles = (rows + kRows - 1) / kRows * n_tiles;
      int sum = tiles;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, sum, o);
        if (lane >= o) sum += v;
      }
      if (e < p.groups) tile0[e] = before + sum - tiles;
      before += __shfl_sync(0xffffffffu, sum, 31);
    }
    if (lane == 0) {
      tile0[p.groups] = before;
      row0[p.groups] = p.group_end ? min(max(p.group_end[p.groups - 1], 0), p.M) : p.M;
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = sh.tmem;
  volatile int* abort = &sh.abort;
  const int n_all = tile0[p.groups];

  if (warp == 0) {
    if (elect_one()) {
      int it = 0, e = 0;
      bool ok = true;
      for (int t = blockIdx.x; t < n_all && ok; t += gridDim.x) {
        while (t >= tile0[e + 1]) ++e;
        const int r = t - tile0[e], m_tiles = (tile0[e + 1] - tile0[e]) / n_tiles;
        const int m0 = row0[e] + r % m_tiles * kRows, n0 = r / m_tiles * kCols;
        const int w0 = e * (DUAL ? 2 * p.N : p.N) + n0;
        for (int kt = 0; kt < k_tiles; ++kt, ++it) {
          const int s = it % kStages;
          if (it >= kStages && !mbar_wait(&sh.empty[s], ((it / kStages) - 1) & 1, abort, LIMIT)) {
            give_up(abort, p.status, kStatusTimeoutEmpty);
            ok = false;
            break;
          }
          uint8_t* a = ring + s * kStageBytes;
          uint8_t* w = a + kRows * kK * 2;
          mbar_arrive_expect_tx(&sh.full[s], kStageBytes);
          tma_load_2d(a, &map_a, (p.group_end ? 0 : e * p.a_gcs) + kt * kK, m0, &sh.full[s]);
          tma_load_2d(w, &map_w, kt * kK, w0, &sh.full[s]);
          if (DUAL) tma_load_2d(w + BN / 2 * kK * 2, &map_w, kt * kK, w0 + p.N, &sh.full[s]);
        }
      }
      sh.loaded = it;
    }
  } else if (warp == 1) {
    if (elect_one()) {
      constexpr uint32_t idesc = make_instr_desc_bf16(kRows, BN, 0, 0);
      int it = 0, i = 0;
      bool ok = true;
      for (int t = blockIdx.x; t < n_all && ok; t += gridDim.x, ++i) {
        const int buf = i & 1;
        if (i >= 2 && !mbar_wait(&sh.acc_empty[buf], ((i >> 1) - 1) & 1, abort, LIMIT)) {
          give_up(abort, p.status, kStatusTimeoutMma);
          break;
        }
        tc_fence_after_sync();
        for (int kt = 0; kt < k_tiles; ++kt, ++it) {
          const int s = it % kStages;
          if (!mbar_wait(&sh.full[s], (it / kStages) & 1, abort, LIMIT)) {
            give_up(abort, p.status, kStatusTimeoutFull);
            ok = false;
            break;
          }
          tc_fence_after_sync();
          const uint32_t a = smem_u32(ring + s * kStageBytes), w = a + kRows * kK * 2;
#pragma unroll
          for (int kk = 0; kk < kK / 16; ++kk)
            mma_bf16_ss(tmem + buf * BN, make_smem_desc(a + kk * 32, 16, 1024), make_smem_desc(w + kk * 32, 16, 1024), idesc,
                        (kt > 0 || kk > 0) ? 1u : 0u);
          mma_commit(&sh.empty[s]);
        }
        if (ok) mma_commit(&sh.acc_full[buf]);
      }
    }
  } else {
    const int quarter = warp & 3;                          // the tensor memory lanes this warp may read
    const int c_first = (warp - 2) / 4 * (kCols / kParts);    // and its part of the columns
    int e = 0, i = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < n_all; t += gridDim.x, ++i) {
      while (t >= tile0[e + 1]) ++e;
      const int r = t - tile0[e], m_tiles = (tile0[e + 1] - tile0[e]) / n_tiles;
      const int end = p.group_end ? row0[e + 1] : p.M;
      const int row = row0[e] + r % m_tiles * kRows + quarter * 32, n0 = r / m_tiles * kCols;
      const int buf = i & 1;
      __nv_bfloat16* dst = p.C + (size_t)row * p.ldc + (p.group_end ? 0 : (size_t)e * p.c_gcs) + n0;
      ok = ok && __all_sync(0xffffffffu, mbar_wait(&sh.acc_full[buf], (i >> 1) & 1, abort, LIMIT));
      if (!ok) {                                           // neither this tile nor those behind it have a result
        give_up(abort, p.status, kStatusTimeoutMma);
        const uint4 nan8 = make_uint4(0x7fff7fffu, 0x7fff7fffu, 0x7fff7fffu, 0x7fff7fffu);
        for (int at = lane; at < 32 * (kCols / kParts / 8); at += 32) {
          const int rr = at / (kCols / kParts / 8), col = c_first + at % (kCols / kParts / 8) * 8;
          if (row + rr < end && n0 + col < p.N) *reinterpret_cast<uint4*>(dst + (size_t)rr * p.ldc + col) = nan8;
        }
        continue;
      }
      tc_fence_after_sync();
      const uint32_t acc = tmem + ((uint32_t)(quarter * 32) << 16) + buf * BN;
      uint8_t* staged = ring + kRing + (warp - 2) * (32 * kChunk * 2);
#pragma unroll 1
      for (int c = c_first; c < c_first + kCols / kParts; c += kChunk) {
        float v[kPieces][8];
        uint32_t g[kChunk];
        if constexpr (DUAL) {
          uint32_t u[kChunk];
          tmem_ld_32x16(acc + c, g);
          tmem_ld_32x16(acc + BN / 2 + c, u);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < kChunk; ++j)
            v[j >> 3][j & 7] = apply_act(__bfloat162float(__float2bfloat16(__uint_as_float(g[j]))), p.act) *
                               __bfloat162float(__float2bfloat16(__uint_as_float(u[j])));
        } else {
          tmem_ld_32x32(acc + c, g);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < kChunk; ++j) v[j >> 3][j & 7] = __uint_as_float(g[j]);
          if (p.act) {
#pragma unroll
            for (int j = 0; j < kChunk; ++j)
              v[j >> 3][j & 7] = apply_act(__bfloat162float(__float2bfloat16(v[j >> 3][j & 7])), p.act);
          }
        }
        // a thread has a row: through shared memory (the 16-byte pieces of a row in swizzled order) to stores in which
        // neighbours write neighbouring pieces
        const int swizzle = kPieces - 1;
#pragma unroll
        for (int j = 0; j < kPieces; ++j)
          store8(reinterpret_cast<__nv_bfloat16*>(staged + lane * (kChunk * 2) + ((j ^ (lane * kPieces / 8 & swizzle)) << 4)), v[j]);
        __syncwarp();
        const int piece = lane % kPieces, col = c + piece * 8;
#pragma unroll
        for (int j = 0; j < kPieces; ++j) {
          const int rr = j * (32 / kPieces) + lane / kPieces;
          const uint4 x = *reinterpret_cast<const uint4*>(staged + rr * (kChunk * 2) + ((piece ^ (rr * kPieces / 8 & swizzle)) << 4));
          if (row + rr < end && n0 + col < p.N) *reinterpret_cast<uint4*>(dst + (size_t)rr * p.ldc + col) = x;
        }
        __syncwarp();
      }
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&sh.acc_empty[buf]);
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  if (*abort) {
    // whichever role gave up: copies and products still in flight end (bounded) before the block gives its memory up
    if (threadIdx.x == 0) {
      for (int i = max(0, sh.loaded - kStages); i < sh.loaded; ++i)
        for (unsigned spin = 0; spin < (1u << 16) && !mbar_test(&sh.full[i % kStages], (i / kStages) & 1); ++spin)
          __nanosleep(64);
    }
    if (warp == 1 && elect_one()) {                        // the lane that issued the products
      mma_commit(&sh.drained);
      for (unsigned spin = 0; spin < (1u << 16) && !mbar_test(&sh.drained, 0); ++spin) __nanosleep(64);
    }
    __syncthreads();
  }
  if (warp == 1) tmem_dealloc(tmem, 2 * BN);
}

template <int BN, bool DUAL>
int launch(const CUtensorMap& map_a, const void* W, const Args& p, bool no_wait, cudaStream_t stream) {
  CUtensorMap map_w;
  const int rc = make_tmap_bf16_2d(&map_w, W, (uint64_t)p.groups * p.N * (DUAL ? 2 : 1), (uint64_t)p.K, (uint64_t)p.K,
                                   DUAL ? BN / 2 : BN);
  if (rc != LLMIE_OK) return rc;
  auto kernel = no_wait ? grouped_tc_kernel<BN, DUAL, 0> : grouped_tc_kernel<BN, DUAL, kSpinLimit>;
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem);
  if (e != cudaSuccess) return (int)e;
  const int kCols = DUAL ? BN / 2 : BN;
  const long long n_tiles = (p.N + kCols - 1) / kCols, m_tiles = (p.M + kRows - 1) / kRows;
  const long long most = n_tiles * (p.group_end ? m_tiles + p.groups : m_tiles * p.groups);
  if (most > 0x3fffffff) return LLMIE_ERR_UNSUPPORTED_SIZE;
  launch_k(kernel, dim3((unsigned)(most < 148 ? most : 148)), dim3(kThreads<DUAL>), kSmem, stream, map_a, map_w, p);
  LLMIE_LAUNCH_CHECK();
  return LLMIE_OK;
}

}  // namespace
}  // namespace llmie

using namespace llmie;

// A [M, lda], W [groups, N or 2 N (dual), K] contiguous, C [M, ldc], all bfloat16 and on 16 bytes. group_end (int32 [groups],
// rising) = the routed form, null = the batched one. Strides, group columns, N and K in multiples of 8 elements; K of the
// batched form a multiple of 64 (a stage of 64 k of A would reach into the next group's columns). At most 1,024 groups.
// no_wait != 0: every wait gives up at once (for tests of that path).
extern "C" int llmie_grouped_gemm_tc_form(const void* A, long long lda, long long a_gcs, const void* W, void* C, long long ldc,
                                          long long c_gcs, const int* group_end, int groups, int M, int N, int K, int dual, int act,
                                          int* status, int no_wait, cudaStream_t stream) {
  if (M < 0 || N <= 0 || K <= 0 || groups <= 0 || a_gcs < 0 || c_gcs < 0 || !status) return LLMIE_ERR_BAD_ARG;
  if (groups > kMostGroups || K % 8 || N % 8 || lda % 8 || ldc % 8 || a_gcs % 8 || c_gcs % 8 || (!group_end && K % 64) ||
      (dual && !group_end) || (group_end && (lda < K || ldc < N)) || (!group_end && (lda < (groups - 1) * a_gcs + K || ldc < (groups - 1) * c_gcs + N)) ||
      (long long)groups * N * 2 > 0x7fffffff || lda > 0x7fffffff)
    return LLMIE_ERR_UNSUPPORTED_SIZE;
  if (!aligned16(A) || !aligned16(W) || !aligned16(C)) return LLMIE_ERR_ALIGNMENT;
  if (M == 0) return LLMIE_OK;
  CUtensorMap map_a;
  const int rc = tc::make_tmap_bf16_2d(&map_a, A, (uint64_t)M, group_end ? (uint64_t)K : (uint64_t)((groups - 1) * a_gcs + K),
                                       (uint64_t)lda, kRows);
  if (rc != LLMIE_OK) return rc;
  const Args p = {(__nv_bfloat16*)C, ldc, c_gcs, group_end, groups, M, N, K, (int)a_gcs, act, status};
  if (dual) return launch<256, true>(map_a, W, p, no_wait, stream);
  if (N <= 64) return launch<64, false>(map_a, W, p, no_wait, stream);
  if (N <= 128) return launch<128, false>(map_a, W, p, no_wait, stream);
  return launch<256, false>(map_a, W, p, no_wait, stream);
}

extern "C" int llmie_grouped_gemm_tc(const void* A, long long lda, long long a_gcs, const void* W, void* C, long long ldc,
                                     long long c_gcs, const int* group_end, int groups, int M, int N, int K, int dual, int act,
                                     int* status, cudaStream_t stream) {
  return llmie_grouped_gemm_tc_form(A, lda, a_gcs, W, C, ldc, c_gcs, group_end, groups, M, N, K, dual, act, status, 0, stream);
}
