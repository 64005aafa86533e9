// True float32 matrix product for the 32-bit path: C[M, N] = A[M, K] * W[N, K]^T, FMA on the
// CUDA cores, for the weights that gemm_f32_tc.cu does not take (few rows or a short or odd K).
//
// One summation order for every shape. K is cut into slices of 128; chain j (j = 0..7) takes the slices j, j + 8, ...
// in turn and keeps two running sums, of its even and of its odd k (the two halves of a packed fma.rn.f32x2); P_j is
// their sum, and the result is ((P_0 + P_1) + P_2) + ... + P_7. Both kernels below compute exactly this, so a row's
// result does not depend on which other rows share the launch, on the tile or on how K was split among blocks.
//
// (Sizes below from before gemm_f32_tc.cu took them; the bounds hold for what is left, weights whose K is short or not whole 128s.)
// What bounds it: up to 16 rows the weights' way from memory (32,000 x 2,048, one row: 45 us, 5.8 TB/s); above, the FMA
// rate (148 SMs x 128 lanes x 2 x 1.965 GHz = 74 TFLOP/s) less what the 128 sums of a thread cost: eight warps an SM, which
// wait for dependent instructions in between (2,048 x 8,192, 301 rows: FMA pipes 60 %, issue 39 %, shared memory 41 %; 16,384
// x 2,048, 512 rows: 48 TFLOP/s). A gated feed-forward of 2,048 / 8,192 at 301 rows: 2,820 us with one plain 64 x 64 tile a
// block, 785 us so (39 TFLOP/s; 301 rows fill tiles of 320); a one-token step of 3 rows 4.4 -> 0.3 ms. Eight chains also
// halve the error against 64-bit sums several times (2,048 terms: 2.0e-6 with one chain, 5e-7 so, relative).
//
// These kernels wait for the one before them and let the next one start when they are done: letting it start early left the
// time of a step as it was.
#include "common.cuh"

namespace llmie {

constexpr int kSlice = 128;
constexpr int kChains = 8;

__device__ __forceinline__ void fma2(float2& acc, const float2& a, const float2& b) {
  unsigned long long& c = reinterpret_cast<unsigned long long&>(acc);
  asm("fma.rn.f32x2 %0, %1, %2, %0;"
      : "+l"(c)
      : "l"(reinterpret_cast<const unsigned long long&>(a)), "l"(reinterpret_cast<const unsigned long long&>(b)));
}

// Copies of 16 bytes (or of four single floats where rows are not 16-byte aligned) from global into shared memory that
// complete asynchronously; `n_valid` floats of the four are read, the others are zeros.
template <bool VEC>
__device__ __forceinline__ void copy4(float* dst, const float* src, const float* safe, int n_valid) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  if (VEC) {
    const int bytes = n_valid <= 0 ? 0 : (n_valid >= 4 ? 16 : 4 * n_valid);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(bytes ? src : safe), "r"(bytes) : "memory");
  } else {
#pragma unroll
    for (int e = 0; e < 4; ++e)
      asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d + 4 * e), "l"(e < n_valid ? src + e : safe),
                   "r"(e < n_valid ? 4 : 0)
                   : "memory");
  }
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int LEFT>
__device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(LEFT) : "memory"); }

__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.aligned;\nbarrier.cluster.wait.aligned;" ::: "memory");
}
__device__ __forceinline__ float4 read_peer(const float4* p, unsigned rank) {
  unsigned a = (unsigned)__cvta_generic_to_shared(p), r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(r));
  return v;
}

// ---------------------------------------------------------------------------------------------------------------
// Tiles for more than kFewRows rows: WM x WN warps, each 32 x 64 outputs, a thread 8 x 8 of them (rows lane / 8 + 4 i,
// columns lane % 8 + 8 j), all 32 k of a stage read as eight 16-byte pieces a row: rows lie 36 floats apart in shared
// memory, so the eight rows a 16-byte access touches fall on different banks. The 8 x 8 packed sums are 128 registers;
// at a chain's end they are added up into shared memory, a slot per thread. `split` blocks of a cluster share a tile's
// chains (8 / split chains each, rank 0 the first ones); their sums meet in distributed shared memory in chain order.
constexpr int kBK = 32, kStride = 36;

template <int WM, int WN>
struct Tile {
  static constexpr int BM = 32 * WM, BN = 64 * WN, kThreads = 32 * WM * WN;
  // two stages of 32 k: four blocks share an SM, a barrier for every 1,024 packed FMAs a thread (2,048 x 8,192, 301 rows: 275
  // us; four stages of 16 k 292, three of 32 k, three blocks an SM, 294)
  static constexpr int kStages = 2;
  static constexpr int kStageFloats = (BM + BN) * kStride;
  static constexpr int kSumFloats = BM * BN;
  // the sums of the last chain of a rank > 0 lie where the stages were
  static constexpr int kRing = kStages * kStageFloats > kSumFloats ? kStages * kStageFloats : kSumFloats;
  static constexpr int smem_bytes() { return 4 * (kRing + kSumFloats); }
};

template <int WM, int WN, bool VEC>
__global__ void __launch_bounds__(32 * WM * WN)
gemm_f32_tile_kernel(const float* A, const float* W, float* __restrict__ C, int M, int N,
                     int K, int lda, int ldw, int ldc, int split) {
  using T = Tile<WM, WN>;
  extern __shared__ float4 smem4[];
  float* ring = reinterpret_cast<float*>(smem4);
  float4* held = smem4 + T::kRing / 4;                    // [16][kThreads]: a thread's 64 sums of earlier chains
  pdl_wait();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int rank = blockIdx.x % split;
  const int m0 = blockIdx.y * T::BM, n0 = (blockIdx.x / split) * T::BN;
  const int row_a = (warp / WN) * 32 + (lane >> 3), row_w = T::BM + (warp % WN) * 64 + (lane & 7);

  const int n_chains = kChains / split, chain0 = rank * n_chains;
  const int n_slices = (K + kSlice - 1) / kSlice;
  // the blocks of 32 k that this block works on, chain by chain: whole slices, and of the last one the blocks that hold a k
  const int last_blocks = (K - (n_slices - 1) * kSlice + kBK - 1) / kBK;
  auto chain_blocks = [&](int j) {
    return j >= n_slices ? 0 : ((n_slices - 1 - j) / kChains + 1) * (kSlice / kBK) -
                                   (j == (n_slices - 1) % kChains ? kSlice / kBK - last_blocks : 0);
  };
  int total_blocks = 0;
  for (int j = chain0; j < chain0 + n_chains; ++j) total_blocks += chain_blocks(j);

  // ---- loading, T::kStages - 1 blocks early. A thread brings piece tid % 8 of the rows tid / 8 + kStep p: rows of A first,
  // then of W. What is left of each piece is an address and a copy, where its rows and its 32 k are all there; looking at every
  // piece's row and k took two instructions for every three of the products.
  constexpr int kStep = T::kThreads / (kBK / 4), kPiecesA = T::BM / kStep, kPiecesW = T::BN / kStep;
  static_assert(T::BM % kStep == 0 && T::BN % kStep == 0, "a piece's row is one of A's or one of W's for all threads");
  const int ld_row = tid / (kBK / 4), ld_c = tid % (kBK / 4) * 4;
  const bool rows_there = m0 + T::BM <= M && n0 + T::BN <= N;
  // how many of this thread's rows there are (they come in order), and its first ones
  const int a_there = M - m0 - ld_row, w_there = N - n0 - ld_row;        // row p is there if p * kStep is below
  const float* a_src = A + (size_t)(a_there > 0 ? m0 + ld_row : 0) * lda + ld_c;
  const float* w_src = W + (size_t)(w_there > 0 ? n0 + ld_row : 0) * ldw + ld_c;
  int ld_chain = chain0, ld_slice = chain0, ld_sub = 0, ld_count = 0, ld_stage = 0;
  auto load_next = [&]() {
    if (ld_count < total_blocks) {
      while (ld_slice >= n_slices) { ++ld_chain; ld_slice = ld_chain; }
      const int k0 = ld_slice * kSlice + ld_sub * kBK;
      float* st = ring + ld_stage * T::kStageFloats + ld_row * kStride + ld_c;
      const unsigned dst = (unsigned)__cvta_generic_to_shared(st);
      if (VEC) {
        const int bytes = min(max(K - k0 - ld_c, 0), 4) * 4;       // of each piece; the rest reads zeros
        const float* a = a_src + k0;
        const float* w = w_src + k0;
        if (rows_there && k0 + kBK <= K) {
#pragma unroll
          for (int p = 0; p < kPiecesA; ++p)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + p * kStep * kStride * 4),
                         "l"(a + (size_t)p * kStep * lda) : "memory");
#pragma unroll
          for (int p = 0; p < kPiecesW; ++p)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + (T::BM + p * kStep) * kStride * 4),
                         "l"(w + (size_t)p * kStep * ldw) : "memory");
        } else {
#pragma unroll
          for (int p = 0; p < kPiecesA; ++p) {
            const bool in = bytes && p * kStep < a_there;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst + p * kStep * kStride * 4),
                         "l"(in ? a + (size_t)p * kStep * lda : A), "r"(in ? bytes : 0) : "memory");
          }
#pragma unroll
          for (int p = 0; p < kPiecesW; ++p) {
            const bool in = bytes && p * kStep < w_there;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst + (T::BM + p * kStep) * kStride * 4),
                         "l"(in ? w + (size_t)p * kStep * ldw : W), "r"(in ? bytes : 0) : "memory");
          }
        }
      } else {
#pragma unroll 1
        for (int p = 0; p < kPiecesA + kPiecesW; ++p) {
          const bool is_a = p < kPiecesA;
          const int g = is_a ? m0 + ld_row + p * kStep : n0 + ld_row + (p - kPiecesA) * kStep;
          const bool in = g < (is_a ? M : N);
          const float* base = is_a ? A : W;
          copy4<VEC>(st + p * kStep * kStride, base + (size_t)(in ? g : 0) * (is_a ? lda : ldw) + k0 + ld_c, base,
                     in ? K - k0 - ld_c : 0);
        }
      }
      if (++ld_sub == (ld_slice == n_slices - 1 ? last_blocks : kSlice / kBK)) { ld_sub = 0; ld_slice += kChains; }
      ld_stage = ld_stage == T::kStages - 1 ? 0 : ld_stage + 1;
      ++ld_count;
    }
    copy_commit();
  };

  float2 acc[8][8];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[i][j] = make_float2(0.f, 0.f);

#pragma unroll
  for (int s = 0; s < T::kStages - 1; ++s) load_next();

  int chain = chain0, stage = 0;
  bool first = true;
  for (int c = 0; c < n_chains; ++c, ++chain) {
    const int blocks = chain_blocks(chain);
    for (int b = 0; b < blocks; ++b) {
      copy_wait<T::kStages - 2>();
      __syncthreads();
      load_next();
      const float* st = ring + stage * T::kStageFloats;
      stage = stage == T::kStages - 1 ? 0 : stage + 1;
#pragma unroll
      for (int k4 = 0; k4 < kBK / 4; ++k4) {
        float4 w[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) w[j] = *reinterpret_cast<const float4*>(st + (row_w + 8 * j) * kStride + 4 * k4);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float4 a = *reinterpret_cast<const float4*>(st + (row_a + 4 * i) * kStride + 4 * k4);
#pragma unroll
          for (int j = 0; j < 8; ++j) fma2(acc[i][j], make_float2(a.x, a.y), make_float2(w[j].x, w[j].y));
#pragma unroll
          for (int j = 0; j < 8; ++j) fma2(acc[i][j], make_float2(a.z, a.w), make_float2(w[j].z, w[j].w));
        }
      }
    }
    if (c == n_chains - 1) break;
    // the chain's sums: the first chain's as they are, later ones added to what is held; a rank > 0 has two chains at
    // most and holds the first apart from the last
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        float4* slot = held + (2 * i + h) * T::kThreads + tid;
        float4 v = first ? make_float4(0.f, 0.f, 0.f, 0.f) : *slot;
        float* e = &v.x;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          float2& s = acc[i][4 * h + q];
          e[q] = first ? s.x + s.y : e[q] + (s.x + s.y);
          s = make_float2(0.f, 0.f);
        }
        *slot = v;
      }
    first = false;
  }
  copy_wait<0>();

  if (split == 1) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int m = m0 + (warp / WN) * 32 + (lane >> 3) + 4 * i;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const float4 v = held[(2 * i + h) * T::kThreads + tid];
        const float e[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int j = 4 * h + q, n = n0 + (warp % WN) * 64 + (lane & 7) + 8 * j;
          if (m < M && n < N) C[(size_t)m * ldc + n] = e[q] + (acc[i][j].x + acc[i][j].y);
        }
      }
    }
    return;
  }
  // ---- a cluster shares the tile: the last chain's sums lie in the ring (rank 0 with two chains adds them to what it
  // holds), then every rank adds up its share of the slots over the ranks, in chain order
  __syncthreads();
  float4* last = smem4;
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int slot = (2 * i + h) * T::kThreads + tid;
      float e[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) e[q] = acc[i][4 * h + q].x + acc[i][4 * h + q].y;
      if (rank == 0 && n_chains > 1) {
        const float4 v = held[slot];
        e[0] = v.x + e[0]; e[1] = v.y + e[1]; e[2] = v.z + e[2]; e[3] = v.w + e[3];
      }
      last[slot] = make_float4(e[0], e[1], e[2], e[3]);
    }
  cluster_barrier();
  for (int s = rank; s < 16; s += split) {
    const int slot = s * T::kThreads + tid;
    float4 v = read_peer(last + slot, 0);
    for (int r = 1; r < split; ++r) {
      if (n_chains > 1) {
        const float4 p = read_peer(held + slot, r);
        v.x += p.x; v.y += p.y; v.z += p.z; v.w += p.w;
      }
      const float4 p = read_peer(last + slot, r);
      v.x += p.x; v.y += p.y; v.z += p.z; v.w += p.w;
    }
    const int m = m0 + (warp / WN) * 32 + (lane >> 3) + 4 * (s >> 1);
    const float e[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int n = n0 + (warp % WN) * 64 + (lane & 7) + 8 * (4 * (s & 1) + q);
      if (m < M && n < N) C[(size_t)m * ldc + n] = e[q];
    }
  }
  cluster_barrier();          // nobody leaves while its shared memory is being read
}

// ---------------------------------------------------------------------------------------------------------------
// Up to kFewRows rows: the weights stream through shared memory once. A thread is RW weight rows of one chain, a warp
// 4 RW rows x 8 chains; a stage brings RUN k of every chain's current slice for the block's weight rows and for all MT
// rows of A. Runs lie RUN + 4 floats apart, so a 16-byte access of 8 chains falls on all banks.
constexpr int kFewRows = 16;

template <int MT, int WARPS, int RW, int STAGES, int RUN> struct Few {
  static constexpr int kRows = 4 * RW * WARPS, kThreads = 32 * WARPS;
  static constexpr int kRunStride = RUN + 4;
  static constexpr int kStageFloats = (kRows + MT) * kChains * kRunStride;
  static constexpr int smem_bytes() { return 4 * STAGES * kStageFloats; }
};

template <int MT, int WARPS, int RW, int STAGES, int RUN, bool VEC>
__global__ void __launch_bounds__(32 * WARPS)
gemm_f32_few_kernel(const float* A, const float* W, float* __restrict__ C, int M, int N,
                    int K, int lda, int ldw, int ldc) {
  using F = Few<MT, WARPS, RW, STAGES, RUN>;
  constexpr int kRunStride = F::kRunStride;
  extern __shared__ float4 smem4[];
  float* ring = reinterpret_cast<float*>(smem4);
  pdl_wait();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int chain = lane & 7, row = warp * 4 * RW + (lane >> 3);
  const int n0 = blockIdx.x * F::kRows;
  const int n_slices = (K + kSlice - 1) / kSlice;
  constexpr int kPerSlice = kSlice / RUN;
  // rounds of a slice a chain; of the last round the runs that hold a k
  const int rounds = (n_slices + kChains - 1) / kChains;
  const int steps = (rounds - 1) * kPerSlice + (min(K - (rounds - 1) * kChains * kSlice, kSlice) + RUN - 1) / RUN;

  auto load = [&](int t) {
    if (t < steps) {
      float* st = ring + (t % STAGES) * F::kStageFloats;
      constexpr int kPieces = (F::kRows + MT) * kChains * (RUN / 4);
#pragma unroll
      for (int p = 0; p < (kPieces + F::kThreads - 1) / F::kThreads; ++p) {
        const int idx = tid + p * F::kThreads;
        if (kPieces % F::kThreads && idx >= kPieces) break;
        const int piece = idx % (RUN / 4), c = idx / (RUN / 4) % kChains, r = idx / (RUN / 4 * kChains);
        const int k = ((t / kPerSlice) * kChains + c) * kSlice + (t % kPerSlice) * RUN + piece * 4;
        const bool is_w = r < F::kRows;
        const int g = is_w ? n0 + r : r - F::kRows;
        const bool in = g < (is_w ? N : M);
        const float* base = is_w ? W : A;
        copy4<VEC>(st + (r * kChains + c) * kRunStride + piece * 4, base + (size_t)(in ? g : 0) * (is_w ? ldw : lda) + k,
                   base, in ? K - k : 0);
      }
    }
    copy_commit();
  };
#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s) load(s);

  float2 acc[RW][MT];
#pragma unroll
  for (int i = 0; i < RW; ++i)
#pragma unroll
    for (int m = 0; m < MT; ++m) acc[i][m] = make_float2(0.f, 0.f);
  for (int t = 0; t < steps; ++t) {
    copy_wait<STAGES - 2>();
    __syncthreads();
    load(t + STAGES - 1);
    const float* st = ring + (t % STAGES) * F::kStageFloats;
    const float* wr = st + (row * kChains + chain) * kRunStride;
    const float* ar = st + (F::kRows * kChains + chain) * kRunStride;
    constexpr int kTogether = MT * RW <= 4 ? 4 : (MT <= 8 ? 2 : 1);     // 16-byte pieces read before they are used
#pragma unroll
    for (int q0 = 0; q0 < RUN / 4; q0 += kTogether) {
      float4 w[kTogether][RW], a[kTogether][MT];
#pragma unroll
      for (int q = 0; q < kTogether; ++q) {
#pragma unroll
        for (int i = 0; i < RW; ++i)
          w[q][i] = *reinterpret_cast<const float4*>(wr + 4 * i * kChains * kRunStride + 4 * (q0 + q));
#pragma unroll
        for (int m = 0; m < MT; ++m) a[q][m] = *reinterpret_cast<const float4*>(ar + m * kChains * kRunStride + 4 * (q0 + q));
      }
#pragma unroll
      for (int q = 0; q < kTogether; ++q) {
#pragma unroll
        for (int i = 0; i < RW; ++i)
#pragma unroll
          for (int m = 0; m < MT; ++m) fma2(acc[i][m], make_float2(a[q][m].x, a[q][m].y), make_float2(w[q][i].x, w[q][i].y));
#pragma unroll
        for (int i = 0; i < RW; ++i)
#pragma unroll
          for (int m = 0; m < MT; ++m) fma2(acc[i][m], make_float2(a[q][m].z, a[q][m].w), make_float2(w[q][i].z, w[q][i].w));
      }
    }
  }
  copy_wait<0>();
#pragma unroll
  for (int i = 0; i < RW; ++i) {
    const int n = n0 + row + 4 * i;
#pragma unroll
    for (int m = 0; m < MT; ++m) {
      const float p = acc[i][m].x + acc[i][m].y;
      float sum = __shfl_sync(0xffffffffu, p, lane & 24);
#pragma unroll
      for (int c = 1; c < kChains; ++c) sum += __shfl_sync(0xffffffffu, p, (lane & 24) + c);
      if (chain == (m & 7) && m < M && n < N) C[(size_t)m * ldc + n] = sum;
    }
  }
}

template <int WM, int WN, bool VEC>
static int launch_tile(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldw, int ldc, int split,
                       cudaStream_t stream) {
  using T = Tile<WM, WN>;
  const int tiles_n = (N + T::BN - 1) / T::BN, tiles_m = (M + T::BM - 1) / T::BM;
  if (tiles_m > 65535) return LLMIE_ERR_UNSUPPORTED_SIZE;
  auto kernel = gemm_f32_tile_kernel<WM, WN, VEC>;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, T::smem_bytes());
  if (e != cudaSuccess) return (int)e;
  if (split == 1)
    launch_k(kernel, dim3(tiles_n, tiles_m), dim3(T::kThreads), T::smem_bytes(), stream, A, W, C, M, N, K, lda, ldw, ldc, 1);
  else
    launch_k_cluster(kernel, dim3(tiles_n * split, tiles_m), dim3(T::kThreads), T::smem_bytes(), stream, (unsigned)split, A,
                     W, C, M, N, K, lda, ldw, ldc, split);
  LLMIE_LAUNCH_CHECK();
  return LLMIE_OK;
}

template <int MT, int WARPS, int RW, int STAGES, int RUN, bool VEC>
static int launch_few(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldw, int ldc,
                      cudaStream_t stream) {
  using F = Few<MT, WARPS, RW, STAGES, RUN>;
  static_assert(F::smem_bytes() <= 227 * 1024, "a block's stages fit its shared memory");
  auto kernel = gemm_f32_few_kernel<MT, WARPS, RW, STAGES, RUN, VEC>;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, F::smem_bytes());
  if (e != cudaSuccess) return (int)e;
  launch_k(kernel, dim3((N + F::kRows - 1) / F::kRows), dim3(F::kThreads), F::smem_bytes(), stream, A, W, C, M, N, K, lda,
           ldw, ldc);
  LLMIE_LAUNCH_CHECK();
  return LLMIE_OK;
}

// The kernels by form: kernel * 10 + blocks that share a tile's chains. 10, 20, 30: up to kFewRows rows. 5x: tiles of 32 x
// 128, 6x: of 64 x 64.
template <bool VEC>
static int dispatch(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldw, int ldc, int form,
                    cudaStream_t stream) {
#define LLMIE_FEW(MAX, MT, WARPS, RW, STAGES, RUN) \
  if (M <= MAX) return launch_few<MT, WARPS, RW, STAGES, RUN, VEC>(A, W, C, M, N, K, lda, ldw, ldc, stream);
  switch (form) {
    case 10:
      LLMIE_FEW(1, 1, 2, 1, 6, 32) LLMIE_FEW(2, 2, 2, 1, 6, 32) LLMIE_FEW(4, 4, 2, 1, 6, 32) LLMIE_FEW(8, 8, 2, 1, 6, 32)
      break;
    case 20:
      LLMIE_FEW(1, 1, 2, 2, 3, 32) LLMIE_FEW(2, 2, 2, 2, 3, 32) LLMIE_FEW(4, 4, 2, 2, 3, 32) LLMIE_FEW(16, 16, 2, 2, 3, 32)
      break;
    case 30:
      LLMIE_FEW(8, 8, 4, 2, 4, 16) LLMIE_FEW(16, 16, 4, 2, 3, 16)
      break;
    case 51: case 54: case 58: return launch_tile<1, 2, VEC>(A, W, C, M, N, K, lda, ldw, ldc, form - 50, stream);
    case 61: case 64: case 68: return launch_tile<2, 1, VEC>(A, W, C, M, N, K, lda, ldw, ldc, form - 60, stream);
    default: return LLMIE_ERR_BAD_ARG;
  }
#undef LLMIE_FEW
  return LLMIE_ERR_UNSUPPORTED_SIZE;
}

// Which form serves which size; microseconds measured with weights beyond L2 (N x K: rows).
// Few rows: 8 weight rows a block and six stages where that gives no SM more than two blocks (2,048 x 8,192, 1 / 8 rows:
// 18 / 35, form 20 26 / 44); 16 weight rows a block above (16,384 x 2,048, 1 / 3 rows: 26 / 30, form 10 29 / 42), and 32
// from 5 rows on, where a thread's reads of A cost more than its weights (16,384 x 2,048, 8 / 13 rows: 38 / 60, form 20
// 49 / 76) or all lanes have little to do (2,048 x 48, 16 rows: 5.0, form 20 6.5). A K of little more than a slice leaves
// most lanes idle there, and from 9 rows on wide outputs take tiles instead (8,192 x 64 / 128 / 160, 16 rows: 8.3 / 11.5 /
// 13.3, form 30 9.6 / 16.2 / 16.2).
// Tiles: 32 rows high up to 32 rows (16,384 x 2,048, 20 rows: 74, 64 high 115), else 64 x 64 (301 rows: 79, 32 x 128 89).
//
// How many blocks share a tile's chains: from 16 slices on, 8 until the tiles alone fill the GPU's 592 places (2,048 x 8,192,
// 301 rows: 275, 4 blocks 320, 1 block 463), 4 until they fill them three times and more (16,384 x 2,048, 301 rows: 499, 8
// 507, 1 516), then one (16,384 x 2,048, 512 rows: 723, 4 blocks 776). Up to 32 rows 8.
// With fewer slices some ranks would have one chain or none, and it follows from what a slice costs a block: 7 us while an SM
// holds one or two blocks (a warp on each quarter), 10.5 with three, 14 with four, which is all that fit; clusters do not
// spread as evenly (14 with three), ranks without a chain hold their places all the same, and every round of clusters costs 2
// us. That sum picks within 20 % of the best of the three forms at 1 to 12 slices and 1 to 4,000 tiles (2,048 x 256, 2,100
// rows: 8 blocks 209, 4 208, 1 64; 2,048 x 512, 128 rows: 18, 21, 32; one plain 64 x 64 tile a block: 122 and 78; from 16
// slices on it is up to 10 % off the rule above).
static float tile_time(long long tiles, int slices, int split) {
  constexpr int kSms = 148, kPlaces = 4 * kSms;
  const long long blocks = tiles * split, full = blocks / kPlaces, rest = blocks % kPlaces;
  const int on_sm = (int)((rest + kSms - 1) / kSms);                          // blocks an SM holds in the last round
  const float last = rest == 0 ? 0.f : (on_sm <= 2 ? 7.f : (split > 1 ? 14.f : 3.5f * on_sm));
  // slices of the busiest rank: it has the first 8 / split chains
  int busiest = 0;
  for (int j = 0; j < kChains / split; ++j) busiest += slices > j ? (slices - 1 - j) / kChains + 1 : 0;
  return (full * 14.f + last) * busiest + (split > 1 ? 2.f * (full + (rest != 0)) : 0.f);
}

static int choose_form(int M, int N, int K) {
  const int slices = (K + kSlice - 1) / kSlice;
  if (M <= kFewRows && !(M > 8 && K > 32 && K <= 192 && N > 2 * 16 * 148)) {
    const bool narrow = N <= 2 * 8 * 148;
    if (narrow) return M <= 8 ? 10 : (K <= 64 ? 30 : 20);
    return M <= 4 ? 20 : 30;
  }
  const bool low = M > kFewRows && M <= 32;
  const long long tiles = low ? (N + 127) / 128 : (long long)((M + 63) / 64) * ((N + 63) / 64);
  if (slices >= 2 * kChains) return low ? 58 : (tiles < 640 ? 68 : (tiles < 1900 ? 64 : 61));
  int best = 1;
  for (int split = 4; split <= kChains; split *= 2)
    if (tile_time(tiles, slices, split) < tile_time(tiles, slices, best)) best = split;
  return (low ? 50 : 60) + best;
}

}  // namespace llmie

using namespace llmie;

// form 0: chosen by size; the others are for tests (every form that takes a size gives the same bits).
extern "C" int llmie_gemm_f32_nt_form(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldw,
                                      int ldc, int form, cudaStream_t stream) {
  if (M < 0 || N <= 0 || K <= 0 || lda < K || ldw < K || ldc < N) return LLMIE_ERR_BAD_ARG;
  if (M == 0) return LLMIE_OK;
  if (form == 0) form = choose_form(M, N, K);
  const bool vec = aligned16(A) && aligned16(W) && lda % 4 == 0 && ldw % 4 == 0;
  return vec ? dispatch<true>(A, W, C, M, N, K, lda, ldw, ldc, form, stream)
             : dispatch<false>(A, W, C, M, N, K, lda, ldw, ldc, form, stream);
}

extern "C" int llmie_gemm_f32_nt(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldw,
                                 int ldc, cudaStream_t stream) {
  return llmie_gemm_f32_nt_form(A, W, C, M, N, K, lda, ldw, ldc, 0, stream);
}
