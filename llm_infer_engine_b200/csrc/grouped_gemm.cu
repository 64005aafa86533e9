// Many small matrix products in one launch: C_g = A_g W_g^T for groups g that share a shape but not their
// weights. Two ways to say which rows belong to which group:
//
//   batched   every group has the same M rows; group g reads columns [g * a_gcs, g * a_gcs + K) of A's rows and
//             writes columns [g * c_gcs, g * c_gcs + N) of C's rows (the heads of an attention layer, each with a
//             matrix of its own); grid.z = groups.
//   routed    rows were sorted by group into tiles of BM positions (`tile_group[tile]` = the group of a tile, -1 =
//             unused tile; `a_rows[pos]` = the row of A at a sorted position, -1 = padding; `c_rows[pos]` = the row of
//             C it writes): the experts of a routed feed-forward. Positions without an indirection are their own row.
//
// W is [groups][N (or 2 N), K], K contiguous. With DUAL the weight of a group is [gate rows | up rows] and the result
// is act(A gate^T) * (A up^T). float32 inputs: one FMA per k in the order k = 0..K-1 whatever the tile or the batch (no
// tensor cores, no reduced precision), so a row's result does not depend on what else is in the launch. bfloat16 inputs:
// the tensor-core kernel further down, float32 accumulators.
#include "common.cuh"

namespace llmie {

struct GroupedArgs {
  const void* A; long long lda; long long a_gcs;
  const int* a_rows;
  const void* W; long long w_gs; long long ldw;
  void* C; long long ldc; long long c_gcs;
  const int* c_rows;
  const int* tile_group;
  int M, N, K, act;
};

constexpr int kGK = 16;

template <typename TA, typename TC, int BM, int BN, int TM, int TN, bool DUAL>
__global__ void __launch_bounds__((BM / TM) * (BN / TN))
grouped_gemm_kernel(const GroupedArgs p) {
  constexpr int kThreads = (BM / TM) * (BN / TN);
  __shared__ float As[kGK][BM + 4];
  __shared__ float Ws[DUAL ? 2 : 1][kGK][BN + 4];
  __shared__ int rowA[BM], rowC[BM];
  pdl_launch_dependents();
  pdl_wait();
  const int tid = threadIdx.x;
  const int tile = blockIdx.y;
  int group = blockIdx.z;
  if (p.tile_group) {
    group = p.tile_group[tile];
    if (group < 0) return;
  }
  const int m0 = tile * BM, n0 = blockIdx.x * BN;
  for (int r = tid; r < BM; r += kThreads) {
    const int pos = m0 + r;
    int ra = -1, rc = -1;
    if (pos < p.M) {
      ra = p.a_rows ? p.a_rows[pos] : pos;
      rc = p.c_rows ? p.c_rows[pos] : pos;
      if (ra < 0 || rc < 0) ra = rc = -1;
    }
    rowA[r] = ra;
    rowC[r] = rc;
  }
  __syncthreads();
  const TA* A = reinterpret_cast<const TA*>(p.A) + (size_t)group * p.a_gcs;
  const TA* W = reinterpret_cast<const TA*>(p.W) + (size_t)group * p.w_gs;
  const int tx = tid % (BN / TN), ty = tid / (BN / TN);
  float acc[DUAL ? 2 : 1][TM][TN];
#pragma unroll
  for (int s = 0; s < (DUAL ? 2 : 1); ++s)
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
      for (int j = 0; j < TN; ++j) acc[s][i][j] = 0.f;

  for (int k0 = 0; k0 < p.K; k0 += kGK) {
    for (int idx = tid; idx < BM * kGK; idx += kThreads) {
      const int r = idx / kGK, c = idx % kGK;
      const int ra = rowA[r], gk = k0 + c;
      As[c][r] = (ra >= 0 && gk < p.K) ? to_f32(A[(size_t)ra * p.lda + gk]) : 0.f;
    }
    for (int idx = tid; idx < BN * kGK; idx += kThreads) {
      const int r = idx / kGK, c = idx % kGK;
      const int gn = n0 + r, gk = k0 + c;
      const bool ok = gn < p.N && gk < p.K;
      Ws[0][c][r] = ok ? to_f32(W[(size_t)gn * p.ldw + gk]) : 0.f;
      if (DUAL) Ws[DUAL ? 1 : 0][c][r] = ok ? to_f32(W[(size_t)(gn + p.N) * p.ldw + gk]) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < kGK; ++kk) {
      float a[TM], w[TN];
#pragma unroll
      for (int i = 0; i < TM; ++i) a[i] = As[kk][ty * TM + i];
#pragma unroll
      for (int s = 0; s < (DUAL ? 2 : 1); ++s) {
#pragma unroll
        for (int j = 0; j < TN; ++j) w[j] = Ws[s][kk][tx * TN + j];
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
          for (int j = 0; j < TN; ++j) acc[s][i][j] = fmaf(a[i], w[j], acc[s][i][j]);
      }
    }
    __syncthreads();
  }
  TC* C = reinterpret_cast<TC*>(p.C) + (size_t)group * p.c_gcs;
#pragma unroll
  for (int i = 0; i < TM; ++i) {
    const int rc = rowC[ty * TM + i];
    if (rc < 0) continue;
#pragma unroll
    for (int j = 0; j < TN; ++j) {
      const int gn = n0 + tx * TN + j;
      if (gn >= p.N) continue;
      float v = acc[0][i][j];
      if (DUAL) {
        // the gate is rounded to the activation type before the activation, as a separate product would leave it
        const float g = to_f32(from_f32<TC>(v)), u = to_f32(from_f32<TC>(acc[DUAL ? 1 : 0][i][j]));
        v = apply_act(g, p.act) * u;
      } else if (p.act) {
        v = apply_act(to_f32(from_f32<TC>(v)), p.act);      // a single product with its activation
      }
      C[(size_t)rc * p.ldc + gn] = from_f32<TC>(v);
    }
  }
}

// ------------------------------------------------------------------------------------------
// The same products for bfloat16 inputs on the tensor cores (mma.sync m16n8k16, float32 accumulators): tiles of BM x 64
// outputs (64 gate and 64 up columns with DUAL), four warps that share out the columns. A row's sums depend on that row
// and the weights alone (the rows of an mma are independent, and every tile height adds up k in the same order), so here
// too a result does not depend on what else is in the launch.
//
// With a few rows a group (the experts of a batched one-token step) the weights' stream is what bounds it, with many rows
// and a short K (the heads of a latent attention layer) the rows' way in and out. So: K steps of 64 arrive in a ring of
// asynchronous copies, 16 bytes each, kStages - 1 steps ahead (two, or four for 16 rows of one matrix); fragments come by
// ldmatrix from rows of 128 bytes whose eight pieces are exchanged by the row's number (no two rows of an 8 x 8 block share a
// bank); only the 16-row slices of a tile that hold rows are multiplied; and results leave through shared memory in whole
// rows.
// `vec`: K, the leading dimensions and the group strides are multiples of 8 elements and the bases 16-byte aligned;
// otherwise the tiles are brought element by element. `cvec`: the same of C, for 16-byte stores.
__device__ __forceinline__ void gg_mma(float (&c)[4], const unsigned (&a)[4], unsigned b0, unsigned b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void gg_ldmatrix(unsigned (&r)[4], unsigned addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr));
}

constexpr int kMmaBK = 64, kMmaBN = 64;

template <int BM, bool DUAL>
struct MmaTile {
  static constexpr int kRows = BM + (DUAL ? 2 : 1) * kMmaBN;            // rows of 128 bytes a stage holds
  static constexpr int kStageBytes = kRows * 2 * kMmaBK;
  // 16 rows: gate and up together in 3 stages, four blocks an SM, so that 16 experts' 512 blocks are all resident (2,048 x
  // 2 x 2,048, 24 to 64 rows: 50 us of 41 for the weights; 5 stages, two blocks an SM, 63); one matrix in 5 (26 us of
  // 20.5; 3 stages 35: what is in flight counts). 64 rows: 3 stages (2: 10 to 30 % slower; the same 40 rows 82 / 40 us).
  static constexpr int kStages = BM == 16 && !DUAL ? 5 : 3;
  static constexpr int kOutPitch = kMmaBN + 4;                          // floats between two rows on their way out
  static constexpr int kOutBytes = BM * kOutPitch * 4;
  // a K of fewer steps leaves the ring's other stages out: 1,805 rows of 32 heads, 64 -> 256 (one step): six blocks an SM
  // instead of four, 22.7 us instead of 26.7
  static int smem_bytes(int steps) {
    const int ring = (steps < kStages ? steps : kStages) * kStageBytes;
    return ring > kOutBytes ? ring : kOutBytes;
  }
};

// Short products of full tiles wait for their loads, and registers set how many blocks wait at once: eight blocks an SM
// (64 registers, nothing spilled) instead of six (78) take a latent-attention layer over 1,805 rows, with two products a
// head, from 163.9 to 162.0 us. Longer rings and pairs of weights are held by shared memory instead.
template <typename TC, int BM, bool DUAL>
__global__ void __launch_bounds__(128, BM == 64 && !DUAL ? 8 : 1)
grouped_gemm_mma_kernel(const GroupedArgs p, const int vec, const int cvec) {
  using T = MmaTile<BM, DUAL>;
  constexpr int NW = DUAL ? 2 : 1, kSlices = BM / 16, BK = kMmaBK, BN = kMmaBN;
  extern __shared__ __align__(128) unsigned char gg_smem[];
  __shared__ int rowA[BM], rowC[BM];
  pdl_launch_dependents();
  pdl_wait();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int tile = blockIdx.y;
  int group = blockIdx.z;
  if (p.tile_group) {
    group = p.tile_group[tile];
    if (group < 0) return;
  }
  const int m0 = tile * BM, n0 = blockIdx.x * BN;
  int last_row = 0;
  for (int r = tid; r < BM; r += 128) {
    const int pos = m0 + r;
    int ra = -1, rc = -1;
    if (pos < p.M) {
      ra = p.a_rows ? p.a_rows[pos] : pos;
      rc = p.c_rows ? p.c_rows[pos] : pos;
      if (ra < 0 || rc < 0) ra = rc = -1;
    }
    rowA[r] = ra;
    rowC[r] = rc;
    if (ra >= 0) last_row = r + 1;
  }
  // slices of 16 rows that hold a row (the positions of a tile are filled from its start; a gap costs time only)
  const int slices = BM == 16 ? 1 : (__syncthreads_or(last_row > 48) ? 4 : __syncthreads_or(last_row > 32) ? 3
                                     : __syncthreads_or(last_row > 16) ? 2 : 1);
  __syncthreads();
  const __nv_bfloat16* A = reinterpret_cast<const __nv_bfloat16*>(p.A) + (size_t)group * p.a_gcs;
  const __nv_bfloat16* W = reinterpret_cast<const __nv_bfloat16*>(p.W) + (size_t)group * p.w_gs;
  const unsigned base = (unsigned)__cvta_generic_to_shared(gg_smem);
  const int steps = (p.K + BK - 1) / BK;

  // a thread brings piece tid % 8 of the stage's rows tid / 8 + 16 j
  auto load = [&](int s) {
    if (s < steps) {
      const int k = s * BK + (tid & 7) * 8;
      const unsigned stage = base + (s % T::kStages) * T::kStageBytes;
#pragma unroll
      for (int j = 0; j < T::kRows / 16; ++j) {
        const int r = (tid >> 3) + 16 * j;
        if (r < BM && r >= 16 * slices) continue;
        const __nv_bfloat16* src = nullptr;
        if (r < BM) {
          if (rowA[r] >= 0) src = A + (size_t)rowA[r] * p.lda;
        } else {
          const int n = n0 + (r - BM) % BN;
          if (n < p.N) src = W + (size_t)(n + ((r - BM) >= BN ? p.N : 0)) * p.ldw;
        }
        const unsigned dst = stage + r * 2 * BK + (((tid & 7) ^ (r & 7)) << 4);
        if (vec) {
          const int bytes = src && k < p.K ? 16 : 0;
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(bytes ? src + k : W), "r"(bytes)
                       : "memory");
        } else {
          alignas(16) __nv_bfloat16 e[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) e[i] = src && k + i < p.K ? src[k + i] : __float2bfloat16_rn(0.f);
          *reinterpret_cast<uint4*>(gg_smem + (dst - base)) = *reinterpret_cast<const uint4*>(e);
        }
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };

  float acc[NW][kSlices][2][4];
#pragma unroll
  for (int s = 0; s < NW; ++s)
#pragma unroll
    for (int i = 0; i < kSlices; ++i)
#pragma unroll
      for (int j = 0; j < 2; ++j) acc[s][i][j][0] = acc[s][i][j][1] = acc[s][i][j][2] = acc[s][i][j][3] = 0.f;
#pragma unroll
  for (int s = 0; s < T::kStages - 1; ++s) load(s);

  // this lane's row within an ldmatrix of A (rows 0-15, then the same rows of the next 8 k) and of W (8 columns, their
  // next 8 k, the next 8 columns, their next 8 k)
  const int a_row = lane & 15, a_k = lane >> 4;
  const int w_row = BM + warp * 16 + (lane & 7) + ((lane >> 4) << 3), w_k = (lane >> 3) & 1;
  for (int s = 0; s < steps; ++s) {
    asm volatile("cp.async.wait_group %0;" ::"n"(T::kStages - 2) : "memory");
    __syncthreads();
    load(s + T::kStages - 1);
    const unsigned stage = base + (s % T::kStages) * T::kStageBytes;
#pragma unroll
    for (int kk = 0; kk < BK / 16; ++kk) {
      unsigned b[NW][4];
#pragma unroll
      for (int q = 0; q < NW; ++q) gg_ldmatrix(b[q], stage + (w_row + q * BN) * 2 * BK + (((2 * kk + w_k) ^ (w_row & 7)) << 4));
#pragma unroll
      for (int i = 0; i < kSlices; ++i) {
        if (i < slices) {
          unsigned a[4];
          gg_ldmatrix(a, stage + (16 * i + a_row) * 2 * BK + (((2 * kk + a_k) ^ (a_row & 7)) << 4));
#pragma unroll
          for (int q = 0; q < NW; ++q) {
            gg_mma(acc[q][i][0], a, b[q][0], b[q][1]);
            gg_mma(acc[q][i][1], a, b[q][2], b[q][3]);
          }
        }
      }
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();

  // out through shared memory (the ring is done with): results as float32, whole rows of 64 columns
  float* out = reinterpret_cast<float*>(gg_smem);
#pragma unroll
  for (int i = 0; i < kSlices; ++i) {
    if (i >= slices) break;
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        float v = acc[0][i][j][e];
        if (DUAL) {
          const float gt = to_f32(from_f32<TC>(v)), up = to_f32(from_f32<TC>(acc[NW - 1][i][j][e]));
          v = apply_act(gt, p.act) * up;
        } else if (p.act) {
          v = apply_act(to_f32(from_f32<TC>(v)), p.act);
        }
        out[(16 * i + (lane >> 2) + 8 * (e >> 1)) * T::kOutPitch + warp * 16 + 8 * j + 2 * (lane & 3) + (e & 1)] = v;
      }
  }
  __syncthreads();
  TC* C = reinterpret_cast<TC*>(p.C) + (size_t)group * p.c_gcs;
  constexpr int kPer = 16 / (int)sizeof(TC), kPieces = BN / kPer;
  for (int idx = tid; idx < 16 * slices * kPieces; idx += 128) {
    const int r = idx / kPieces, c = idx % kPieces * kPer;
    const int rc = rowC[r];
    if (rc < 0 || n0 + c >= p.N) continue;
    const float* v = out + r * T::kOutPitch + c;
    TC* dst = C + (size_t)rc * p.ldc + n0 + c;
    if (cvec && n0 + c + kPer <= p.N) {
      alignas(16) TC e[kPer];
#pragma unroll
      for (int i = 0; i < kPer; ++i) e[i] = from_f32<TC>(v[i]);
      *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<const uint4*>(e);
    } else {
#pragma unroll
      for (int i = 0; i < kPer; ++i)
        if (n0 + c + i < p.N) dst[i] = from_f32<TC>(v[i]);
    }
  }
}

template <typename TC, int BM, bool DUAL>
static int launch_mma_tile(const GroupedArgs& p, dim3 grid, int vec, int cvec, cudaStream_t stream) {
  using T = MmaTile<BM, DUAL>;
  auto kernel = grouped_gemm_mma_kernel<TC, BM, DUAL>;
  const int smem = T::smem_bytes((p.K + kMmaBK - 1) / kMmaBK);
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, T::smem_bytes(T::kStages));
  if (e != cudaSuccess) return (int)e;
  launch_k(kernel, grid, dim3(128), smem, stream, p, vec, cvec);
  return LLMIE_OK;
}

template <typename TC, bool DUAL>
static int launch_grouped_mma(const GroupedArgs& p, int n_tiles, int groups_z, bool small, int vec, cudaStream_t stream) {
  dim3 grid((p.N + kMmaBN - 1) / kMmaBN, n_tiles, groups_z);
  if (grid.y > 65535 || grid.z > 65535) return LLMIE_ERR_UNSUPPORTED_SIZE;
  constexpr int kPer = 16 / (int)sizeof(TC);
  const int cvec = p.ldc % kPer == 0 && p.c_gcs % kPer == 0 && aligned16(p.C);
  return small ? launch_mma_tile<TC, 16, DUAL>(p, grid, vec, cvec, stream)
               : launch_mma_tile<TC, 64, DUAL>(p, grid, vec, cvec, stream);
}

template <typename TA, typename TC, bool DUAL>
static int launch_grouped(const GroupedArgs& p, int n_tiles_small, int n_tiles_big, int groups_z, bool small,
                          cudaStream_t stream) {
  if (small) {
    dim3 grid((p.N + 31) / 32, n_tiles_small, groups_z);
    if (grid.y > 65535 || grid.z > 65535) return LLMIE_ERR_UNSUPPORTED_SIZE;
    launch_k(grouped_gemm_kernel<TA, TC, 16, 32, 2, 2, DUAL>, grid, dim3(128), 0, stream, p);
  } else {
    dim3 grid((p.N + 63) / 64, n_tiles_big, groups_z);
    if (grid.y > 65535 || grid.z > 65535) return LLMIE_ERR_UNSUPPORTED_SIZE;
    launch_k(grouped_gemm_kernel<TA, TC, 64, 64, 4, 4, DUAL>, grid, dim3(256), 0, stream, p);
  }
  return LLMIE_OK;
}

}  // namespace llmie

using namespace llmie;

// Rows per tile of the two forms; the sort that prepares a routed call must use the same number.
extern "C" int llmie_grouped_gemm_tile_rows(int small) { return small ? 16 : 64; }

// A, W of in_dtype; C of out_dtype. `groups` > 0 with tile_group == null: the batched form over M rows. tile_group !=
// null: the routed form over `n_tiles` tiles of sorted positions (M = number of positions, padding included).
// `small` picks tiles of 16 rows (few rows per group) instead of 64. dual: W holds [gate | up], act is applied to the
// gate; without dual a non-zero act is applied to the product itself.
extern "C" int llmie_grouped_gemm_nt(const void* A, long long lda, long long a_gcs, const int* a_rows, const void* W,
                                     long long w_gs, long long ldw, void* C, long long ldc, long long c_gcs,
                                     const int* c_rows, const int* tile_group, int n_tiles, int groups, int M, int N,
                                     int K, int dual, int act, int small, int in_dtype, int out_dtype,
                                     cudaStream_t stream) {
  if (!A || !W || !C || M < 0 || N <= 0 || K <= 0 || lda < 0 || ldw < K || ldc < 0 || act < 0 || act > 4)
    return LLMIE_ERR_BAD_ARG;
  if (!tile_group && groups <= 0) return LLMIE_ERR_BAD_ARG;
  if (tile_group && n_tiles < 0) return LLMIE_ERR_BAD_ARG;
  if ((in_dtype != LLMIE_F32 && in_dtype != LLMIE_BF16) || (out_dtype != LLMIE_F32 && out_dtype != LLMIE_BF16))
    return LLMIE_ERR_DTYPE;
  if (in_dtype == LLMIE_F32 && out_dtype != LLMIE_F32) return LLMIE_ERR_DTYPE;
  if (M == 0 || (tile_group && n_tiles == 0)) return LLMIE_OK;
  GroupedArgs p{A, lda, a_gcs, a_rows, W, w_gs, ldw, C, ldc, c_gcs, c_rows, tile_group, M, N, K, act};
  const int bm = small ? 16 : 64;
  const int tiles = tile_group ? n_tiles : (M + bm - 1) / bm;
  const int gz = tile_group ? 1 : groups;
  int rc;
  if (in_dtype == LLMIE_F32)
    rc = dual ? launch_grouped<float, float, true>(p, tiles, tiles, gz, small, stream)
              : launch_grouped<float, float, false>(p, tiles, tiles, gz, small, stream);
  else {
    const int vec = K % 8 == 0 && lda % 8 == 0 && a_gcs % 8 == 0 && ldw % 8 == 0 && w_gs % 8 == 0 && aligned16(A) &&
                    aligned16(W);
    if (out_dtype == LLMIE_F32)
      rc = dual ? launch_grouped_mma<float, true>(p, tiles, gz, small, vec, stream)
                : launch_grouped_mma<float, false>(p, tiles, gz, small, vec, stream);
    else
      rc = dual ? launch_grouped_mma<__nv_bfloat16, true>(p, tiles, gz, small, vec, stream)
                : launch_grouped_mma<__nv_bfloat16, false>(p, tiles, gz, small, vec, stream);
  }
  if (rc != LLMIE_OK) return rc;
  LLMIE_LAUNCH_CHECK();
  return LLMIE_OK;
}
