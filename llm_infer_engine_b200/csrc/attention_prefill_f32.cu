// Causal attention for prompts of the float32 path, over the paged cache: FMA on the CUDA cores, float32 throughout, no
// tensor cores. Scores q.k * scale, online softmax with float32 running maximum, sum and accumulator (the math of the plain
// kernel in attention_simt.cu, a warp per (token, head), which keeps the options and sizes this one does not take).
//
// One block = 16 RI query tokens of one sequence and head, 128 threads; a warp owns 4 RI rows and works through its rows'
// keys a cache page (64 keys) at a time, so that a page is fetched once for all rows (the plain kernel fetches it once for
// every row, 4 bytes at a time for the values). Lanes lie as 4 rows x 8 columns; a thread has RI rows (lane / 8 + 4 i) and
// of the page's keys the columns lane % 8 + 8 j, of the output the columns 4 (lane % 8) + 32 j.
//   S = Q K^T   packed FMAs (fma.rn.f32x2) over pairs of the head size, rows of Q and K 16 bytes apart on different banks
//   softmax     eight lanes a row; P to shared memory, read back by the same warp only
//   O += P V    packed FMAs over pairs of output columns, keys in order
// K of the next page is fetched while P V runs, V while the next scores do. The order of a row's sums does not depend on RI
// or on the rows beside it. Keys that a row may not see have weight 0; so that a value that is not finite does not reach
// the rows in front of it, pages that the causal line or the window's end crosses are looked at for such values first, and
// keys beyond the sequence's last are never read.
//
// What bounds it: three blocks of four warps an SM (168 registers, 68 KB), which wait for dependent instructions and for one
// another at the pages' barriers (22 % of the issue rate, 21 % of the FMA pipes, 16 % of shared memory). Prompts of 217, 118
// and 130 tokens, 32 heads of 64: 185 us with the plain kernel, 57 us so.
#include "common.cuh"
#include <math.h>

namespace llmie {

constexpr int kPfKeys = 64, kPfThreads = 128, kPfPitch = kPfKeys + 4;

struct PrefillF32Args {
  const float* q;
  const float* k_cache;
  const float* v_cache;
  float* out;
  const int* cu_q;
  const int* seq_slot;
  const int* seq_start;
  const int* block_table;
  int max_pages, n_q, n_kv, window;
  float scale;
};

__device__ __forceinline__ void pf_fma2(float2& acc, const float2& a, const float2& b) {
  unsigned long long& c = reinterpret_cast<unsigned long long&>(acc);
  asm("fma.rn.f32x2 %0, %1, %2, %0;"
      : "+l"(c)
      : "l"(reinterpret_cast<const unsigned long long&>(a)), "l"(reinterpret_cast<const unsigned long long&>(b)));
}
__device__ __forceinline__ void pf_copy16(float* dst, const float* src, bool there) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src),
               "r"(there ? 16 : 0)
               : "memory");
}

template <int HD, int RI> struct PrefillF32 {
  static constexpr int kRows = 16 * RI, kKPitch = HD + 4;
  static constexpr int kFloats = kRows * kKPitch + kPfKeys * kKPitch + kPfKeys * HD + kRows * kPfPitch;
  static constexpr int smem_bytes() { return 4 * kFloats; }
};

// three blocks an SM at head size 64 (68 KB each): 168 registers a thread
template <int HD, int RI>
__global__ void __launch_bounds__(kPfThreads, HD == 64 ? 3 : 1)
attention_prefill_f32_kernel(const PrefillF32Args p) {
  using C = PrefillF32<HD, RI>;
  extern __shared__ __align__(16) float pf_smem[];
  float* Qs = pf_smem;
  float* Ks = Qs + C::kRows * C::kKPitch;
  float* Vs = Ks + kPfKeys * C::kKPitch;
  float* Ps = Vs + kPfKeys * HD;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int head = blockIdx.x, seq = blockIdx.z;
  const int q_begin = p.cu_q[seq], q_len = p.cu_q[seq + 1] - q_begin;
  const int t0 = (gridDim.y - 1 - blockIdx.y) * C::kRows;       // late tiles see the most keys: they start first
  if (t0 >= q_len) return;
  const int start = p.seq_start[seq], hk = head / (p.n_q / p.n_kv);
  const int rows_here = min(C::kRows, q_len - t0);
  const int last_key = start + t0 + rows_here - 1;
  const int page_lo = first_visible_key(start + t0, p.window) / kPfKeys, page_hi = last_key / kPfKeys;
  const int last_lo = first_visible_key(last_key, p.window);
  const int* pages = p.block_table + (size_t)p.seq_slot[seq] * p.max_pages;

  constexpr int kChunks = HD / 4;
  auto load_page = [&](const float* cache, float* dst, int pitch, int pg) {
    const float* src = cache + ((size_t)pages[pg] * p.n_kv + hk) * kPfKeys * HD;
    const int n = last_key - pg * kPfKeys + 1;                   // keys of the page that exist
    for (int c = tid; c < kPfKeys * kChunks; c += kPfThreads) {
      const int r = c / kChunks, e = c % kChunks * 4;
      pf_copy16(dst + r * pitch + e, src + (r < n ? r * HD + e : 0), r < n);
    }
  };
  for (int c = tid; c < C::kRows * kChunks; c += kPfThreads) {
    const int r = c / kChunks, e = c % kChunks * 4;
    const bool there = r < rows_here;
    pf_copy16(Qs + r * C::kKPitch + e, p.q + ((size_t)(q_begin + t0 + (there ? r : 0)) * p.n_q + head) * HD + e, there);
  }
  load_page(p.k_cache, Ks, C::kKPitch, page_lo);
  asm volatile("cp.async.commit_group;" ::: "memory");
  load_page(p.v_cache, Vs, HD, page_lo);
  asm volatile("cp.async.commit_group;" ::: "memory");

  const int row0 = warp * 4 * RI + (lane >> 3), col = lane & 7;
  constexpr int kOut = HD / 32;
  float2 o[RI][kOut][2];
  float m_run[RI], l_run[RI];
#pragma unroll
  for (int i = 0; i < RI; ++i) {
    m_run[i] = -INFINITY;
    l_run[i] = 0.f;
#pragma unroll
    for (int j = 0; j < kOut; ++j) o[i][j][0] = o[i][j][1] = make_float2(0.f, 0.f);
  }
  // a warp none of whose rows exist only helps with the copies
  const bool idle = warp * 4 * RI >= rows_here;

  for (int pg = page_lo; pg <= page_hi; ++pg) {
    const int key0 = pg * kPfKeys;
    const bool edge = key0 + kPfKeys - 1 > start + t0 || key0 < last_lo;
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();                                             // K (and, the first time, Q) is there
    if (!idle) {
      float2 s[RI][8];
#pragma unroll
      for (int i = 0; i < RI; ++i)
#pragma unroll
        for (int j = 0; j < 8; ++j) s[i][j] = make_float2(0.f, 0.f);
#pragma unroll 4
      for (int d = 0; d < HD; d += 4) {
        float4 k[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) k[j] = *reinterpret_cast<const float4*>(Ks + (col + 8 * j) * C::kKPitch + d);
#pragma unroll
        for (int i = 0; i < RI; ++i) {
          const float4 a = *reinterpret_cast<const float4*>(Qs + (row0 + 4 * i) * C::kKPitch + d);
#pragma unroll
          for (int j = 0; j < 8; ++j) pf_fma2(s[i][j], make_float2(a.x, a.y), make_float2(k[j].x, k[j].y));
#pragma unroll
          for (int j = 0; j < 8; ++j) pf_fma2(s[i][j], make_float2(a.z, a.w), make_float2(k[j].z, k[j].w));
        }
      }
#pragma unroll
      for (int i = 0; i < RI; ++i) {
        const int pos = start + t0 + row0 + 4 * i;
        const int lo = first_visible_key(pos, p.window);
        float x[8], mx = -INFINITY;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const int key = key0 + col + 8 * j;
          x[j] = (!edge || (key <= pos && key >= lo)) ? (s[i][j].x + s[i][j].y) * p.scale : -INFINITY;
          mx = fmaxf(mx, x[j]);
        }
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 4));
        const float m_new = fmaxf(m_run[i], mx);
        const float m_use = m_new == -INFINITY ? 0.f : m_new;    // a row that has seen no key yet
        const float alpha = expf(m_run[i] - m_use);
        float sum = 0.f;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float w = expf(x[j] - m_use);
          Ps[(row0 + 4 * i) * kPfPitch + col + 8 * j] = w;
          sum += w;
        }
        sum += __shfl_xor_sync(0xffffffffu, sum, 1);
        sum += __shfl_xor_sync(0xffffffffu, sum, 2);
        sum += __shfl_xor_sync(0xffffffffu, sum, 4);
        l_run[i] = l_run[i] * alpha + sum;
        m_run[i] = m_new;
#pragma unroll
        for (int j = 0; j < kOut; ++j)
#pragma unroll
          for (int h = 0; h < 2; ++h) { o[i][j][h].x *= alpha; o[i][j][h].y *= alpha; }
      }
    }
    __syncthreads();                                             // K is done with
    if (pg < page_hi) load_page(p.k_cache, Ks, C::kKPitch, pg + 1);
    asm volatile("cp.async.commit_group;" ::: "memory");
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    // V is there once all have come; with it the answer whether an edge page holds a value that is not finite
    int odd = 0;
    if (edge) {
      __syncthreads();
      for (int c = tid; c < kPfKeys * kChunks; c += kPfThreads) {
        const float4 v = reinterpret_cast<const float4*>(Vs)[c];
        odd |= !(fabsf(v.x) < INFINITY) | !(fabsf(v.y) < INFINITY) | !(fabsf(v.z) < INFINITY) | !(fabsf(v.w) < INFINITY);
      }
    }
    odd = __syncthreads_or(odd);
    if (!idle) {
#pragma unroll 2
      for (int k4 = 0; k4 < kPfKeys; k4 += 4) {
        float4 w[RI];
#pragma unroll
        for (int i = 0; i < RI; ++i) w[i] = *reinterpret_cast<const float4*>(Ps + (row0 + 4 * i) * kPfPitch + k4);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          float4 v[kOut];
#pragma unroll
          for (int j = 0; j < kOut; ++j) v[j] = *reinterpret_cast<const float4*>(Vs + (k4 + e) * HD + 4 * col + 32 * j);
#pragma unroll
          for (int i = 0; i < RI; ++i) {
            const float wi = e == 0 ? w[i].x : e == 1 ? w[i].y : e == 2 ? w[i].z : w[i].w;
            if (odd) {
              const int key = key0 + k4 + e, pos = start + t0 + row0 + 4 * i;
              if (key > pos || key < first_visible_key(pos, p.window)) continue;
            }
#pragma unroll
            for (int j = 0; j < kOut; ++j) {
              pf_fma2(o[i][j][0], make_float2(wi, wi), make_float2(v[j].x, v[j].y));
              pf_fma2(o[i][j][1], make_float2(wi, wi), make_float2(v[j].z, v[j].w));
            }
          }
        }
      }
    }
    __syncthreads();                                             // V is done with
    if (pg < page_hi) load_page(p.v_cache, Vs, HD, pg + 1);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
  for (int i = 0; i < RI; ++i) {
    const int r = row0 + 4 * i;
    if (r >= rows_here) continue;
    const float inv = 1.f / l_run[i];
    float* dst = p.out + ((size_t)(q_begin + t0 + r) * p.n_q + head) * HD + 4 * col;
#pragma unroll
    for (int j = 0; j < kOut; ++j)
      *reinterpret_cast<float4*>(dst + 32 * j) =
          make_float4(o[i][j][0].x * inv, o[i][j][0].y * inv, o[i][j][1].x * inv, o[i][j][1].y * inv);
  }
}

template <int HD, int RI>
static int launch_prefill_f32(const PrefillF32Args& a, int n_seqs, int max_q_len, cudaStream_t stream) {
  using C = PrefillF32<HD, RI>;
  const int tiles = (max_q_len + C::kRows - 1) / C::kRows;
  if (tiles > 65535) return LLMIE_ERR_UNSUPPORTED_SIZE;
  const cudaError_t e = cudaFuncSetAttribute(attention_prefill_f32_kernel<HD, RI>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, C::smem_bytes());
  if (e != cudaSuccess) return (int)e;
  attention_prefill_f32_kernel<HD, RI><<<dim3(a.n_q, tiles, n_seqs), kPfThreads, C::smem_bytes(), stream>>>(a);
  LLMIE_LAUNCH_CHECK();
  return LLMIE_OK;
}

}  // namespace llmie

using namespace llmie;

// q, out float32 [n_tokens, n_q hd], sequences packed one after another (cu_q [n_seqs + 1]); caches float32 [pages, n_kv, 64,
// hd], hd 64 or 128. seq_start[i]: tokens sequence i held before this step. window: 0, n > 0 a sliding window, -n < 0 chunks
// of n positions. max_q_len: the longest new run, for the grid.
extern "C" int llmie_attention_prefill_f32(const float* q, const float* k_cache, const float* v_cache, float* out,
                                           const int* cu_q, const int* seq_slot, const int* seq_start,
                                           const int* block_table, int max_pages, int n_seqs, int max_q_len, int n_q,
                                           int n_kv, int hd, float scale, int window, cudaStream_t stream) {
  if (n_seqs < 0 || max_q_len < 0 || n_q <= 0 || n_kv <= 0 || n_q % n_kv || max_pages <= 0) return LLMIE_ERR_BAD_ARG;
  if (hd != 64 && hd != 128) return LLMIE_ERR_UNSUPPORTED_SIZE;
  if (!aligned16(q) || !aligned16(k_cache) || !aligned16(v_cache) || !aligned16(out)) return LLMIE_ERR_ALIGNMENT;
  if (n_seqs == 0 || max_q_len == 0) return LLMIE_OK;
  if (n_seqs > 65535) return LLMIE_ERR_UNSUPPORTED_SIZE;
  const PrefillF32Args a{q, k_cache, v_cache, out, cu_q, seq_slot, seq_start, block_table, max_pages, n_q, n_kv, window, scale};
  // pieces of up to 16 tokens: tiles of 16 rows (a row's bits are the same in both)
  if (max_q_len <= 16)
    return hd == 64 ? launch_prefill_f32<64, 1>(a, n_seqs, max_q_len, stream) : launch_prefill_f32<128, 1>(a, n_seqs, max_q_len, stream);
  return hd == 64 ? launch_prefill_f32<64, 4>(a, n_seqs, max_q_len, stream) : launch_prefill_f32<128, 4>(a, n_seqs, max_q_len, stream);
}
