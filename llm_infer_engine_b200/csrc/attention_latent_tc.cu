// Prompts of latent attention on the 5th-generation tensor cores: tcgen05.mma with TMEM accumulators, operands brought in
// by TMA. All query heads share ONE key head whose rows [latent | rotated part] are key and, in their first hdv columns,
// value at once, so a key page is fetched once for both products.
//
// The rows of the problem are the (token, head) pairs of a sequence, row r = token * heads + head: rows that lie beside
// each other in q and out. One block = 128 consecutive rows, 320 threads:
//   warp 0      TMA producer: the rows of Q once ({64 columns, 128 rows} boxes; columns beyond the head size read zeros),
//               then a cache page of 64 keys at a time into a ring of three
//   warp 1      owns TMEM (output hdv columns, two score buffers of 64); one lane issues S = Q K^T two pages ahead and
//               O += P V when P is there; V is the page itself as an MN-major operand
//   warps 2..9  softmax, two threads per row (each 32 of a page's keys and half of the output's columns): scores into
//               registers, mask, running maximum and sum, P as bfloat16 into shared memory
// The output stays in tensor memory. A row's reference maximum moves only when a page's maximum lies more than 2^8 above
// it (its probabilities are then at most 2^8 and keep their relative precision in bfloat16 as in the float32 sums); the
// warp then multiplies its rows' output by the change before it lets the next product go. Every wait is bounded; a block
// that gives up waits for its copies and products (again bounded), leaves NaN in its rows and a code in the status word.
//
// A key that a row may not see has weight 0, and 0 times a value that is not finite is NaN. So pages that the causal line or
// a window's end crosses (one or two of a block's, with whatever the page held behind the sequence's last key) are looked at
// for such values first; where there is one, that page's share of the output is added up on the CUDA cores, over the keys that
// a row sees, and the product is left zeros. Two prompts, 1,805 tokens: 57 us, without the look 55.
//
// What bounds it: a page of 64 keys is 544 (hd + hdv) x 128 x 64 products, 544 tensor cycles at hd 288, hdv 256, and as
// many cycles of exponentials; Q and the ring take 216 KB, one block an SM. Two prompts, 1,805 tokens, 32 heads of 288 /
// 256: 323 us with the mma.sync kernel of 32 rows (attention_rows_mma.cu), 57 us so.
#include "tcgen05.cuh"
#include <math.h>

namespace llmie {
using namespace tc;

constexpr int kLtRows = 128, kLtKeys = 64, kLtStages = 3;
constexpr int kLtSoftmax = 256, kLtThreads = 64 + kLtSoftmax;
constexpr int kLtQSub = kLtRows * 128, kLtKSub = kLtKeys * 128;      // bytes of 64 columns of Q's rows, of a page's
constexpr int kLtMaxSubs = 5;                                         // head sizes up to 320
constexpr int kLtScoreCol = 256;                                      // TMEM columns: output 0.., scores 256 and 320
constexpr float kLtSlack = 8.f;                                       // log2: how far a maximum may run ahead

constexpr int lt_smem_bytes(int subs) { return subs * kLtQSub + kLtQSub + kLtStages * subs * kLtKSub + 1024; }

struct LatentArgs {
  __nv_bfloat16* out;            // [T * heads, hdv]
  const int* cu_q;
  const int* seq_slot;
  const int* seq_start;
  const int* block_table;
  int max_pages, heads, hd, hdv, window, sink;
  float scale;
  const float* sink_vals;        // [heads] or null
  int* status;
};

struct LatentShared {
  uint64_t q_full, k_full[kLtStages], k_empty[kLtStages], s_full[2], s_free[2], p_ready, pv_full, pair_bar[4];
  uint64_t looked[kLtStages], odd_bar, drained;
  uint32_t tmem_base;
  int abort;
  int odd[kLtStages];             // 1 + the last of a stage's pages that held a value that is not finite
  int out_begun;                  // 1: the output holds something before the first product
  float row_val[2][2][kLtRows];
};

__device__ __forceinline__ float lt_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// LIMIT: polls before a wait gives up (a constant: read from the arguments it cost 5 % of the time).
template <unsigned LIMIT>
__global__ void __launch_bounds__(kLtThreads, 1)
attention_latent_tc_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                           const LatentArgs p) {
  extern __shared__ uint8_t lt_smem[];
  __shared__ LatentShared sh;
  const int subs = (p.hd + 63) / 64;
  uint8_t* q_smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(lt_smem) + 1023) & ~(uintptr_t)1023);
  uint8_t* p_smem = q_smem + subs * kLtQSub;
  uint8_t* k_smem = p_smem + kLtQSub;
  const int stage_bytes = subs * kLtKSub;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int seq = blockIdx.x;
  const int q_begin = p.cu_q[seq], n_rows = (p.cu_q[seq + 1] - q_begin) * p.heads;
  const int r0 = (gridDim.y - 1 - blockIdx.y) * kLtRows;      // late rows see the most keys: they start first
  if (r0 >= n_rows) return;                                   // uniform for the block: nothing was set up yet
  const int start = p.seq_start[seq];
  const int rows_here = min(kLtRows, n_rows - r0);
  const int pos_first = start + r0 / p.heads, pos_last = start + (r0 + rows_here - 1) / p.heads;
  const int page_lo = first_visible_key(pos_first, p.window) / kLtKeys;
  const int n_tiles = pos_last / kLtKeys - page_lo + 1;
  const int* pages = p.block_table + (size_t)p.seq_slot[seq] * p.max_pages + page_lo;

  auto load_page = [&](int jt) {
    const int st = jt % kLtStages;
    mbar_arrive_expect_tx(&sh.k_full[st], stage_bytes);
    for (int s = 0; s < subs; ++s)
      tma_load_2d(k_smem + st * stage_bytes + s * kLtKSub, &map_k, s * 64, pages[jt] * kLtKeys, &sh.k_full[st]);
  };
  if (threadIdx.x == 0) {
    mbar_init(&sh.q_full, 1);
    for (int s = 0; s < kLtStages; ++s) {
      mbar_init(&sh.k_full[s], 1);
      mbar_init(&sh.k_empty[s], 1);
      mbar_init(&sh.looked[s], 1);
      sh.odd[s] = 0;
    }
    for (int b = 0; b < 2; ++b) { mbar_init(&sh.s_full[b], 1); mbar_init(&sh.s_free[b], kLtSoftmax); }
    mbar_init(&sh.p_ready, kLtSoftmax);
    mbar_init(&sh.pv_full, 1);
    for (int i = 0; i < 4; ++i) mbar_init(&sh.pair_bar[i], 64);
    mbar_init(&sh.odd_bar, kLtSoftmax);
    mbar_init(&sh.drained, 1);
    sh.abort = sh.out_begun = 0;
    fence_mbar_init();
    tma_prefetch_desc(&map_q);
    tma_prefetch_desc(&map_k);
    mbar_arrive_expect_tx(&sh.q_full, subs * kLtQSub);
    for (int s = 0; s < subs; ++s)
      tma_load_2d(q_smem + s * kLtQSub, &map_q, s * 64, q_begin * p.heads + r0, &sh.q_full);
    load_page(0);
  }
  if (warp == 1) {
    tmem_alloc(&sh.tmem_base, 512);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = sh.tmem_base;
  volatile int* abort = &sh.abort;
  // an edge page holds a key that some row here does not see (the same answer for the whole block)
  const int last_lo = first_visible_key(pos_last, p.window);  // the latest first key among the block's rows
  auto edge_page = [&](int jt) {
    const int key0 = (page_lo + jt) * kLtKeys;
    return key0 + kLtKeys - 1 > pos_first || key0 < last_lo;
  };
  auto chunk_odd = [](const uint4& x) {                       // holds a bfloat16 whose exponent is all ones
    const uint32_t e = 0x7f807f80u, one = 0x00800080u;
    return (((x.x & e) + one) | ((x.y & e) + one) | ((x.z & e) + one) | ((x.w & e) + one)) & 0x80008000u;
  };
  int issued = 1;                                             // pages asked for (thread 0)
  auto wait = [&](uint64_t* bar, uint32_t parity) { return mbar_wait(bar, parity, abort, LIMIT); };
#define LLMIE_FAIL(code) do { if (!*abort) { *abort = 1; atomicExch(p.status, (code)); } } while (0)

  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer (page 0 is on its way); the whole
    // warp looks at each edge page one page behind the loads, long before its turn comes
    for (int jt = 1; jt <= n_tiles; ++jt) {
      if (jt < n_tiles) {
        const bool room = jt < kLtStages || lane != 0 || wait(&sh.k_empty[jt % kLtStages], ((jt / kLtStages) - 1) & 1);
        if (!__all_sync(0xffffffffu, room)) { LLMIE_FAIL(kStatusTimeoutEmpty); break; }
        if (lane == 0) load_page(jt);
        issued = jt + 1;
      }
      const int st = (jt - 1) % kLtStages;
      if (edge_page(jt - 1)) {
        if (!__all_sync(0xffffffffu, wait(&sh.k_full[st], ((jt - 1) / kLtStages) & 1))) { LLMIE_FAIL(kStatusTimeoutFull); break; }
        // only the keys that some row does not see: those behind the first row's, or all where a window ends
        const int key0 = (page_lo + jt - 1) * kLtKeys, from = key0 < last_lo ? 0 : max(pos_first + 1 - key0, 0);
        uint32_t bad = 0;
        for (int s = 0; s < p.hdv / 64; ++s) {
          const uint4* rows = reinterpret_cast<const uint4*>(k_smem + st * stage_bytes + s * kLtKSub) + from * 8;
#pragma unroll 4
          for (int c = lane; c < (kLtKeys - from) * 8; c += 32) bad |= chunk_odd(rows[c]);
        }
        if (__any_sync(0xffffffffu, bad) && lane == 0) *reinterpret_cast<volatile int*>(&sh.odd[st]) = jt;
      }
      if (lane == 0) mbar_arrive(&sh.looked[st]);
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ MMA issuer
    if (elect_one()) {
      constexpr uint32_t idesc_s = make_instr_desc_bf16(kLtRows, kLtKeys, 0, 0);
      const uint32_t idesc_pv = make_instr_desc_bf16(kLtRows, p.hdv, 0, 1);      // V is MN-major
      const uint32_t q_addr = smem_u32(q_smem), p_addr = smem_u32(p_smem);
      const int k_steps = p.hd / 16;
      bool ok = wait(&sh.q_full, 0);
      if (!ok) LLMIE_FAIL(kStatusTimeoutFull);
      auto issue_scores = [&](int jt) -> bool {
        const int st = jt % kLtStages, b = jt & 1, use = jt >> 1;
        if (!wait(&sh.k_full[st], (jt / kLtStages) & 1)) { LLMIE_FAIL(kStatusTimeoutFull); return false; }
        if (use >= 1 && !wait(&sh.s_free[b], (use - 1) & 1)) { LLMIE_FAIL(kStatusTimeoutMma); return false; }
        tc_fence_after_sync();
        const uint32_t k_addr = smem_u32(k_smem + st * stage_bytes);
        for (int kk = 0; kk < k_steps; ++kk)
          mma_bf16_ss(tmem + kLtScoreCol + b * kLtKeys,
                      make_smem_desc(q_addr + (kk >> 2) * kLtQSub + (kk & 3) * 32, 16, 1024),
                      make_smem_desc(k_addr + (kk >> 2) * kLtKSub + (kk & 3) * 32, 16, 1024), idesc_s, kk > 0 ? 1u : 0u);
        mma_commit(&sh.s_full[b]);
        return true;
      };
      if (ok) ok = issue_scores(0);
      if (ok && n_tiles > 1) ok = issue_scores(1);
      for (int jt = 0; ok && jt < n_tiles; ++jt) {
        if (!wait(&sh.p_ready, jt & 1)) { LLMIE_FAIL(kStatusTimeoutMma); break; }
        tc_fence_after_sync();
        const uint32_t v_addr = smem_u32(k_smem + (jt % kLtStages) * stage_bytes);
        const bool begun = jt > 0 || *reinterpret_cast<volatile int*>(&sh.out_begun) != 0;
#pragma unroll
        for (int kk = 0; kk < kLtKeys / 16; ++kk)
          // A = P, K-major: 16 keys = 32 bytes. B = V, MN-major: 16 keys = 16 rows, 64 value columns a block.
          mma_bf16_ss(tmem, make_smem_desc(p_addr + kk * 32, 16, 1024), make_smem_desc(v_addr + kk * 2048, kLtKSub, 1024),
                      idesc_pv, (kk > 0 || begun) ? 1u : 0u);
        mma_commit(&sh.pv_full);
        mma_commit(&sh.k_empty[jt % kLtStages]);
        if (jt + 2 < n_tiles && !issue_scores(jt + 2)) break;
      }
    }
  } else {
    // ------------------------------------------------------------------ softmax, two threads per row
    const int quarter = warp & 3, half = (warp - 2) >> 2;
    const int r = quarter * 32 + lane;                   // row of the tile = TMEM lane
    const uint32_t lane_addr = tmem + ((uint32_t)(quarter * 32) << 16);
    const int qpos = start + (r0 + r) / p.heads;
    const int lo = first_visible_key(qpos, p.window);
    const unsigned span = (unsigned)(qpos - lo);
    const float sl2 = p.scale * 1.4426950408889634f;     // exp(x * scale) = exp2(x * scale * log2 e)
    const int out_cols = p.hdv / 2;
    float m_ref = -INFINITY, l_run = 0.f;                // l_run: the sum over this thread's keys only
    bool ok = true;
    int n_exchanges = 0, n_meetings = 0;
    // hands `mine` to the row's other thread and takes its value
    auto exchange = [&](float mine, float& theirs) -> bool {
      const int buf = n_exchanges & 1;
      sh.row_val[buf][half][r] = mine;
      mbar_arrive(&sh.pair_bar[quarter]);
      const bool ok_ = wait(&sh.pair_bar[quarter], n_exchanges & 1);
      theirs = sh.row_val[buf][half ^ 1][r];
      ++n_exchanges;
      return ok_;
    };
    for (int jt = 0; jt < n_tiles; ++jt) {
      const int b = jt & 1;
      // every decision to give up is the whole warp's: the tensor-memory accesses are warp-wide instructions
      if (!__all_sync(0xffffffffu, wait(&sh.s_full[b], (jt >> 1) & 1))) { LLMIE_FAIL(kStatusTimeoutMma); ok = false; break; }
      tc_fence_after_sync();
      uint32_t v[32];
      tmem_ld_32x32(lane_addr + kLtScoreCol + b * kLtKeys + half * 32, v);
      tmem_ld_wait();
      tc_fence_before_sync();
      mbar_arrive(&sh.s_free[b]);
      const int key0 = (page_lo + jt) * kLtKeys;
      const bool edge = edge_page(jt);
      if (edge) {
        const int lo_rel = lo - key0 - half * 32;          // key c of this thread is seen if lo <= key <= qpos
#pragma unroll
        for (int i = 0; i < 32; ++i)
          if ((unsigned)(i - lo_rel) > span) v[i] = 0xff800000u;
      }
      float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int i = 0; i < 32; ++i) mx[i & 3] = fmaxf(mx[i & 3], __uint_as_float(v[i]));
      float m_tile = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])), other;
      if (!__all_sync(0xffffffffu, exchange(m_tile, other))) { LLMIE_FAIL(kStatusTimeoutMma); ok = false; break; }
      m_tile = fmaxf(m_tile, other);
      // the reference moves when the page's maximum is far above it (always from -inf); both threads decide alike
      const bool move = m_tile > m_ref && !((m_tile - m_ref) * sl2 <= kLtSlack);
      const float m_new = move ? m_tile : m_ref;
      const float m_use = m_new == -INFINITY ? 0.f : m_new;        // a row that has seen no key yet
      const float alpha = move ? lt_exp2((m_ref - m_use) * sl2) : 1.f;
      const float m_scaled = m_use * sl2;
      float ls[4] = {0.f, 0.f, 0.f, 0.f};
      uint32_t w[16];
#pragma unroll
      for (int i = 0; i < 32; i += 2) {
        const float a = lt_exp2(fmaf(__uint_as_float(v[i]), sl2, -m_scaled));
        const float c = lt_exp2(fmaf(__uint_as_float(v[i + 1]), sl2, -m_scaled));
        ls[i & 2] += a;
        ls[(i & 2) + 1] += c;
        const __nv_bfloat162 pr = __floats2bfloat162_rn(a, c);
        w[i >> 1] = *reinterpret_cast<const uint32_t*>(&pr);
      }
      const int st = jt % kLtStages;
      if (edge && !__all_sync(0xffffffffu, wait(&sh.looked[st], (jt / kLtStages) & 1))) { LLMIE_FAIL(kStatusTimeoutFull); ok = false; break; }
      const bool odd = edge && *reinterpret_cast<volatile int*>(&sh.odd[st]) == jt + 1;
      // the product before this one is done with P, and with the output where that has to be brought to a new reference
      if (jt > 0 && !__all_sync(0xffffffffu, wait(&sh.pv_full, (jt - 1) & 1))) { LLMIE_FAIL(kStatusTimeoutMma); ok = false; break; }
#pragma unroll
      for (int ch = 0; ch < 4; ++ch)
        *reinterpret_cast<uint4*>(p_smem + swizzle128_offset(r, half * 4 + ch)) =
            make_uint4(w[4 * ch], w[4 * ch + 1], w[4 * ch + 2], w[4 * ch + 3]);
      if (odd) {
        uint8_t* page = k_smem + st * stage_bytes;
        auto meet = [&]() {
          mbar_arrive(&sh.odd_bar);
          return __all_sync(0xffffffffu, wait(&sh.odd_bar, n_meetings++ & 1));
        };
        if (!meet()) { LLMIE_FAIL(kStatusTimeoutMma); ok = false; break; }     // all of P is there
        tc_fence_after_sync();
        for (int c = half * out_cols; c < (half + 1) * out_cols; c += 32) {
          uint32_t o[32];
          if (jt > 0) {
            tmem_ld_32x32(lane_addr + c, o);
            tmem_ld_wait();
          }
#pragma unroll
          for (int i = 0; i < 32; ++i) o[i] = jt > 0 ? __float_as_uint(__uint_as_float(o[i]) * alpha) : 0u;
          const uint8_t* sub = page + (c >> 6) * kLtKSub;
          for (int k = 0; k < kLtKeys; ++k) {
            if ((unsigned)(k - (lo - key0)) > span) continue;
            const float pk = __bfloat162float(
                *reinterpret_cast<const __nv_bfloat16*>(p_smem + swizzle128_offset(r, k >> 3) + (k & 7) * 2));
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              float x[8];
              load8(reinterpret_cast<const __nv_bfloat16*>(sub + swizzle128_offset(k, ((c & 63) >> 3) + q)), x);
#pragma unroll
              for (int e = 0; e < 8; ++e) o[8 * q + e] = __float_as_uint(fmaf(pk, x[e], __uint_as_float(o[8 * q + e])));
            }
          }
          __syncwarp();
          tmem_st_32x32(lane_addr + c, o);
        }
        tmem_st_wait();
        tc_fence_before_sync();
        if (!meet()) { LLMIE_FAIL(kStatusTimeoutMma); ok = false; break; }     // nobody reads P or the page any more
        const uint4 none = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
        for (int ch = 0; ch < 4; ++ch) *reinterpret_cast<uint4*>(p_smem + swizzle128_offset(r, half * 4 + ch)) = none;
        for (int c = threadIdx.x - 64; c < p.hdv / 64 * (kLtKSub / 16); c += kLtSoftmax)
          if (chunk_odd(reinterpret_cast<const uint4*>(page)[c])) reinterpret_cast<uint4*>(page)[c] = none;
        if (threadIdx.x == 64) *reinterpret_cast<volatile int*>(&sh.out_begun) = 1;
      } else if (jt > 0 && __any_sync(0xffffffffu, move)) {
        tc_fence_after_sync();
        for (int c = 0; c < out_cols; c += 32) {
          uint32_t o[32];
          tmem_ld_32x32(lane_addr + half * out_cols + c, o);
          tmem_ld_wait();
#pragma unroll
          for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
          tmem_st_32x32(lane_addr + half * out_cols + c, o);
        }
        tmem_st_wait();
        tc_fence_before_sync();
      }
      fence_proxy_async_smem();                            // P is visible to the tensor core's reads
      mbar_arrive(&sh.p_ready);
      l_run = fmaf(l_run, alpha, (ls[0] + ls[1]) + (ls[2] + ls[3]));
      m_ref = m_new;
    }
    if (ok && !__all_sync(0xffffffffu, wait(&sh.pv_full, (n_tiles - 1) & 1))) { LLMIE_FAIL(kStatusTimeoutMma); ok = false; }
    float other = 0.f;
    if (ok && !__all_sync(0xffffffffu, exchange(l_run, other))) { LLMIE_FAIL(kStatusTimeoutMma); ok = false; }
    if (ok) {
      tc_fence_after_sync();
      float l = l_run + other;
      // the sink: one more term in the denominator (a score far above the maximum makes it infinite, the output zero)
      if (p.sink) l += lt_exp2((p.sink_vals ? p.sink_vals[(r0 + r) % p.heads] * 1.4426950408889634f : 0.f) - m_ref * sl2);
      const float inv = 1.f / l;
      __nv_bfloat16* dst = p.out + ((size_t)q_begin * p.heads + r0 + r) * p.hdv + half * out_cols;
      for (int c = 0; c < out_cols; c += 32) {
        uint32_t o[32];
        tmem_ld_32x32(lane_addr + half * out_cols + c, o);
        tmem_ld_wait();
        if (r < rows_here) {
#pragma unroll
          for (int i = 0; i < 32; i += 8) {
            float v8[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) v8[e] = __uint_as_float(o[i + e]) * inv;
            store8(dst + c + i, v8);
          }
        }
      }
    }
  }
#undef LLMIE_FAIL
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  if (*abort) {
    // copies and products still in flight land before the block gives its memory up; the rows are no result
    if (threadIdx.x == 0) {
      for (unsigned spin = 0; spin < (1u << 16) && !mbar_test(&sh.q_full, 0); ++spin) __nanosleep(64);
      for (int jt = max(0, issued - kLtStages); jt < issued; ++jt)
        for (unsigned spin = 0; spin < (1u << 16) && !mbar_test(&sh.k_full[jt % kLtStages], (jt / kLtStages) & 1); ++spin)
          __nanosleep(64);
    }
    if (warp == 1 && elect_one()) {                            // the lane that issued the products
      mma_commit(&sh.drained);
      for (unsigned spin = 0; spin < (1u << 16) && !mbar_test(&sh.drained, 0); ++spin) __nanosleep(64);
    }
    uint4* rows = reinterpret_cast<uint4*>(p.out + ((size_t)q_begin * p.heads + r0) * p.hdv);
    const uint4 nan8 = make_uint4(0x7fff7fffu, 0x7fff7fffu, 0x7fff7fffu, 0x7fff7fffu);
    for (int i = threadIdx.x; i < rows_here * p.hdv / 8; i += kLtThreads) rows[i] = nan8;
    __syncthreads();
  }
  if (warp == 1) tmem_dealloc(tmem, 512);
}

}  // namespace llmie

using namespace llmie;

// Whether the kernel takes these sizes (no launch).
extern "C" int llmie_attention_latent_tc_supported(int hd, int hdv, int page_size) {
  return hd > 0 && hd % 16 == 0 && hd <= 64 * kLtMaxSubs && hdv > 0 && hdv % 64 == 0 && hdv <= 256 && hdv <= hd &&
         page_size == kLtKeys;
}

// q bfloat16 [n_tokens, heads hd], out [n_tokens, heads hdv]; cache bfloat16 [n_pages, 1, 64, hd], the values its rows'
// first hdv columns. cu_q, seq_slot, seq_start, block_table, window as in llmie_attention_prefill_tc; scale > 0. sink != 0:
// one more softmax term without a value, of score 0 or sink_vals float32 [heads].
// no_wait != 0: every wait gives up at once (for tests of that path).
extern "C" int llmie_attention_latent_tc_form(const void* q, const void* cache, void* out, const int* cu_q, const int* seq_slot,
                                         const int* seq_start, const int* block_table, int max_pages, int n_pages,
                                         int n_tokens, int n_seqs, int max_q_len, int heads, int hd, int hdv, float scale,
                                         int window, const float* sink_vals, int sink, int* status, int no_wait,
                                         cudaStream_t stream) {
  if (n_tokens < 0 || n_seqs < 0 || heads <= 0 || max_pages <= 0 || n_pages <= 0 || !(scale > 0.f) || !status ||
      (sink_vals && !sink))
    return LLMIE_ERR_BAD_ARG;
  if (!llmie_attention_latent_tc_supported(hd, hdv, kLtKeys)) return LLMIE_ERR_UNSUPPORTED_SIZE;
  if (!aligned16(q) || !aligned16(cache) || !aligned16(out)) return LLMIE_ERR_ALIGNMENT;
  if (n_tokens == 0 || n_seqs == 0 || max_q_len <= 0) return LLMIE_OK;
  const long long row_blocks = ((long long)max_q_len * heads + kLtRows - 1) / kLtRows;
  if (row_blocks > 65535 || (long long)n_tokens * heads > 0x7fffffffLL) return LLMIE_ERR_UNSUPPORTED_SIZE;
  CUtensorMap map_q, map_k;
  int rc = tc::make_tmap_bf16_2d(&map_q, q, (uint64_t)n_tokens * heads, hd, hd, kLtRows);
  if (rc != LLMIE_OK) return rc;
  rc = tc::make_tmap_bf16_2d(&map_k, cache, (uint64_t)n_pages * kLtKeys, hd, hd, kLtKeys);
  if (rc != LLMIE_OK) return rc;
  const int smem = lt_smem_bytes((hd + 63) / 64);
  auto kernel = no_wait ? attention_latent_tc_kernel<0> : attention_latent_tc_kernel<kSpinLimit>;
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, lt_smem_bytes(kLtMaxSubs));
  if (e != cudaSuccess) return (int)e;
  const LatentArgs a{(__nv_bfloat16*)out, cu_q, seq_slot, seq_start, block_table, max_pages, heads, hd, hdv, window,
                     sink ? 1 : 0, scale, sink_vals, status};
  kernel<<<dim3(n_seqs, (unsigned)row_blocks), kLtThreads, smem, stream>>>(map_q, map_k, a);
  LLMIE_LAUNCH_CHECK();
  return LLMIE_OK;
}

extern "C" int llmie_attention_latent_tc(const void* q, const void* cache, void* out, const int* cu_q, const int* seq_slot,
                                         const int* seq_start, const int* block_table, int max_pages, int n_pages,
                                         int n_tokens, int n_seqs, int max_q_len, int heads, int hd, int hdv, float scale,
                                         int window, const float* sink_vals, int sink, int* status, cudaStream_t stream) {
  return llmie_attention_latent_tc_form(q, cache, out, cu_q, seq_slot, seq_start, block_table, max_pages, n_pages, n_tokens,
                                         n_seqs, max_q_len, heads, hd, hdv, scale, window, sink_vals, sink, status, 0,
                                         stream);
}
