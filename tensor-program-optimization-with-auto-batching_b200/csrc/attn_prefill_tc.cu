// Causal attention for prompt rows on the 5th-generation tensor cores (tcgen05 + TMEM): the ragged prefill path of
// paged_kv_cache.attention_with_fused_qkv (tvm/llama_auto_batcher/llama_for_causal_lm.py:55-64, prefill call
// llama_exec_graph.py:75-85) after the rows' keys and values have been appended to the pages.
//
// One CTA = one tile of up to 128 consecutive prompt rows of ONE sequence x one head.  Per block of 128 keys:
//   S = Q K^T      tcgen05.mma, M = 128 queries, N = 128 keys, K = head_dim 128; Q and K both K-major in 128-byte-swizzled
//                  shared memory -- Q by one TMA load per tile, K by one TMA load per page (16 keys) through the block table;
//   softmax        one thread per query row (= TMEM lane): its 128 scores by tcgen05.ld, twice -- causal mask and maximum, then
//                  probabilities as bf16 back into TMEM over the scores, and their sum;
//   P V            A = P from TMEM, N = 128 head dims, K = 128 keys; V arrives by TMA exactly as the pages hold it,
//                  [key][dim], and is used as an MN-major B operand (the dimension is the contiguous one): no transpose;
//   O = O * exp2(m_old - m_new) + P V    in registers (128 fp32 per thread), while the tensor pipe is at the next S.
// Scores are taken relative to the exact running maximum, so that the largest probability of a row is 1, which bf16 holds
// exactly.  (A reference that lags behind the maximum, with O summed up in TMEM, is 5 % faster -- 354 us against 374 for 2 x 4096
// rows -- but rounds dominating probabilities, which the sum does not see: 1.7 to 3.4 x the error for peaked rows.)
//
// What bounds it: the softmax -- 16384 exponentials per block are 1024 cycles of an SM, the two MMAs are 1024 cycles of
// tensor pipe -- and the chain S -> softmax -> P V of a CTA.  Two CTAs share an SM (96 KB of shared memory, 256 TMEM
// columns and 168 registers per thread each) and fill each other's gaps; a CTA's own copies are off the chain: K of the next
// block is fetched from the moment S = Q K^T has read it, V from the moment P V has.  Scores and P V come 16 columns at a
// time, the next 16 on their way while one is at work (32 at a time, each waited for: 681 us instead of 362 at 2 x 4096).
// CTAs of late tiles (most keys) start first.
// Measured (32 heads of 128, keys and values dense, CUDA events), one buffer of K / V and P through shared memory -> this:
// 2 x 4096 rows 589 -> 374 us (735 TFLOP/s), 16 x 512 148 -> 109, 64 x 128 95 -> 75, 1 x 8192 1085 -> 672 (818); from pages,
// 2 x 4096: 362 us where they lie in order (eight per copy), 418 shuffled.
// Every wait is bounded; a CTA that gives up writes zeros.
#include <math.h>

#include <atomic>
#include <type_traits>

#include "common.cuh"
#include "tc_ptx.cuh"

namespace mlora {
namespace {

constexpr int kPS = 16;            // keys per copy of the paged form: a page, or a part of one
constexpr int kTile = 128;         // query rows per CTA = keys per block
constexpr int kPfThreads = 160;    // warps 0..3: one thread per query row; warp 4: TMA + MMA issue
constexpr int kSub = kTile * 64 * 2;  // one [128 x 64] bf16 sub-tile: 16 KB
constexpr float kLog2e = 1.4426950408889634f;

__device__ __forceinline__ float fast_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

struct PfArgs {
  const int32_t* block_table;  // paged form
  int max_pages;
  const int32_t* tiles;  // [n_tiles][4]: cache slot (dense form: row of the sequence's key 0), first row (index into qkv /
                         // out), rows, position of the first row
  int Hq, Hkv;
  bf16* out;
  int64_t ld_out;
  int32_t* status;  // optional: set to 1 when a wait expired
  float scale;      // of the scores
  const bf16* gate; // dense form: a head's result of row t is multiplied by sigmoid(gate[t * ld_gate + head]); NULL: no gate
  int64_t ld_gate;
  int v_col;        // dense form: column of head 0's values in a row of keys and values
  int page_parts;   // paged form: page size in 16s
  int chunk;        // > 0: a row sees only positions of its own chunk of this many (counted from position 0)
  const float* sink;  // [Hq] or NULL: a logit per head that only enters the softmax's sum
  int n_tiles;
  int runs;         // paged form: the maps of eight pages are there (pages of 16)
};

// NK, NV: query/key and value size of a head in 64s.  PAGED: keys and values come 16 at a time through the block table,
// from the first page of the chunk that the tile's first row lies in; else they are consecutive rows [key][head 0's key, head 1's key, ..., head 0's value, ...], one TMA
// box per 128 keys.
template <int NK, int NV, bool PAGED>
__global__ void __launch_bounds__(kPfThreads, 2) prefill_attn_tc_kernel(const __grid_constant__ CUtensorMap map_q,
                                                                         const __grid_constant__ CUtensorMap map_k,
                                                                         const __grid_constant__ CUtensorMap map_v,
                                                                         const __grid_constant__ CUtensorMap map_k8,
                                                                         const __grid_constant__ CUtensorMap map_v8,
                                                                         PfArgs a) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* sq = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint8_t* sk = sq + NK * kSub;  // K block   [128 keys][128 d]   as two d-halves
  uint8_t* sv = sk + NK * kSub;  // V block   [128 keys][128 d]   as two d-halves, exactly as the pages hold it
  __shared__ uint64_t kbar, vbar;  // a block's K (the first: and Q) / V has landed
  __shared__ uint64_t sbar;        // S = Q K^T has retired, and every P V before it
  __shared__ uint64_t pbar;        // the four softmax warps have written P, and taken the P V before into O
  __shared__ uint64_t obar;        // P V has retired
  __shared__ uint32_t tmem_slot;
  __shared__ int s_abort;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int tile = a.n_tiles - 1 - (int)(blockIdx.x / a.Hq), h = blockIdx.x % a.Hq;
  const int rep = a.Hq / a.Hkv, kvh = h / rep;
  const int slot = a.tiles[tile * 4 + 0], row0 = a.tiles[tile * 4 + 1], rows = a.tiles[tile * 4 + 2], pos0 = a.tiles[tile * 4 + 3];
  if (rows <= 0) return;  // (the whole CTA, before it has asked for anything)
  const int32_t* bt = PAGED ? a.block_table + (size_t)slot * a.max_pages : nullptr;
  constexpr int kDv = NV * 64;
  const int chunk = a.chunk > 0 ? a.chunk : 0x7fffffff;
  const int key0 = PAGED ? (pos0 - pos0 % chunk) / kPS * kPS : 0;  // first key that is read
  const int lo_last = pos0 + rows - 1 - (pos0 + rows - 1) % chunk;  // first key the last row sees
  const int n_keys = pos0 + rows;                       // keys any row of the tile may see
  const int n_blocks = (n_keys - key0 + kTile - 1) / kTile;
  const int n_pages = (n_keys + kPS - 1) / kPS;

  if (tid == 0) {
    s_abort = 0;
    mbar_init(&kbar, 1);
    mbar_init(&vbar, 1);
    mbar_init(&sbar, 1);
    mbar_init(&pbar, 4);
    mbar_init(&obar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    tma_prefetch_desc(&map_q);
    tma_prefetch_desc(&map_k);
    tma_prefetch_desc(&map_v);
    if (PAGED && a.runs) {
      tma_prefetch_desc(&map_k8);
      tma_prefetch_desc(&map_v8);
    }
  }
  if (warp == 4) tmem_alloc(&tmem_slot, 256);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = tmem_slot, tmem_o = tmem_base + kTile;

  if (warp == 4) {
    // ---- copies and MMAs: lane 0 waits and issues, eight lanes copy a page each -----------------------------------------
    constexpr uint32_t idesc = make_idesc(kTile, kTile);
    constexpr uint32_t idesc_pv = make_idesc(kTile, kDv) | (1u << 16);  // B operand MN-major
    auto wait = [&](uint64_t* bar, uint32_t par) {
      int w = 1;
      if (lane == 0) w = mbar_wait(bar, par, &s_abort) ? 1 : 0;
      w = __shfl_sync(0xffffffffu, w, 0);
      if (!w) s_abort = 1;
      return w != 0;
    };
    // Block-table entries are read one block ahead (lane p keeps page p of the block's eight), so that no block starts with
    // a dependent chain of two global round trips.
    // (row of the first of 16 keys in the pages seen as rows)
    auto page_of = [&](int kb) {
      const int pg = key0 / kPS + kb * (kTile / kPS) + lane;
      return PAGED && lane < kTile / kPS && pg < n_pages
                 ? ((bt[pg / a.page_parts] * a.Hkv + kvh) * a.page_parts + pg % a.page_parts) * kPS : -kPS;
    };
    auto copy = [&](int kb, int page, uint8_t* dst, const CUtensorMap* map, const CUtensorMap* map8, uint64_t* bar, int parts, int col,
                    uint32_t more) {
      const int valid = PAGED ? min(kTile / kPS, n_pages - key0 / kPS - kb * (kTile / kPS)) : 0;
      if (PAGED && a.runs && valid == kTile / kPS) {
        // eight pages one after the other in the pool, as a pool that has not been churned hands them out: one copy per
        // 64-column part instead of eight (copies of 2 KB are bound by their number)
        const int first = __shfl_sync(0xffffffffu, page, 0);
        if (__all_sync(0xffffffffu, lane >= kTile / kPS || page == first + lane * a.Hkv * kPS)) {
          if (lane == 0) {
            mbar_expect_tx(bar, (uint32_t)(parts * kSub) + more);
            for (int j = 0; j < parts; ++j) tma_load_4d(dst + j * kSub, map8, j * 64, 0, kvh, (first / kPS - kvh) / a.Hkv, bar);
          }
          __syncwarp();
          return;
        }
      }
      if (lane == 0) {
        mbar_expect_tx(bar, (PAGED ? (uint32_t)(valid * parts * kPS * 128) : (uint32_t)(parts * kSub)) + more);
        if constexpr (!PAGED)  // rows past the sequence's last key belong to the next one (or are zeros): masked
          for (int j = 0; j < parts; ++j) tma_load_2d(dst + j * kSub, map, col + j * 64, slot + kb * kTile, bar);
      }
      __syncwarp();
      if (PAGED && lane < valid)  // 16 keys per lane, every 64-column part
        for (int j = 0; j < parts; ++j) tma_load_2d(dst + j * kSub + lane * (kPS * 128), map, j * 64, page, bar);
      __syncwarp();
    };
    const int k_col = h * NK * 64, v_col = a.v_col + h * NV * 64;
    int page = page_of(0), page_next = page_of(1);
    copy(0, page, sk, &map_k, &map_k8, &kbar, NK, k_col, NK * kSub);
    if (lane == 0)
      for (int j = 0; j < NK; ++j) tma_load_2d(sq + j * kSub, &map_q, k_col + j * 64, row0, &kbar);
    copy(0, page, sv, &map_v, &map_v8, &vbar, NV, v_col, 0);
    for (int kb = 0; kb < n_blocks; ++kb) {
      const uint32_t par = kb & 1;
      if (!wait(&kbar, par)) break;
      if (lane == 0) {
        tc_fence_after();
#pragma unroll
        for (int j = 0; j < NK; ++j) {
          const uint64_t adesc = make_smem_desc(smem_u32(sq + j * kSub));
          const uint64_t bdesc = make_smem_desc(smem_u32(sk + j * kSub));
#pragma unroll
          for (int k = 0; k < 4; ++k) umma_bf16(tmem_base, adesc + 2 * k, bdesc + 2 * k, idesc, (j > 0 || k > 0) ? 1u : 0u);
        }
        umma_commit(&sbar);
      }
      if (kb > 0) {  // V's place is free once the P V before has retired (as it has when this S retires)
        if (!wait(&obar, par ^ 1)) break;
        copy(kb, page, sv, &map_v, &map_v8, &vbar, NV, v_col, 0);
      }
      if (kb + 1 < n_blocks) {
        if (!wait(&sbar, par)) break;
        page = page_next;
        page_next = page_of(kb + 2);
        copy(kb + 1, page, sk, &map_k, &map_k8, &kbar, NK, k_col, 0);
      }
      if (!wait(&vbar, par) || !wait(&pbar, par)) break;
      if (lane == 0) {
        tc_fence_after();
        // A = P in TMEM, two keys per column: 16 keys are 8 columns.  B = V as the pages hold it, [key][dim]: the dimension
        // (N) is the contiguous one ("MN-major"), 64 of it per 128-byte row, the second 64 one sub-tile (leading byte
        // offset) further, 8 keys per 1024-byte swizzle group (stride byte offset), 16 keys = 2048 bytes.
#pragma unroll
        for (int k = 0; k < kTile / 16; ++k)
          umma_bf16_ta(tmem_o, tmem_base + k * 8, make_smem_desc_mn(smem_u32(sv + k * 2048), kSub, 1024), idesc_pv,
                       k > 0 ? 1u : 0u);
        umma_commit(&obar);
      }
      __syncwarp();
    }
    if (s_abort && lane == 0)  // copies may still be in flight: let them land before the shared memory goes to another CTA
      for (int i = 0; i < 64; ++i) __nanosleep(1000);
  } else {
    // ---- softmax: one thread per query row --------------------------------------------------------------------------------
    const int q_pos = pos0 + tid;  // position of this thread's query row
    const int q_lo = q_pos - q_pos % chunk;  // first key it sees
    const float scale = a.scale * kLog2e;
    const uint32_t lanes = (uint32_t)(warp * 32) << 16;
    // maximum of the row's scores so far, and their sum relative to it (a sink: a score of its own without a value)
    float o[kDv];
#pragma unroll
    for (int i = 0; i < kDv; ++i) o[i] = 0.f;
    float m_run = a.sink ? a.sink[h] * kLog2e : -INFINITY, l_run = a.sink ? 1.f : 0.f;
    bool ok = true;
    for (int kb = 0; kb < n_blocks && ok; ++kb) {
      const uint32_t par = kb & 1;
      const int kstart = key0 + kb * kTile;  // first key of the block
      ok = __all_sync(0xffffffffu, mbar_wait(&sbar, par, &s_abort));
      if (!ok) break;
      tc_fence_after();
      // Only the blocks on or past the diagonal need the causal / length mask, and those before the last row's chunk the
      // chunk's (uniform per CTA): every row of the tile sees every key of the blocks between.
      const bool need_mask = kstart + kTile - 1 > pos0 || kstart < lo_last;
      const int hi = min(q_pos, n_keys - 1) - kstart, lo = q_lo - kstart;  // keys of the block that this row sees
      const uint32_t s_addr = tmem_base + lanes;
      float buf[2][16];  // 16 scores at work, the next 16 on their way
      // pass 1: row maximum (of the raw scores: the scale is positive)
      float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
      auto maximum = [&](auto masked) {
        tmem_ld16_issue(s_addr, buf[0]);
#pragma unroll
        for (int c = 0; c < kTile / 16; ++c) {
          tmem_wait_ld16(buf[c & 1]);
          if (c + 1 < kTile / 16) tmem_ld16_issue(s_addr + (c + 1) * 16, buf[(c + 1) & 1]);
#pragma unroll
          for (int i = 0; i < 16; ++i)
            if (!masked() || (c * 16 + i <= hi && c * 16 + i >= lo)) mx[i & 3] = fmaxf(mx[i & 3], buf[c & 1][i]);
        }
      };
      if (need_mask)
        maximum(std::true_type{});
      else
        maximum(std::false_type{});
      const float m_new = fmaxf(m_run, fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])) * scale);
      const float corr = m_run == -INFINITY ? 0.f : fast_exp2(m_run - m_new);  // (m_new == -inf: nothing seen yet, l and o are 0)
      const float neg_m = m_new == -INFINITY ? 0.f : -m_new;                   // (then every key of the block is masked)
      // pass 2: probabilities -> P (bf16 pairs, over scores that have been read), row sum
      float sum = 0.f;
      auto probabilities = [&](auto masked) {
        tmem_ld16_issue(s_addr, buf[0]);
#pragma unroll
        for (int c = 0; c < kTile / 16; ++c) {
          tmem_wait_ld16(buf[c & 1]);
          if (c + 1 < kTile / 16) tmem_ld16_issue(s_addr + (c + 1) * 16, buf[(c + 1) & 1]);
          uint32_t pk[8];
#pragma unroll
          for (int i = 0; i < 16; i += 2) {
            float p[2];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              const int key = c * 16 + i + e;
              p[e] = fast_exp2(fmaf(buf[c & 1][i + e], scale, neg_m));
              if (masked() && !(key <= hi && key >= lo)) p[e] = 0.f;
              sum += p[e];
            }
            const __nv_bfloat162 b = __floats2bfloat162_rn(p[0], p[1]);
            pk[i / 2] = *reinterpret_cast<const uint32_t*>(&b);
          }
          tmem_st8_issue(s_addr + c * 8, pk);
        }
        tmem_wait_st();
      };
      if (need_mask)
        probabilities(std::true_type{});
      else
        probabilities(std::false_type{});
      l_run = fmaf(l_run, corr, sum);
      m_run = m_new;
      if (n_keys - kstart < kTile) {
        // Last block, not full: the V rows of keys that do not exist (the tail of the last page, whatever the cache holds
        // there, and the pages that were not loaded) are zeroed once the copies have landed -- their probabilities are 0,
        // but 0 * NaN is not.  K needs nothing: those scores are masked.  (A swizzled row stays inside its own 128 bytes.)
        ok = __all_sync(0xffffffffu, mbar_wait(&vbar, par, &s_abort));
        if (!ok) break;
        if (tid >= n_keys - kstart) {
#pragma unroll
          for (int half = 0; half < NV; ++half)
#pragma unroll
            for (int c = 0; c < 8; ++c) reinterpret_cast<uint4*>(sv + half * kSub + tid * 128)[c] = make_uint4(0u, 0u, 0u, 0u);
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&pbar);
      // O = O * corr + P V, while the tensor pipe is at the next block's scores
      ok = __all_sync(0xffffffffu, mbar_wait(&obar, par, &s_abort));
      if (!ok) break;
      tc_fence_after();
      tmem_ld16_issue(tmem_o + lanes, buf[0]);
#pragma unroll
      for (int c = 0; c < kDv / 16; ++c) {
        tmem_wait_ld16(buf[c & 1]);
        if (c + 1 < kDv / 16) tmem_ld16_issue(tmem_o + lanes + (c + 1) * 16, buf[(c + 1) & 1]);
#pragma unroll
        for (int i = 0; i < 16; ++i) o[c * 16 + i] = fmaf(o[c * 16 + i], corr, buf[c & 1][i]);
      }
    }
    if (!ok) s_abort = 1;
    // ---- write ----------------------------------------------------------------------------------------------------------
    float inv = (ok && l_run > 0.f) ? 1.f / l_run : 0.f;
    if constexpr (!PAGED)
      if (a.gate && tid < rows) inv /= 1.f + __expf(-__bfloat162float(a.gate[(size_t)(row0 + tid) * a.ld_gate + h]));
    uint4* dst = reinterpret_cast<uint4*>(a.out + (size_t)(row0 + tid) * a.ld_out + (size_t)h * kDv);
    if (tid < rows) {
#pragma unroll
      for (int c = 0; c < kDv / 8; ++c) {
        float f[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) f[i] = o[c * 8 + i] * inv;
        dst[c] = pack8(f);
      }
    }
    if (!ok && tid == 0 && a.status) atomicOr(a.status, 1);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 4) tmem_dealloc(tmem_base, 256);
}

// Pages [n_pages][Hkv][16][D] with a box of eight pages of one head, 64 columns: the same 128 rows of 128 bytes in shared memory
// that eight copies of a page write.
int make_pages_map(CUtensorMap* m, const void* ptr, int n_pages, int Hkv, int D) {
  EncodeTiledFn fn = encode_fn();
  if (!fn) return fail(MLORA_ECUDA, "prefill_attention: cuTensorMapEncodeTiled is not available from this driver");
  cuuint64_t dims[4] = {(cuuint64_t)D, (cuuint64_t)kPS, (cuuint64_t)Hkv, (cuuint64_t)n_pages};
  cuuint64_t strides[3] = {(cuuint64_t)D * 2, (cuuint64_t)kPS * D * 2, (cuuint64_t)Hkv * kPS * D * 2};
  cuuint32_t box[4] = {64, (cuuint32_t)kPS, 1, (cuuint32_t)(kTile / kPS)};
  cuuint32_t estr[4] = {1, 1, 1, 1};
  CUresult r = fn(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(MLORA_ECUDA, "prefill_attention: cuTensorMapEncodeTiled (pages) failed with %d", (int)r);
  return MLORA_OK;
}

template <int NK, int NV, bool PAGED>
int launch_prefill(const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv, const CUtensorMap& mk8, const CUtensorMap& mv8, PfArgs a, int n_tiles, cudaStream_t st) {
  if ((long long)n_tiles * a.Hq > 2147483647ll) return fail(MLORA_ESIZE, "prefill_attention: too many tiles x heads");
  a.n_tiles = n_tiles;
  constexpr int smem = (2 * NK + NV) * kSub + 1024;  // Q, K, V
  static std::atomic<unsigned long long> attr_done{0};
  int dev = 0;
  cudaGetDevice(&dev);
  if (!((attr_done.load(std::memory_order_acquire) >> (dev & 63)) & 1ull)) {
    cudaError_t e = cudaFuncSetAttribute(prefill_attn_tc_kernel<NK, NV, PAGED>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return fail(MLORA_ECUDA, "prefill_attention: cudaFuncSetAttribute: %s", cudaGetErrorString(e));
    attr_done.fetch_or(1ull << (dev & 63), std::memory_order_release);
  }
  prefill_attn_tc_kernel<NK, NV, PAGED><<<(unsigned)((long long)n_tiles * a.Hq), kPfThreads, smem, st>>>(mq, mk, mv, mk8, mv8, a);
  count_launch();
  MLORA_CHECK_LAUNCH("prefill_attn_tc_kernel");
  return MLORA_OK;
}

}  // namespace
}  // namespace mlora

using namespace mlora;

extern "C" int mlora_prefill_attention_masked(const void* d_q, int64_t ld, const void* d_k_pages, const void* d_v_pages,
                                              int32_t n_pages_total, const int32_t* d_block_table, int32_t max_pages,
                                              const int32_t* d_tiles, int32_t n_tiles, int32_t Hq, int32_t Hkv, int32_t D,
                                              int32_t page_size, float scale, int32_t chunk, const float* d_sink, int32_t T,
                                              void* d_out, int64_t ld_out, int32_t* d_status, void* stream) {
  MLORA_REQUIRE((D == 64 || D == 128) && page_size > 0 && page_size % kPS == 0,
                "prefill_attention: head_dim 64 or 128 and pages of a multiple of 16 only (got %d, %d)", D, page_size);
  MLORA_REQUIRE(scale > 0.f && chunk >= 0, "prefill_attention: the scale must be positive, the chunk not negative");
  MLORA_REQUIRE(n_tiles >= 0 && T >= 0 && Hq > 0 && Hkv > 0 && Hq % Hkv == 0 && n_pages_total > 0 && max_pages > 0,
                "prefill_attention: bad sizes");
  MLORA_REQUIRE(d_q && d_k_pages && d_v_pages && d_block_table && d_tiles && d_out, "prefill_attention: null pointer");
  MLORA_REQUIRE(aligned16(d_q) && aligned16(d_k_pages) && aligned16(d_v_pages) && aligned16(d_out) && (ld * 2) % 16 == 0 &&
                    (ld_out * 2) % 16 == 0,
                "prefill_attention: 16-byte alignment of tensors and row pitches");
  MLORA_REQUIRE(n_tiles <= 2147483647 / 4 && Hq <= 65535, "prefill_attention: too many tiles / heads");
  if (n_tiles == 0 || T == 0) return MLORA_OK;
  CUtensorMap mq, mk, mv;
  int rc = make_map(&mq, d_q, T, Hq * D, ld, kTile, 64);  // only the q part of every row is mapped
  if (rc) return rc;
  rc = make_map(&mk, d_k_pages, (long long)n_pages_total * Hkv * page_size, D, D, kPS, 64);
  if (rc) return rc;
  rc = make_map(&mv, d_v_pages, (long long)n_pages_total * Hkv * page_size, D, D, kPS, 64);
  if (rc) return rc;
  PfArgs a{d_block_table, max_pages, d_tiles, Hq, Hkv, (bf16*)d_out, ld_out, d_status, scale, nullptr, 0, 0,
           page_size / kPS, chunk, d_sink, 0, 0};
  CUtensorMap mk8 = mk, mv8 = mv;
  if (page_size == kPS) {
    rc = make_pages_map(&mk8, d_k_pages, n_pages_total, Hkv, D);
    if (rc) return rc;
    rc = make_pages_map(&mv8, d_v_pages, n_pages_total, Hkv, D);
    if (rc) return rc;
    a.runs = 1;
  }
  return D == 64 ? launch_prefill<1, 1, true>(mq, mk, mv, mk8, mv8, a, n_tiles, (cudaStream_t)stream)
                 : launch_prefill<2, 2, true>(mq, mk, mv, mk8, mv8, a, n_tiles, (cudaStream_t)stream);
}

extern "C" int mlora_prefill_attention(const void* d_qkv, int64_t ld, const void* d_k_pages, const void* d_v_pages,
                                       int32_t n_pages_total, const int32_t* d_block_table, int32_t max_pages,
                                       const int32_t* d_tiles, int32_t n_tiles, int32_t Hq, int32_t Hkv, int32_t D,
                                       int32_t page_size, int32_t T, void* d_out, int64_t ld_out, int32_t* d_status,
                                       void* stream) {
  MLORA_REQUIRE(D == 128 && page_size == kPS, "prefill_attention: head_dim 128 and page size 16 only (got %d, %d)", D, page_size);
  return mlora_prefill_attention_masked(d_qkv, ld, d_k_pages, d_v_pages, n_pages_total, d_block_table, max_pages, d_tiles, n_tiles,
                                        Hq, Hkv, D, page_size, 1.f / sqrtf((float)D), 0, nullptr, T, d_out, ld_out, d_status,
                                        stream);
}

extern "C" int mlora_prefill_attention_dense(const void* d_q, int64_t ld, const void* d_kv, int64_t ld_kv, int32_t kv_rows,
                                             int32_t v_col, const int32_t* d_tiles, int32_t n_tiles, int32_t H, int32_t Dk,
                                             int32_t Dv, float scale, const void* d_gate, int64_t ld_gate, int32_t T, void* d_out,
                                             int64_t ld_out, int32_t* d_status, void* stream) {
  MLORA_REQUIRE((Dk == 64 || Dk == 128) && (Dv == 64 || Dv == 128), "prefill_attention_dense: head sizes 64 and 128 (got %d, %d)", Dk, Dv);
  MLORA_REQUIRE(scale > 0.f, "prefill_attention_dense: the scale must be positive");
  MLORA_REQUIRE(n_tiles >= 0 && T >= 0 && H > 0 && H <= 65535 && kv_rows > 0 && v_col >= H * Dk && v_col % 64 == 0 &&
                    ld_kv >= (int64_t)v_col + (int64_t)H * Dv && ld >= (int64_t)H * Dk && ld_out >= (int64_t)H * Dv,
                "prefill_attention_dense: bad sizes");
  MLORA_REQUIRE(d_q && d_kv && d_tiles && d_out, "prefill_attention_dense: null pointer");
  MLORA_REQUIRE(aligned16(d_q) && aligned16(d_kv) && aligned16(d_out) && (ld * 2) % 16 == 0 && (ld_kv * 2) % 16 == 0 && (ld_out * 2) % 16 == 0,
                "prefill_attention_dense: 16-byte alignment of tensors and row pitches");
  if (n_tiles == 0 || T == 0) return MLORA_OK;
  CUtensorMap mq, mkv;
  int rc = make_map(&mq, d_q, T, H * Dk, ld, kTile, 64);
  if (rc) return rc;
  rc = make_map(&mkv, d_kv, kv_rows, v_col + H * Dv, ld_kv, kTile, 64);
  if (rc) return rc;
  PfArgs a{nullptr, 0, d_tiles, H, H, (bf16*)d_out, ld_out, d_status, scale, (const bf16*)d_gate, ld_gate, v_col, 1, 0, nullptr, 0, 0};
  cudaStream_t st = (cudaStream_t)stream;
  if (Dk == 64 && Dv == 64) return launch_prefill<1, 1, false>(mq, mkv, mkv, mkv, mkv, a, n_tiles, st);
  if (Dk == 64) return launch_prefill<1, 2, false>(mq, mkv, mkv, mkv, mkv, a, n_tiles, st);
  if (Dv == 64) return launch_prefill<2, 1, false>(mq, mkv, mkv, mkv, mkv, a, n_tiles, st);
  return launch_prefill<2, 2, false>(mq, mkv, mkv, mkv, mkv, a, n_tiles, st);
}
