// Prompt-size projections on pairs of CTAs (tcgen05 cta_group::2): y[T,out] = x[T,in] W[out,in]^T with hundreds of rows or
// more, plain (with the LoRA expand and the fused activations of linear_tc.cuh) or grouped.
//
// What bounds it: the tensor pipe, once the operands get through shared memory.  A CTA on its own with a 128 x 256 tile
// writes 16 + 32 KB per k-block and its MMAs read them back: 768 cycles of a shared memory that moves 128 bytes per cycle,
// against 512 cycles of MMA -- the pipe is two thirds busy at best.  Here the two CTAs of a cluster compute one tile of
// 256 weight rows x up to 256 tokens: each stages its own 128 weight rows and HALF of the tokens, and the pair's MMA (issued
// by the even CTA) reads both shared memories: 16 + 16 KB per CTA and k-block, 512 cycles against 512, and a third less
// from L2.  Measured at T = 8192 (CUDA events, no adapters), one CTA per tile -> pairs:
//   4096 -> 12288: 683 -> 541 us (1525 TFLOP/s)      4096 -> 4096: 277 -> 190 us (1449)
//   11008 -> 4096: 724 -> 489 us (1512)              4096 -> 22016 with SiLU*up: 1388 -> 1115 us (1325)
//
// Persistent, one pair per two SMs; whole tiles only, dealt round robin (see pair_tile).  Warps of a CTA: 0 = operand
// producer (TMA; the copies of both CTAs complete on the even CTA's barriers), 1 = MMA issuer (even CTA only), 2..5 = output,
// 6..9 = builders of the LoRA operands.
// Two TMEM accumulators of 256 columns, so the output of a tile overlaps the MMAs of the next.
//
// LoRA: after a tile's k-blocks come stages whose A operand is B_all[slot, rows of the tile] and whose B operand is
// scale * u of the tokens that use the adapter.  The builder warps of each CTA list the tile's adapters and write their half
// of those operands to shared memory while the tile's own MMAs run (they have that long; done by the output warps, between two
// tiles, it held the tensor pipe up).  The room holds a number of adapters at a time ("batch").
//
// Every wait on an mbarrier is bounded, and the warps of a role that meet at a named barrier leave together or not at all
// (bar_all); on expiry the CTA records a code in the status word, stops issuing work and goes to the teardown,
// where the pair meets before either CTA leaves or frees its TMEM.
#include <atomic>

#include "linear_tc.cuh"

namespace mlora {
namespace {

constexpr int pair_threads(bool lora) { return lora ? 320 : 192; }
constexpr int kPairN = 256;                       // widest token tile
constexpr int kPairABytes = BM * BK * 2;          // weight rows of one CTA, one k-block
constexpr int kPairStage = 2 * kPairABytes;       // + half of a 256-token tile
constexpr int kPairCache = 32 * 1024;             // a CTA's half of the LoRA operands
constexpr int kPairOut = 2 * 32 * BM * 2;         // two output chunks of 32 tokens
constexpr int kPairAux = 256 + 3 * kPairN * 4 + 16 * 16 + 64 + kPairN * 16;
constexpr int pair_stages(bool lora) { return (227 * 1024 - 1024 - 64 - kPairOut - kPairAux - (lora ? kPairCache : 0)) / kPairStage; }
constexpr int pair_smem(bool lora) { return 1024 + pair_stages(lora) * kPairStage + (lora ? kPairCache : 0) + kPairOut + kPairAux; }

struct PairParams {
  LinearArgs a;
  Groups g;        // GRP only
  int k_blocks, row_tiles, row_pairs, bn, tok_tiles;
  int gt;          // token tiles per group of the walk
  int w_image, b_image;  // the maps of W / B_all see the packed image (rows of 128 bytes) instead of the matrix
  int lora_sub, n_sub;
  int tma_store;
  int32_t* status;
};

// ---- pair-wide PTX -----------------------------------------------------------------------------------
// the even CTA's copy of a shared-memory object, as a shared::cluster address
__device__ __forceinline__ uint32_t lead_addr(const void* p) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(smem_u32(p)));
  return r;
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(addr) : "memory");
}
__device__ __forceinline__ bool mbar_wait_pair(const void* bar, uint32_t parity, volatile int* abort) {
  const uint32_t addr = smem_u32(bar);
  for (uint32_t i = 0; i < kSpinLimit; ++i) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(addr), "r"(parity)
        : "memory");
    if (ok) return true;
    if ((i & 255) == 255 && *abort) return false;
  }
  return false;
}
// TMA load into this CTA's shared memory that completes on a barrier of the even CTA
__device__ __forceinline__ void tma_load_2d_pair(void* dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
      ::"r"(smem_u32(dst)), "l"(map), "r"(x), "r"(y), "r"(bar)
      : "memory");
}
__device__ __forceinline__ void tma_gather4_pair(void* dst, const CUtensorMap* map, int x, const int4& rows, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile::gather4.mbarrier::complete_tx::bytes [%0], "
      "[%1, {%2, %3, %4, %5, %6}], [%7];"
      ::"r"(smem_u32(dst)), "l"(map), "r"(x), "r"(rows.x), "r"(rows.y), "r"(rows.z), "r"(rows.w), "r"(bar)
      : "memory");
}
__device__ __forceinline__ void umma_bf16_pair(uint32_t d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(acc)
      : "memory");
}
// arrives at the barrier of this offset in both CTAs once the MMAs issued so far have retired
__device__ __forceinline__ void umma_commit_pair(uint32_t addr) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
               ::"r"(addr), "h"((uint16_t)3)
               : "memory");
}

// Tile `idx` of the walk.  The token tiles are taken in groups of `gt`; within a group the tiles are ordered row pair major,
// token tile minor and pair w takes tiles w, w + pairs, ...: the tiles in flight at one time are all token tiles of a group
// against a handful of neighbouring row pairs, so both operands come from L2 but for their first use.
struct PairTile {
  int row_pair, tok_tile;
};
__device__ __forceinline__ PairTile pair_tile(const PairParams& p, int idx, int tok_tiles) {
  const int per = p.gt * p.row_pairs;
  const int grp = idx / per, rem = idx - grp * per;
  const int w = min(p.gt, tok_tiles - grp * p.gt);
  const int row = rem / w;
  return PairTile{row, grp * p.gt + (rem - row * w)};
}
// Row tile of this CTA in a row pair, or -1, and the pair's module.  A pair never spans two modules (their LoRA operands
// differ): a module with an odd number of row tiles ends in a pair of one.
struct PairRows {
  int tile, module;
};
__device__ __forceinline__ PairRows pair_rows(const PairParams& p, int row_pair, int rank) {
  int m = 0, first = 0, end = p.row_tiles;
  if (p.a.n_mod > 1) {
#pragma unroll 1
    for (;; ++m) {
      first = p.a.mod_off[m] / BM;
      end = m + 1 < p.a.n_mod ? p.a.mod_off[m + 1] / BM : p.row_tiles;
      const int n = (end - first + 1) / 2;
      if (row_pair < n || m + 1 >= p.a.n_mod) break;
      row_pair -= n;
    }
  }
  const int t = first + 2 * row_pair + rank;
  return PairRows{t < end ? t : -1, m};
}

template <bool LORA, bool GRP>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(pair_threads(LORA), 1)
    linear_pair_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x,
                       const __grid_constant__ CUtensorMap map_b, const __grid_constant__ CUtensorMap map_y, PairParams p) {
  constexpr int NS = pair_stages(LORA);
  extern __shared__ uint8_t smem_raw[];
  uint8_t* ring = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint8_t* s_cache = ring + NS * kPairStage;
  uint8_t* s_out = s_cache + (LORA ? kPairCache : 0);
  uint8_t* aux = s_out + kPairOut;
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(aux);  // [NS]  even CTA's are used: both CTAs' copies of a stage have landed
  uint64_t* empty_bar = full_bar + NS;                    // [NS]  the stage's MMAs have retired
  uint64_t* acc_full = empty_bar + NS;                    // [2]
  uint64_t* acc_empty = acc_full + 2;                     // [2]   even CTA's: eight output warps
  uint64_t* info_bar = acc_empty + 2;                     // the tile's adapters are listed (own CTA)
  uint64_t* info_empty = info_bar + 1;                    // the producer has read the list (own CTA)
  uint64_t* cache_full = info_empty + 1;                  // even CTA's: both halves of a batch of LoRA operands are written
  uint64_t* cache_empty = cache_full + 1;                 // the MMAs of a batch have retired
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(cache_empty + 1);
  int* s_slots = reinterpret_cast<int*>(aux + 256);       // [256]
  int* s_list = s_slots + kPairN;                         // [256] distinct adapters of the token tile
  float* s_scale = reinterpret_cast<float*>(s_list + kPairN);
  int4* s_tab = reinterpret_cast<int4*>(s_scale + kPairN);  // [16] run layout: (first column, rows, row offset of the operand)
  int* s_info = reinterpret_cast<int*>(s_tab + 16);       // adapters, run layout?, adapters per batch, operand rows of the run layout
  int4* s_loc = reinterpret_cast<int4*>(s_info + 16);     // [256] run layout, per operand row of this CTA: (token row or -1,
                                                          //       its position in rows, rows of the run, scale)
  __shared__ int s_abort;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int rank = (int)cluster_rank();
  const int worker = (int)blockIdx.x >> 1, workers = (int)gridDim.x >> 1;
  const LinearArgs& a = p.a;
  int tok_tiles = p.tok_tiles;
  if constexpr (GRP) {
    if (p.g.table != nullptr) {
      pdl_wait();  // the table is written by the kernel before this one
      tok_tiles = p.g.table[0];
    }
  }
  const int n_tiles = tok_tiles * p.row_pairs;
  if (worker >= n_tiles) return;  // the whole pair (uniform)

  if (tid == 0) {
    s_abort = 0;
    for (int s = 0; s < NS; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&acc_full[b], 1);
      mbar_init(&acc_empty[b], 8);
    }
    mbar_init(info_bar, 1);
    mbar_init(info_empty, 1);
    mbar_init(cache_full, 2);
    mbar_init(cache_empty, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    tma_prefetch_desc(&map_w);
    tma_prefetch_desc(&map_x);
    if (LORA) tma_prefetch_desc(&map_b);
    if (p.tma_store) tma_prefetch_desc(&map_y);
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(2 * kPairN)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync();
  tc_fence_after();
  pdl_launch_dependents();
  pdl_wait();
  const uint32_t tmem_base = *tmem_slot;
  const int half = p.bn >> 1;                      // tokens staged by each CTA
  const uint32_t rb = LORA ? p.lora_sub * 2 : 32;  // row bytes of a LoRA operand
  const int group = kPairABytes / (BM * (int)rb);  // LoRA A operands per ring slot

  if (warp == 0) {
    // ---- operand producer (one thread; the whole warp where rows are gathered) ---------------------
    if (lane == 0 || (GRP && p.g.gather != nullptr)) {
      const uint32_t full0 = lead_addr(full_bar);
      const uint32_t tx = 2 * (kPairABytes + half * BK * 2);
      int s = 0, n_lora = 0;
      uint32_t par = 1;
      bool ok = true;
      auto stage = [&](uint32_t bytes) {  // waits for the slot and announces the pair's bytes
        if (lane == 0) {
          if (!mbar_wait_pair(&empty_bar[s], par, &s_abort)) {
            s_abort = 1;
            atomicOr(p.status, 1);
            ok = false;
          } else if (rank == 0) {
            mbar_expect_tx(&full_bar[s], bytes);
          }
        }
        if (GRP && p.g.gather != nullptr) ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
        return ok;
      };
      auto next = [&]() {
        if (++s == NS) {
          s = 0;
          par ^= 1;
        }
      };
      for (int idx = worker; idx < n_tiles && ok; idx += workers) {
        const PairTile pt = pair_tile(p, idx, tok_tiles);
        PairRows pr = pair_rows(p, pt.row_pair, rank);
        if (pr.tile < 0) pr.tile = pair_rows(p, pt.row_pair, 0).tile;  // a pair of one: the odd CTA repeats it, and stores nothing
        int x_row = pt.tok_tile * p.bn + rank * half, x_col = 0, w_row = 0;
        int4 src = make_int4(0, 0, 0, 0);
        if constexpr (GRP) {
          const GroupTile gt = group_tile(p.g, p.a.T, pt.tok_tile, p.bn);
          x_row = gt.row0 + rank * half;
          x_col = gt.group * p.g.x_cols;
          w_row = gt.group * (p.row_tiles * p.k_blocks * BM);
          if (p.g.gather != nullptr) {  // half = 128 rows, four per lane; rows past the tile's last repeat it (not stored)
            const int r = rank * half + lane * 4;
            const int32_t* gi = p.g.gather + gt.row0;
            src = make_int4(gi[min(r, gt.rows - 1)], gi[min(r + 1, gt.rows - 1)], gi[min(r + 2, gt.rows - 1)], gi[min(r + 3, gt.rows - 1)]);
          }
        }
        w_row += pr.tile * (p.w_image ? p.k_blocks * BM : BM);
        for (int kb = 0; kb < p.k_blocks; ++kb) {
          if (!stage(tx)) break;
          uint8_t* st = ring + s * kPairStage;
          const uint32_t bar = full0 + 8 * s;
          if (lane == 0) {
            tma_load_2d_pair(st, &map_w, p.w_image ? 0 : kb * BK, p.w_image ? w_row + kb * BM : w_row, bar);
            if (!GRP || p.g.gather == nullptr) tma_load_2d_pair(st + kPairABytes, &map_x, x_col + kb * BK, x_row, bar);
          }
          if constexpr (GRP) {
            if (p.g.gather != nullptr) tma_gather4_pair(st + kPairABytes + lane * 512, &map_x, x_col + kb * BK, src, bar);
          }
          next();
        }
        if constexpr (LORA) {
          if (!ok) break;
          if (!mbar_wait_pair(info_bar, n_lora & 1, &s_abort)) {
            s_abort = 1;
            atomicOr(p.status, 32);
            break;
          }
          ++n_lora;
          const int n_seg = s_info[0], per_batch = s_info[2];
          for (int j0 = 0; j0 < n_seg && ok; j0 += per_batch) {
            const int l1 = min(n_seg, j0 + per_batch) * p.n_sub;
            for (int l0 = j0 * p.n_sub; l0 < l1; l0 += group) {
              const int n = min(l1 - l0, group);
              if (!stage(2 * n * BM * rb)) break;
              for (int l = l0; l < l0 + n; ++l) {
                const int slot = s_list[l / p.n_sub], sb = l % p.n_sub;
                uint8_t* dst = ring + s * kPairStage + (l - l0) * BM * rb;
                if (p.b_image)  // a tile is BM * rb contiguous bytes = rb rows of 128
                  tma_load_2d_pair(dst, &map_b, 0, ((slot * p.row_tiles + pr.tile) * p.n_sub + sb) * (int)rb, full0 + 8 * s);
                else
                  tma_load_2d_pair(dst, &map_b, sb * p.lora_sub, slot * a.out + pr.tile * BM, full0 + 8 * s);
              }
              next();
            }
          }
          mbar_arrive(info_empty);
        }
      }
      // the even CTA's last commits arrive in both CTAs: none of those arrivals may be on its way when a CTA leaves
      for (int i = 0; i < NS && lane == 0 && ok && !s_abort; ++i, next()) {
        if (!mbar_wait_pair(&empty_bar[s], par, &s_abort)) {
          s_abort = 1;
          atomicOr(p.status, 1);
        }
      }
    }
  } else if (warp == 1) {
    // ---- MMA issuer: one thread of the even CTA ----------------------------------------------------
    if (rank == 0 && lane == 0) {
      const uint32_t idesc = make_idesc(2 * BM, p.bn);
      const uint32_t full0 = smem_u32(full_bar), empty0 = smem_u32(empty_bar);
      const uint64_t adesc0 = make_smem_desc(smem_u32(ring)), bdesc0 = make_smem_desc(smem_u32(ring + kPairABytes));
      int s = 0, j = 0, n_batch = 0;
      uint32_t par = 0;
      bool ok = true;
      for (int idx = worker; idx < n_tiles && ok; idx += workers, ++j) {
        const int buf = j & 1;
        const uint32_t d_tmem = tmem_base + buf * kPairN;
        if (!mbar_wait_pair(&acc_empty[buf], ((j >> 1) & 1) ^ 1, &s_abort)) {
          s_abort = 1;
          atomicOr(p.status, 8);
          break;
        }
        tc_fence_after();
        for (int kb = 0; kb < p.k_blocks; ++kb) {
          if (!mbar_wait_a(full0 + 8 * s, par, &s_abort)) {
            s_abort = 1;
            atomicOr(p.status, 2);
            ok = false;
            break;
          }
          tc_fence_after();
          const uint64_t adesc = adesc0 + (uint64_t)(s * (kPairStage >> 4)), bdesc = bdesc0 + (uint64_t)(s * (kPairStage >> 4));
          umma_bf16_pair(d_tmem, adesc, bdesc, idesc, kb > 0 ? 1u : 0u);
#pragma unroll
          for (int k = 1; k < BK / 16; ++k) umma_bf16_pair(d_tmem, adesc + 2 * k, bdesc + 2 * k, idesc, 1u);
          umma_commit_pair(empty0 + 8 * s);
          if (++s == NS) {
            s = 0;
            par ^= 1;
          }
        }
        if constexpr (LORA) {
          int n_seg = 0, runs = 0, per_batch = 1;
          bool first = true;
          for (int j0 = 0; ok && (first || j0 < n_seg); j0 += per_batch) {
            if (!mbar_wait_pair(cache_full, n_batch & 1, &s_abort)) {
              s_abort = 1;
              atomicOr(p.status, 64);
              ok = false;
              break;
            }
            ++n_batch;
            tc_fence_after();
            if (first) {
              n_seg = s_info[0];
              runs = s_info[1];
              per_batch = s_info[2];
              first = false;
            }
            const int l1 = min(n_seg, j0 + per_batch) * p.n_sub;
            for (int l0 = j0 * p.n_sub; l0 < l1; l0 += group) {
              if (!mbar_wait_a(full0 + 8 * s, par, &s_abort)) {
                s_abort = 1;
                atomicOr(p.status, 2);
                ok = false;
                break;
              }
              tc_fence_after();
              for (int l = l0; l < min(l1, l0 + group); ++l) {
                const int sgi = l / p.n_sub, sb = l - sgi * p.n_sub;
                const uint64_t adesc = make_smem_desc(smem_u32(ring + s * kPairStage + (l - l0) * BM * rb), rb);
                // run layout: the adapter's own 16-row blocks only, half of them in each CTA; else the whole tile, masked
                const int4 tb = runs ? s_tab[sgi] : make_int4(0, p.bn, (sgi - j0) * half, 0);
                const uint64_t bdesc = make_smem_desc(smem_u32(s_cache + (size_t)(tb.z * p.n_sub + sb * (tb.y >> 1)) * rb), rb);
                const uint32_t idesc_l = make_idesc(2 * BM, tb.y);
                for (int k = 0; k < p.lora_sub / 16; ++k) umma_bf16_pair(d_tmem + tb.x, adesc + 2 * k, bdesc + 2 * k, idesc_l, 1u);
              }
              umma_commit_pair(empty0 + 8 * s);
              if (++s == NS) {
                s = 0;
                par ^= 1;
              }
            }
            if (ok) umma_commit_pair(smem_u32(cache_empty));
          }
        }
        if (ok) umma_commit_pair(smem_u32(&acc_full[buf]));
      }
    }
  } else if (!LORA || warp < 6) {
    // ---- output warps 2..5: TMEM lane quarter = warp % 4 -------------------------------------------
    const int q = warp & 3;
    const int etid = q * 32 + lane;  // 0..127 = weight row inside the CTA's row tile
    const bool silu = (a.flags & MLORA_SILU_MUL) != 0;
    const int act = a.flags & (MLORA_ACT_RELU2 | MLORA_ACT_GELU);
    const uint32_t acc_empty_lead = lead_addr(acc_empty);
    int j = 0, n_out = 0;

    for (int idx = worker; idx < n_tiles; idx += workers, ++j) {
      const PairTile pt = pair_tile(p, idx, tok_tiles);
      const PairRows pr = pair_rows(p, pt.row_pair, rank);
      const int buf = j & 1;
      int t0 = pt.tok_tile * p.bn, t_end = min(a.T, t0 + p.bn), y_col = 0, grp = 0;
      if constexpr (GRP) {
        const GroupTile gt = group_tile(p.g, p.a.T, pt.tok_tile, p.bn);
        t0 = gt.row0;
        t_end = gt.row0 + gt.rows;
        grp = gt.group;
        y_col = gt.group * p.g.y_cols;
      }
      if (!bar_all(1, mbar_wait_pair(&acc_full[buf], (j >> 1) & 1, &s_abort))) {
        if (!s_abort) {
          s_abort = 1;
          atomicOr(p.status, 4);
        }
        break;
      }
      tc_fence_after();
      const uint32_t t_addr = tmem_base + ((uint32_t)(q * 32) << 16) + buf * kPairN;
      const int row = pr.tile * BM + etid;
#pragma unroll 1
      for (int c0 = 0; c0 < p.bn; c0 += 32) {
        float v[32];
        tmem_ld32(t_addr + c0, v);
        if (c0 + 32 >= p.bn) {  // accumulator fully read: hand it back to the MMA thread
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive_cluster(acc_empty_lead + 8 * buf);
        }
        if (pr.tile < 0 || t0 + c0 >= t_end) continue;  // (uniform over the output warps)
        if constexpr (!LORA) apply_act<32>(v, act);
        if constexpr (GRP) {
          if (p.g.gate != nullptr) {  // one row's gate per lane, handed round
            const int t = t0 + c0 + lane;
            float gt = 0.f;
            if (t < t_end) gt = __fdividef(1.f, 1.f + __expf(-__bfloat162float(p.g.gate[(size_t)t * p.g.ld_gate + grp])));
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] *= __shfl_sync(0xffffffffu, gt, i);
          }
        }
        if (p.tma_store) {
          // registers -> shared memory [tokens][outputs of the tile] -> one TMA store.  Plain: the map clips tokens >= T and
          // outputs >= out.  Grouped: a chunk must not touch the rows or columns of the next group, so only whole ones leave
          // by TMA, ragged ones row by row with 16-byte stores.
          if (etid == 0) asm volatile("cp.async.bulk.wait_group.read 1;" ::: "memory");  // the chunk before last has been read
          __syncwarp();
          epi_bar_sync();
          bf16* so = reinterpret_cast<bf16*>(s_out + (n_out++ & 1) * (kPairOut / 2));
          if (!GRP && silu) {
#pragma unroll
            for (int i = 0; i < 32; ++i) {
              const float other = __shfl_xor_sync(0xffffffffu, v[i], 8);
              if ((etid & 8) == 0) so[i * (BM / 2) + (etid >> 4) * 8 + (etid & 7)] = __float2bfloat16_rn(silu_mul(v[i], other));
            }
          } else {
#pragma unroll
            for (int i = 0; i < 32; ++i) so[i * BM + etid] = __float2bfloat16_rn(v[i]);
          }
          if (!GRP || (t0 + c0 + 32 <= t_end && pr.tile * BM + BM <= a.out)) {
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            epi_bar_sync();
            if (etid == 0) tma_store_2d(&map_y, so, y_col + (silu ? pr.tile * (BM / 2) : pr.tile * BM), t0 + c0);
          } else {
            if (etid == 0) asm volatile("cp.async.bulk.commit_group;" ::: "memory");  // (an empty group: the count above stays right)
            epi_bar_sync();
            bf16* y = reinterpret_cast<bf16*>(a.y);
            for (int i = etid; i < 32 * (BM / 8); i += kEpiThreads) {
              const int t = t0 + c0 + i / (BM / 8), col = pr.tile * BM + (i % (BM / 8)) * 8;
              if (t < t_end && col < a.out)
                *reinterpret_cast<uint4*>(y + (size_t)t * a.ldy + y_col + col) = reinterpret_cast<const uint4*>(so)[i];
            }
            epi_bar_sync();  // read before the buffer's turn comes again
          }
          continue;
        }
#pragma unroll
        for (int i = 0; i < 32; ++i) {
          const int t = t0 + c0 + i;
          const bool live = t < t_end && row < a.out;
          if (!GRP && silu) {
            const float other = __shfl_xor_sync(0xffffffffu, v[i], 8);
            if (live && (etid & 8) == 0) store_out(a, t, (row >> 4) * 8 + (row & 7), silu_mul(v[i], other));
          } else if (live) {
            store_out(a, t, y_col + row, v[i]);
          }
        }
      }
    }
    if (p.tma_store && etid == 0) bulk_wait_read0();  // shared memory must stay valid until the stores have read it
  } else if constexpr (LORA) {
    // ---- builders 6..9 -----------------------------------------------------------------------------
    const int bt = tid - 6 * 32;
    const uint32_t cache_lead = lead_addr(cache_full);
    const int r_tot = a.r_max * a.n_mod;
    const int chunk_log = 31 - __clz(p.lora_sub / 8), row_log = 31 - __clz(a.r_max / 8);  // 16-byte chunks of a slice / of a row
    int e_tok = -1, e_key = -1, n_batch = 0, j = 0;
    bool ok = true;
    auto bar = [] {
      __syncwarp();
      asm volatile("bar.sync 2, 128;" ::: "memory");
    };
    // one lane waits for its warp; the four warps go on, or give up, together
    auto wait = [&](uint64_t* b, uint32_t parity) {
      int w = 1;
      if (lane == 0) w = mbar_wait_pair(b, parity, &s_abort) ? 1 : 0;
      w = __shfl_sync(0xffffffffu, w, 0);
      if (!w) {
        s_abort = 1;
        atomicOr(p.status, 32);
      }
      return bar_all(2, w != 0);
    };
    for (int idx = worker; idx < n_tiles && ok; idx += workers, ++j) {
      const PairTile pt = pair_tile(p, idx, tok_tiles);
      const int module = pair_rows(p, pt.row_pair, rank).module;
      const int t0 = pt.tok_tile * p.bn, tile_rows = min(a.T - t0, p.bn);
      // the previous tile's list has been read by the producer, and by the MMA thread with the last batch
      if (j > 0 && !(wait(info_empty, (j - 1) & 1) && wait(cache_empty, (n_batch - 1) & 1))) break;
      if (pt.tok_tile != e_tok) {
        bar();
        if (warp == 6) {
          const int n_seg = distinct_slots_n(a, t0, tile_rows, kPairN, s_slots, s_list);
          const int n_run = adapter_runs_n(kPairN, s_slots, s_list, n_seg, s_tab);
          for (int i = lane; i < n_seg; i += 32) s_scale[i] = a.scales[s_list[i]];
          const bool runs = n_run >= 0 && n_run * p.n_sub * (int)rb <= 2 * kPairCache;
          __syncwarp();
          if (runs && lane < n_seg) s_tab[lane].z >>= 1;  // rows per CTA
          if (lane == 0) {
            s_info[0] = n_seg;
            s_info[1] = runs ? 1 : 0;
            s_info[2] = runs ? max(n_seg, 1) : kPairCache / (half * p.n_sub * (int)rb);
            s_info[3] = n_run >> 1;
          }
        }
        bar();
        if (s_info[1]) {
          for (int lr = bt; lr < s_info[3]; lr += 128) {
            int sg = 0;
            while (sg + 1 < s_info[0] && lr >= s_tab[sg + 1].z) ++sg;
            const int4 tb = s_tab[sg];
            const int local = lr - tb.z, row = tb.x + rank * (tb.y >> 1) + local;
            s_loc[lr] = make_int4(s_slots[row] == s_list[sg] ? row : -1, tb.z * p.n_sub + local, tb.y >> 1, __float_as_int(s_scale[sg]));
          }
          bar();
        }
        e_tok = pt.tok_tile;
        e_key = -1;
      }
      if (bt == 0) mbar_arrive(info_bar);
      const int n_seg = s_info[0], per_batch = s_info[2];
      const bool runs = s_info[1] != 0;
      for (int j0 = 0; j0 == 0 || j0 < n_seg; j0 += per_batch) {
        const int n_ad = min(n_seg - j0, per_batch);
        if (j0 > 0 && !wait(cache_empty, (n_batch - 1) & 1)) {  // the batch before is still being read
          ok = false;
          break;
        }
        if (module != e_key) {
          // scale * u of the rows that use the adapter, zero for the others, swizzled K-major; four items per thread and
          // step, their shrink outputs (L2 round trips) requested before the first is used
          const int items = (runs ? s_info[3] : n_ad * half) << row_log;
          for (int base = bt; base < items; base += 128 * 4) {
            float4 lo[4], hi[4];
            float sc[4];
            int at[4];
#pragma unroll
            for (int b = 0; b < 4; ++b) {
              const int i = base + b * 128;
              at[b] = -1;
              if (i >= items) continue;
              const int lr = i >> row_log, rem = i & ((1 << row_log) - 1), sb = rem >> chunk_log, c = rem & ((1 << chunk_log) - 1);
              int row, pos;
              if (runs) {
                const int4 e = s_loc[lr];
                row = e.x;
                pos = e.y + sb * e.z;
                sc[b] = __int_as_float(e.w);
              } else {
                const int sg = lr / half, local = lr - sg * half;
                row = rank * half + local;
                if (s_slots[row] != s_list[j0 + sg]) row = -1;
                pos = sg * half * p.n_sub + sb * half + local;
                sc[b] = s_scale[j0 + sg];
              }
              const int sw = rb == 128 ? (pos & 7) : rb == 64 ? ((pos >> 1) & 3) : ((pos >> 2) & 1);
              at[b] = pos * (int)rb + ((c ^ sw) << 4);
              lo[b] = hi[b] = make_float4(0.f, 0.f, 0.f, 0.f);
              if (row >= 0) {
                const float* ur = a.u + (size_t)(t0 + row) * r_tot + module * a.r_max + sb * p.lora_sub + c * 8;
                lo[b] = *reinterpret_cast<const float4*>(ur);
                hi[b] = *reinterpret_cast<const float4*>(ur + 4);
              }
            }
#pragma unroll
            for (int b = 0; b < 4; ++b) {
              if (at[b] < 0) continue;
              const float f[8] = {lo[b].x * sc[b], lo[b].y * sc[b], lo[b].z * sc[b], lo[b].w * sc[b],
                                  hi[b].x * sc[b], hi[b].y * sc[b], hi[b].z * sc[b], hi[b].w * sc[b]};
              *reinterpret_cast<uint4*>(s_cache + at[b]) = pack8(f);
            }
          }
          if (n_seg <= per_batch) e_key = module;
        }
        asm volatile("fence.proxy.async;" ::: "memory");
        bar();
        if (bt == 0) mbar_arrive_cluster(cache_lead);
        ++n_batch;
      }
    }
    if (ok) wait(cache_empty, (n_batch - 1) & 1);  // (as for the ring: the last batch's commit arrives in both CTAs)
  }

  // ---- teardown: the peer's copies, MMAs and arrivals reach into this CTA until the pair has met -------
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (s_abort) {
    for (int i = 0; i < 64; ++i) __nanosleep(1000);  // copies that may still be in flight land
  }
  cluster_sync();
  tc_fence_after();
  if (warp == 1)
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(2 * kPairN) : "memory");
}

// ---- host side -------------------------------------------------------------------------------------
struct PairPlan {
  int bn, tok_tiles, row_pairs, gt;
  long long cost;  // tensor or shared-memory cycles of the busiest pair
};

// Token tiles of up to 256 rows: the width (a multiple of 32) whose tiles fill whole rounds of the pairs best.  A k-block of a
// tile of bn tokens costs 2 bn cycles of MMA or 256 + bn of shared memory, whichever is longer.
PairPlan pair_plan(int T, int in, int row_pairs) {
  const int pairs = sm_count() / 2, k_blocks = (in + BK - 1) / BK;
  PairPlan best{};
  best.cost = -1;
  for (int bn = kPairN; bn >= 64; bn -= 32) {
    PairPlan pl;
    pl.bn = bn;
    pl.row_pairs = row_pairs;
    pl.tok_tiles = (T + bn - 1) / bn;
    const long long steps = ((long long)pl.tok_tiles * row_pairs + pairs - 1) / pairs;
    pl.cost = steps * k_blocks * (2 * bn > 256 + bn ? 2 * bn : 256 + bn);
    // token tiles of a group: resident in L2 next to the weight tiles in flight (<= 48 MB of 126), groups of equal width
    const double tile = (double)bn * in * 2.0;
    int most = 16;
    while (most > 1 && most * tile > 48e6) --most;
    const int groups = (pl.tok_tiles + most - 1) / most;
    pl.gt = (pl.tok_tiles + groups - 1) / groups;
    if (best.cost < 0 || pl.cost < best.cost) best = pl;
  }
  return best;
}

template <bool LORA, bool GRP>
int launch_pair(const CUtensorMap& mw, const CUtensorMap& mx, const CUtensorMap& mb, const CUtensorMap& my, const PairParams& p, int grid,
                cudaStream_t st) {
  // the shared-memory opt-in is a per-device attribute
  static std::atomic<unsigned long long> attr_done{0};
  int dev = 0;
  cudaGetDevice(&dev);
  if (!((attr_done.load(std::memory_order_acquire) >> (dev & 63)) & 1ull)) {
    cudaError_t e = cudaFuncSetAttribute(linear_pair_kernel<LORA, GRP>, cudaFuncAttributeMaxDynamicSharedMemorySize, pair_smem(LORA));
    if (e != cudaSuccess) return fail(MLORA_ECUDA, "linear: cudaFuncSetAttribute: %s", cudaGetErrorString(e));
    attr_done.fetch_or(1ull << (dev & 63), std::memory_order_release);
  }
  launch_pdl_if(pdl_enabled_gemm(), linear_pair_kernel<LORA, GRP>, grid, pair_threads(LORA), pair_smem(LORA), st, mw, mx, mb, my, p);
  count_launch();
  MLORA_CHECK_LAUNCH("linear_pair_kernel");
  return MLORA_OK;
}

// A packed operand as rows of 128 bytes (no swizzle: the image already is what the MMA reads), `box` rows to a tile.
int make_image_map(CUtensorMap* m, const void* ptr, long long bytes, int box) {
  return make_out_map(m, const_cast<void*>(ptr), (int)(bytes / 128), 64, 64, box, 64, false);
}

int pair_row_pairs(const LinearArgs& a) {
  const int row_tiles = (a.out + BM - 1) / BM;
  if (a.n_mod <= 1) return (row_tiles + 1) / 2;
  int n = 0;
  for (int m = 0; m < a.n_mod; ++m) {
    const int end = m + 1 < a.n_mod ? a.mod_off[m + 1] / BM : row_tiles;
    n += (end - a.mod_off[m] / BM + 1) / 2;
  }
  return n;
}

}  // namespace

// When pairs are faster than the one-CTA kernel, which splits a tile's k-blocks over CTAs where there are few tiles: from
// three quarters of the pairs busy with tiles of 128 tokens.  Measured, one CTA -> pairs (us): 4096 -> 12288 at T = 160
// (96 tiles) 44 -> 31, 1024 151 -> 78; 2048 -> 8192 at 160 (64) 29 -> 23; 4096 -> 4096 at 256 (32) 26 -> 34, 384 (48) 36 -> 36,
// 512 (64) 40 -> 37, 1024 67 -> 41; 11008 -> 4096 at 384 (48) 67 -> 76, 512 (64) 83 -> 78, 1024 141 -> 78.
bool linear_pair_supported(const LinearArgs& a) {
  if (a.T <= 128) return false;
  if (a.u != nullptr) {  // the expand runs on the tensor cores only (the other forms: linear_tc.cu)
    if (!(a.r_max == 16 || a.r_max == 32 || a.r_max == 64 || a.r_max == 128)) return false;
    for (int m = 1; m < a.n_mod; ++m)
      if (a.mod_off[m] % BM != 0) return false;
  }
  return 4ll * ((a.T + 127) / 128) * pair_row_pairs(a) >= 3ll * (sm_count() / 2);
}

void linear_pair_plan(const LinearArgs& a, int32_t* v) {
  const PairPlan pl = pair_plan(a.T, a.in, pair_row_pairs(a));
  const long long tiles = (long long)pl.tok_tiles * pl.row_pairs;
  v[0] = pl.bn;
  v[1] = (int)(tiles < sm_count() / 2 ? tiles : sm_count() / 2);
  v[2] = (a.out + BM - 1) / BM;
  v[3] = pl.tok_tiles;
  v[4] = pl.row_pairs;
  v[5] = pl.gt;
}

int launch_linear_pair(const LinearArgs& a, void* work, cudaStream_t st) {
  PairParams p{};
  p.a = a;
  p.row_tiles = (a.out + BM - 1) / BM;
  p.k_blocks = (a.in + BK - 1) / BK;
  const PairPlan pl = pair_plan(a.T, a.in, pair_row_pairs(a));
  p.row_pairs = pl.row_pairs;
  p.bn = pl.bn;
  p.tok_tiles = pl.tok_tiles;
  p.gt = pl.gt;
  p.status = (int32_t*)work;
  CUtensorMap mw, mx, mb, my;
  int rc = make_map(&mx, a.x, a.T, a.in, a.ldx, p.bn / 2);
  if (rc) return rc;
  p.w_image = (a.flags & MLORA_W_PACKED) != 0;
  rc = p.w_image ? make_image_map(&mw, a.W, (long long)packed_weight_bytes(a.out, a.in), BM) : make_map(&mw, a.W, a.out, a.in, a.in, BM);
  if (rc) return rc;
  mb = mw;
  my = mx;
  if (a.u != nullptr) {
    p.lora_sub = a.r_max < 64 ? a.r_max : 64;
    p.n_sub = a.r_max / p.lora_sub;
    p.b_image = (a.flags & MLORA_B_PACKED) != 0;
    rc = p.b_image ? make_image_map(&mb, a.B_all, (long long)packed_lora_b_bytes(a.n_adapters, a.out, a.r_max), p.lora_sub * 2)
                   : make_map(&mb, a.B_all, (long long)a.n_adapters * a.out, a.r_max, a.r_max, BM, p.lora_sub);
    if (rc) return rc;
  }
  const bool f32 = (a.flags & MLORA_OUT_F32) != 0, silu = (a.flags & MLORA_SILU_MUL) != 0;
  const int cols = silu ? a.out / 2 : a.out;
  p.tma_store = !f32 && aligned16(a.y) && a.ldy % 8 == 0 && cols % 8 == 0;
  if (p.tma_store) {
    rc = make_out_map(&my, a.y, a.T, cols, a.ldy, 32, silu ? BM / 2 : BM, false);
    if (rc) return rc;
  }
  const long long tiles = (long long)p.tok_tiles * p.row_pairs;
  const int pairs = sm_count() / 2, grid = 2 * (int)(tiles < pairs ? tiles : pairs);
  return a.u != nullptr ? launch_pair<true, false>(mw, mx, mb, my, p, grid, st) : launch_pair<false, false>(mw, mx, mb, my, p, grid, st);
}

// Grouped form, 256-row tiles.
int launch_grouped_pair(const GroupedArgs& ga, void* work, cudaStream_t st) {
  const LinearArgs& a = ga.a;
  PairParams p{};
  p.a = a;
  p.row_tiles = (a.out + BM - 1) / BM;
  p.row_pairs = (p.row_tiles + 1) / 2;
  p.k_blocks = (a.in + BK - 1) / BK;
  p.bn = kPairN;
  p.gt = 1;  // neighbouring pairs share a token tile and walk the weight of one group
  p.w_image = 1;
  p.lora_sub = 16;
  p.n_sub = 1;
  p.g.table = ga.table;
  p.g.gather = ga.gather;
  p.g.tiles_per_group = ga.table ? 1 : (a.T + kPairN - 1) / kPairN;
  p.g.x_cols = ga.x_cols;
  p.g.y_cols = ga.y_cols;
  p.g.gate = ga.gate;
  p.g.ld_gate = ga.ld_gate;
  p.tok_tiles = ga.table ? 0 : ga.n_groups * p.g.tiles_per_group;
  p.status = (int32_t*)work;
  CUtensorMap mw, mx, my;
  int rc = make_map(&mx, a.x, ga.x_rows, ga.x_cols ? (int)a.ldx : a.in, a.ldx, ga.gather ? 1 : kPairN / 2);
  if (rc) return rc;
  rc = make_image_map(&mw, a.W, (long long)packed_weight_bytes(a.out, a.in) * ga.n_groups, BM);
  if (rc) return rc;
  my = mx;
  // (a ragged chunk never leaves by TMA, so the map needs no row count)
  p.tma_store = !(a.flags & MLORA_OUT_F32) && aligned16(a.y) && a.ldy % 8 == 0 && ga.y_cols % 8 == 0 && a.out % 8 == 0;
  if (p.tma_store) {
    rc = make_out_map(&my, a.y, 1 << 30, (int)a.ldy, a.ldy, 32, BM, false);
    if (rc) return rc;
  }
  return launch_pair<false, true>(mw, mx, mx, my, p, sm_count() / 2 * 2, st);
}

}  // namespace mlora
