// Decode-size projections (T <= 32) with whole output rows per CTA: y[T,out] = x[T,in] W[out,in]^T (+ LoRA expand, + activation).
//
// What bounds it: the weights' way from HBM, once, and around that the chain of a launch -- rows arrive, products, sums, store.
// The stream-K kernel (linear_tc.cuh) cuts (tile, k-block) ranges, so that nearly every 128-row tile of a narrow projection
// is shared by five CTAs that end at the same time, and its finisher then fetches 16 KB of partial sums from each of the others.
// Here a CTA owns out / SMs rows (in groups of 8, the height of a swizzle atom of the packed weight) over the whole of `in`:
// nothing is handed over through memory.  The price is that every CTA reads all of x from L2: with 32 rows as much as the weights of a
// narrow projection, through the same shared memory.
//
// Tokens are the M operand (16 per mma.sync m16n8k16) and a group of 8 weight rows the N operand: groups of 8 deal 4096 rows
// evenly to 148 SMs, which 128-row tiles with the weights as M cannot, and sums in registers need no way through TMEM.  (tcgen05 with the
// tokens as M would deal them as evenly; it was not built.)  The stream sets the pace, the products cost 1 us at one row and 9 to 16 % at
// 32: without the mma.syncs (a copy that skips them) 4096 -> 12288 takes 18.3 / 19.6 / 20.7 us at 1 / 16 / 32 rows instead of
// 19.4 / 21.0 / 22.6, 4096 -> 4096 12.1 instead of 14.4 at 32, 4096 -> 22016 SiLU*up 32.2 instead of 36.0.
//
// Measured behind a RMSNorm launch (CUDA events over a graph, us for both, stream-K -> this; the weights' bytes at 6458 GB/s):
//              4096 -> 12288    4096 -> 4096    4096 -> 22016 SiLU*up    11008 -> 4096
//    1 row     22.2 -> 19.4     12.6 -> 11.3    35.6 -> 30.2             23.3 -> 21.9
//   16 rows    22.6 -> 21.0     13.3 -> 12.1    36.2 -> 31.8             24.7 -> 24.9 (not taken)
//   32 rows    24.3 -> 22.6     15.4 -> 14.4    39.3 -> 36.0
//   (bytes)    15.6             5.2             27.9                     14.0
// with 16 adapters, behind a shrink, 32 rows: rank 16 4096 -> 12288 30.6 -> 28.4, 4096 -> 4096 17.9 -> 16.9; rank 64 56.1 -> 40.1, 31.3 -> 19.7.
//
// Warps: 0..7 products and output; 8, 9 copies (weights before the kernels in front have completed, token rows after); 10, 11
// (LORA) list the batch's adapters and write scale * u as bf16.  A ring slot holds two to eight k-blocks of the CTA's weight rows
// and of all tokens; a product warp takes 16 columns of every other k-block.  At the end the eight partial sums of an output are
// added in warp order.
//
// LoRA: behind the k-blocks come slots with the CTA's rows of B of some adapters each, which the product warps share out by
// (adapter, 16 ranks) and multiply with u, rows of other adapters masked: the sums go on in the same registers.  In the ring they
// come with the stream; fetched beside it by warps of their own every round trip took 3 to 5 us behind the weights (32 rows,
// 16 rank-64 adapters on 4096 -> 4096: 52 us).
//
// All waits on mbarriers are bounded; a role that gives up raises s_abort, after which no wait waits, every warp still goes
// through all its named barriers, and the status word says that the outputs are undefined.
#include <atomic>

#include "linear_tc.cuh"

namespace mlora {
namespace {

constexpr int kRwProducts = 8;  // product warps
constexpr int kRwMaxSlots = 16;
constexpr int kRwBudget = 227 * 1024 - 1024 /*alignment slack*/ - 64 /*static*/;
constexpr int kRwCopies = 2;    // copy warps, every other ring slot each
constexpr int kRwExpand = 2;    // LORA: warps that stage the adapters' side (twelve warps in all: 168 registers each)
constexpr int rw_threads(bool lora) { return (kRwProducts + kRwCopies + (lora ? kRwExpand : 0)) * 32; }

template <int XR>  // token rows staged: 16 or 32
struct RwCfg {
  static constexpr int MT = XR > 16 ? 2 : 1;       // 16-token tiles
  static constexpr int kMaxG = XR > 16 ? 12 : 20;  // row groups of one pass: up to 96 accumulators per thread
  static constexpr int kXBytes = XR * BK * 2;      // token rows of one k-block
  static constexpr int kRed = kRwProducts * 4 * XR * 8 * 4;  // partial sums of four row groups
  static constexpr int kMaxRank = 192;             // widest row of shrink outputs (all modules)
  static constexpr int kU = XR * (kMaxRank + 8) * 2;
  static constexpr int kAux = 1024;
  static constexpr int ring(bool lora) { return (kRwBudget - kRed - kAux - (lora ? kU : 0)) & ~1023; }
  static constexpr int smem(bool lora) { return 1024 + ring(lora) + kRed + kAux + (lora ? kU : 0); }
  static_assert(kRed >= 4 * 1024, "products past the last group stay inside shared memory");
  static_assert(3 * 2 * (kMaxG * 1024 + kXBytes) <= kRwBudget - kRed - kAux - kU - 1023, "fewer than three ring slots");
};

struct RwParams {
  LinearArgs a;
  int k_blocks, row_tiles;
  int units, unit;      // row groups are dealt in units of 1, or 2 (SiLU: 8 gate rows and their 8 up rows)
  int passes;           // every CTA takes its groups in this many parts
  int kj;               // a slot holds 2 kj k-blocks
  int slot_bytes, slots;
  int lora_sub, n_sub;  // layout of a packed B_all
  int vec;              // y takes four outputs per store
  int32_t* status;
};

__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}
__device__ __forceinline__ void mma16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
template <int ID, int N>
__device__ __forceinline__ void named_sync() {
  __syncwarp();
  asm volatile("bar.sync %0, %1;" ::"n"(ID), "n"(N) : "memory");
}
// One k16 step of a product warp: all tokens x 2 NP row groups.  NP is a template argument because a dozen tests of a group's
// index cost more than the products of a narrow CTA (4 groups of 11008 columns: 47 us with them, 18 without any products).
template <int XR, int NP>
struct RwStep {
  static constexpr int MT = RwCfg<XR>::MT;
  static constexpr int NB = NP < 4 ? NP : 4;  // weight fragments held at a time
  uint32_t xa[MT][4], b[NB][4];
  __device__ __forceinline__ void load(uint32_t xb, uint32_t wb) {
#pragma unroll
    for (int m = 0; m < MT; ++m) ldsm4(xa[m], xb + m * 16 * 128);
#pragma unroll
    for (int i = 0; i < NB; ++i) ldsm4(b[i], wb + i * 2048);
  }
  __device__ __forceinline__ void multiply(float (&acc)[2 * NP][MT][4], uint32_t wb) {
#pragma unroll
    for (int i = 0; i < NP; ++i) {
#pragma unroll
      for (int m = 0; m < MT; ++m) {
        mma16816(acc[2 * i][m], xa[m], b[i % NB][0], b[i % NB][1]);
        mma16816(acc[2 * i + 1][m], xa[m], b[i % NB][2], b[i % NB][3]);
      }
      if (i + NB < NP) ldsm4(b[i % NB], wb + (i + NB) * 2048);
    }
  }
};

template <int XR, int NP, bool LORA>
__global__ void __launch_bounds__(rw_threads(LORA), 1) linear_rows_kernel(const __grid_constant__ CUtensorMap map_x, RwParams p) {
  using C = RwCfg<XR>;
  constexpr int MT = C::MT, G = 2 * NP;  // row groups multiplied per pass
  extern __shared__ uint8_t smem_raw[];
  uint8_t* ring = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  float* s_red = reinterpret_cast<float*>(ring + C::ring(LORA));  // [8][4][XR][8]
  uint8_t* aux = reinterpret_cast<uint8_t*>(s_red) + C::kRed;
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(aux);          // [16]
  uint64_t* empty_bar = full_bar + kRwMaxSlots;                   // [16]
  int* s_tok = reinterpret_cast<int*>(aux + 2 * kRwMaxSlots * 8);  // [32] adapter slot of every token
  int* s_list = s_tok + 32;                                       // [32] distinct ones
  uint64_t* list_bar = reinterpret_cast<uint64_t*>(s_list + 32);  // LORA: the adapters are listed
  uint64_t* u_bar = list_bar + 1;                                 //       u is written
  bf16* s_u = reinterpret_cast<bf16*>(aux + C::kAux);             // LORA: [XR][r_tot + 8] scale * u
  __shared__ int s_abort, s_nseg;

  const LinearArgs& a = p.a;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int u0 = (int)((long long)p.units * blockIdx.x / gridDim.x), u1 = (int)((long long)p.units * (blockIdx.x + 1) / gridDim.x);
  const int passes = p.passes;
  auto pass_first = [&](int i) { return (u0 + (u1 - u0) * i / passes) * p.unit; };  // first row group of a pass
  const int kps = 2 * p.kj, n_st = (p.k_blocks + kps - 1) / kps;
  const int ad_rows = 8 * a.r_max * 2;  // LORA: bytes of B of one adapter and row group

  if (tid == 0) {
    s_abort = 0;
    for (int s = 0; s < p.slots; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], kRwProducts);
    }
    mbar_init(list_bar, 1);
    mbar_init(u_bar, kRwExpand);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    tma_prefetch_desc(&map_x);
  }
  __syncthreads();
  pdl_launch_dependents();

  if (warp >= kRwProducts && warp < kRwProducts + kRwCopies) {
    // ---- copies: two warps, every other slot each; a copy per lane ---------------------------------------------
    // A pass's row groups (1 KB each per k-block) are contiguous inside a tile of 128 rows: at most three pieces.  Lanes 3 h .. 3 h + 2
    // take the pieces of a slot's k-block h, lane h its token rows; what does not change with the slot is worked out once per pass.
    const uint64_t pol = l2_policy_evict_first();
    const int wh = lane / 3, piece = lane - wh * 3;
    const uint8_t* src = nullptr;
    uint32_t bytes = 0, dst = 0;
    int g0 = 0, ng = 0, cur = -1;
    auto part = [&](int i, int& n) {  // first row group and length of a piece
      int g = g0;
      n = 0;
      for (int k = 0; k <= i; ++k) {
        g += n;
        n = min(g0 + ng - g, 16 - (g & 15));
      }
      return g;
    };
    auto begin_pass = [&](int pass) {
      g0 = pass_first(pass);
      ng = pass_first(pass + 1) - g0;
      int n;
      const int g = part(piece, n);
      bytes = wh < kps ? n * 1024 : 0;
      dst = (wh * ng + g - g0) * 1024;
      src = reinterpret_cast<const uint8_t*>(a.W) + ((size_t)(g >> 4) * p.k_blocks + wh) * (BM * BK * 2) + (g & 15) * 1024;
      cur = pass;
    };
    auto weights = [&](int pass, int st, int slot) {
      if (pass != cur) begin_pass(pass);
      if (lane == 0) mbar_expect_tx(&full_bar[slot], min(kps, p.k_blocks - kps * st) * (ng * 1024 + C::kXBytes));
      __syncwarp();
      if (bytes && kps * st + wh < p.k_blocks)
        bulk_load_hint(ring + slot * p.slot_bytes + dst, src + (size_t)st * kps * (BM * BK * 2), bytes, &full_bar[slot], pol);
    };
    auto rows = [&](int pass, int st, int slot) {
      if (pass != cur) begin_pass(pass);
      if (lane < kps && kps * st + lane < p.k_blocks)
        tma_load_2d(ring + slot * p.slot_bytes + kps * ng * 1024 + lane * C::kXBytes, &map_x, (kps * st + lane) * BK, 0, &full_bar[slot]);
    };
    // adapters [j0, j1) of the list: their rows of B, [adapter][slice of the rank][row group]
    auto adapters = [&](int pass, int j0, int j1, int slot) {
      if (pass != cur) begin_pass(pass);
      const int rb = p.lora_sub * 2;
      if (lane == 0) mbar_expect_tx(&full_bar[slot], (j1 - j0) * ng * ad_rows);
      __syncwarp();
      for (int i = lane; i < (j1 - j0) * p.n_sub * 3; i += 32) {
        const int l = i / 3, j = l / p.n_sub, sb = l - j * p.n_sub;
        int n;
        const int g = part(i - l * 3, n);
        if (n > 0)
          bulk_load(ring + slot * p.slot_bytes + j * ng * ad_rows + (sb * ng + g - g0) * 8 * rb,
                    reinterpret_cast<const uint8_t*>(a.B_all) + (((size_t)s_list[j0 + j] * p.row_tiles + (g >> 4)) * p.n_sub + sb) * (BM * rb) + (g & 15) * 8 * rb,
                    n * 8 * rb, &full_bar[slot]);
      }
    };
    const int first = warp - kRwProducts, ahead = min(p.slots, n_st);
    for (int i = first; i < ahead; i += kRwCopies) weights(0, i, i);
    pdl_wait();
    for (int i = first; i < ahead; i += kRwCopies) rows(0, i, i);
    int slot = first, pass = 0, st = first, n_seg = LORA ? -1 : 0, per_slot = 1, n_all = n_st;  // n_all: slots of a pass
    uint32_t round = 0;
    for (int i = first;; i += kRwCopies) {
      if (i >= ahead) {
        if (LORA && n_seg < 0 && st >= n_st) {  // from here on the number of adapters counts
          int ok = 1;
          if (lane == 0) ok = mbar_wait(list_bar, 0, &s_abort) ? 1 : 0;
          if (!__shfl_sync(0xffffffffu, ok, 0)) {
            if (lane == 0) {
              s_abort = 1;
              atomicOr(p.status, 4);
            }
            break;
          }
          __syncwarp();  // (the list as lane 0 has waited for it; a shuffle orders no memory)
          n_seg = s_nseg;
        }
        if (LORA && n_seg >= 0) {
          if (pass != cur) begin_pass(pass);
          per_slot = max(1, p.slot_bytes / (ng * ad_rows));
          n_all = n_st + (n_seg + per_slot - 1) / per_slot;
        }
        while ((!LORA || n_seg >= 0) && pass < passes && st >= n_all) {
          st -= n_all;
          if (++pass < passes) {
            begin_pass(pass);
            if (LORA) {
              per_slot = max(1, p.slot_bytes / (ng * ad_rows));
              n_all = n_st + (n_seg + per_slot - 1) / per_slot;
            }
          }
        }
        if (pass >= passes) break;
        int ok = 1;
        if (lane == 0 && round > 0) ok = mbar_wait(&empty_bar[slot], (round - 1) & 1, &s_abort) ? 1 : 0;
        if (!__shfl_sync(0xffffffffu, ok, 0)) {
          if (lane == 0) {
            s_abort = 1;
            atomicOr(p.status, 1);
          }
          break;
        }
        if (st < n_st) {
          weights(pass, st, slot);
          rows(pass, st, slot);
        } else {
          adapters(pass, (st - n_st) * per_slot, min(n_seg, (st - n_st + 1) * per_slot), slot);
        }
      }
      st += kRwCopies;
      if ((slot += kRwCopies) >= p.slots) {
        slot -= p.slots;
        ++round;
      }
    }
  } else if (warp < kRwProducts) {
    // ---- products and output --------------------------------------------------------------------------
    const int half = warp >> 2, ks = warp & 3;  // this warp's 16 columns of a slot
    const int g = lane >> 2, c = lane & 3;
    // ldmatrix row addresses inside a 64-column tile with 128-byte swizzle: 16-byte chunk ^ (row mod 8)
    const int lr = lane & 7, lm = lane >> 3;
    const uint32_t x_off = (lr + (lm & 1) * 8) * 128 + (((2 * ks + (lm >> 1)) ^ lr) << 4);
    const uint32_t w_off = (lm >> 1) * 1024 + lr * 128 + (((2 * ks + (lm & 1)) ^ lr) << 4);
    const uint32_t ring0 = smem_u32(ring), full0 = smem_u32(full_bar);
    const bool silu = (a.flags & MLORA_SILU_MUL) != 0, out_f32 = (a.flags & MLORA_OUT_F32) != 0;
    const int out_cols = silu ? a.out / 2 : a.out;
    auto store = [&](int t, int col, const float (&o)[4]) {
      const size_t at = (size_t)t * a.ldy + col;
      if (p.vec && col + 4 <= out_cols) {
        if (out_f32) {
          *reinterpret_cast<float4*>(reinterpret_cast<float*>(a.y) + at) = make_float4(o[0], o[1], o[2], o[3]);
        } else {
          uint2 v;
          *reinterpret_cast<__nv_bfloat162*>(&v.x) = __floats2bfloat162_rn(o[0], o[1]);
          *reinterpret_cast<__nv_bfloat162*>(&v.y) = __floats2bfloat162_rn(o[2], o[3]);
          *reinterpret_cast<uint2*>(reinterpret_cast<bf16*>(a.y) + at) = v;
        }
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (col + e < out_cols) store_out(a, t, col + e, o[e]);
      }
    };
    int slot = 0;
    uint32_t par = 0;
    pdl_wait();
    for (int pass = 0; pass < passes; ++pass) {
      const int g0 = pass_first(pass), ng = pass_first(pass + 1) - g0;
      auto leave = [&]() {  // done with the slot: what was read has arrived in registers when the warp meets
        __syncwarp();
        if (lane == 0) mbar_arrive(&empty_bar[slot]);
        if (++slot == p.slots) {
          slot = 0;
          par ^= 1;
        }
      };
      // (groups past the pass's last are multiplied too: kilobytes further on in shared memory, sums that nobody looks at)
      // Narrow CTAs sum every other step in a second set, which halves the chains: a mma rounds its sum towards zero, and K / 128
      // of them in a row were further off than stream-K's (8192 -> 2048: 9.9e-7 of the result against 8.4e-7).
      constexpr int SETS = G * MT <= 8 ? 2 : 1;
      float sums[SETS][G][MT][4];
      float (&acc)[G][MT][4] = sums[0];
#pragma unroll
      for (int s = 0; s < SETS; ++s)
#pragma unroll
        for (int i = 0; i < G; ++i)
#pragma unroll
          for (int m = 0; m < MT; ++m)
#pragma unroll
            for (int e = 0; e < 4; ++e) sums[s][i][m][e] = 0.f;
      const uint32_t xo = kps * ng * 1024 + half * C::kXBytes + x_off, wo = half * ng * 1024 + w_off;
      // Narrow CTAs have two steps in registers, so that the next one's operands are on their way while one is multiplied.
      constexpr int DEPTH = NP <= 4 ? 2 : 1;
      RwStep<XR, NP> step[DEPTH];
      int st = 0, left = 0;  // slots entered, steps of the present one that are not loaded yet
      uint32_t xb = 0, wb = 0;
      auto load = [&](RwStep<XR, NP>& t) {  // the next step's operands; false: none left
        while (left == 0) {
          if (st == n_st) return false;
          if (!mbar_wait_a(full0 + 8 * slot, par, &s_abort) && !s_abort) {
            s_abort = 1;
            atomicOr(p.status, 2);
          }
          const uint32_t base = ring0 + slot * p.slot_bytes;
          xb = base + xo;
          wb = base + wo;
          left = max(0, min(p.kj, (p.k_blocks - kps * st - half + 1) >> 1));  // this warp's k-blocks that exist
          ++st;
          if (left == 0) leave();
        }
        t.load(xb, wb);
        return true;
      };
      auto next = [&]() {  // past a step whose operands are all in registers
        xb += 2 * C::kXBytes;
        wb += 2 * ng * 1024;
        if (--left == 0) leave();
      };
      if constexpr (DEPTH == 1) {
        while (load(step[0])) {
          step[0].multiply(acc, wb);
          next();
        }
      } else {
        bool more = load(step[0]);
        while (more) {
          next();
          more = load(step[1]);
          step[0].multiply(acc, 0);
          if (!more) break;
          next();
          more = load(step[0]);
          step[1].multiply(sums[SETS - 1], 0);
        }
      }
      if constexpr (SETS > 1) {
#pragma unroll
        for (int i = 0; i < G; ++i)
#pragma unroll
          for (int m = 0; m < MT; ++m)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[i][m][e] += sums[1][i][m][e];
      }
      if constexpr (LORA) {
        if (!mbar_wait(u_bar, 0, &s_abort) && !s_abort) {
          s_abort = 1;
          atomicOr(p.status, 4);
        }
        const int n_seg = s_abort ? 0 : s_nseg, n_ks = a.r_max >> 4, per_sub = p.lora_sub >> 4, rb = p.lora_sub * 2;
        const int per_slot = max(1, p.slot_bytes / (ng * ad_rows)), pitch = a.r_max * a.n_mod + 8;
        const int sw = rb == 128 ? lr : rb == 64 ? (lr >> 1) & 3 : (lr >> 2) & 1;
        // the pass's groups lie in at most three modules (whole tiles of 16 groups): the first one's, and from next1 / next2 on
        const int mod0 = module_of(a, g0 * 8);
        const int next1 = mod0 + 1 < a.n_mod ? a.mod_off[mod0 + 1] / 8 - g0 : G, next2 = mod0 + 2 < a.n_mod ? a.mod_off[mod0 + 2] / 8 - g0 : G;
        for (int j0 = 0; j0 < n_seg; j0 += per_slot) {
          if (!mbar_wait_a(full0 + 8 * slot, par, &s_abort) && !s_abort) {
            s_abort = 1;
            atomicOr(p.status, 2);
          }
          const uint32_t base = ring0 + slot * p.slot_bytes;
          const int items = min(per_slot, n_seg - j0) * n_ks;
          for (int it = warp; it < items; it += kRwProducts) {
            const int ad = it / n_ks, k16 = it - ad * n_ks, sb = k16 / per_sub, id = s_list[j0 + ad];
            const uint32_t wb = base + ad * ng * ad_rows + sb * ng * 8 * rb + ((lm >> 1) * 8 + lr) * rb + (((2 * (k16 - sb * per_sub) + (lm & 1)) ^ sw) << 4);
#pragma unroll
            for (int m = 0; m < MT; ++m) {
              const bool t0 = s_tok[m * 16 + g] == id, t1 = s_tok[m * 16 + g + 8] == id;
              if (!__any_sync(0xffffffffu, t0 || t1)) continue;
              uint32_t ua[4];
              int have = -1;
#pragma unroll
              for (int i = 0; i < G; i += 2) {
                if (i >= ng) break;
                uint32_t b[4];
                ldsm4(b, wb + i * 8 * rb);
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                  const int u_off = (mod0 + (i + e >= next1) + (i + e >= next2)) * a.r_max;
                  if (u_off != have) {  // (uniform) the tokens' u of this module, zero where another adapter is used
                    have = u_off;
                    const bf16* ur = s_u + (m * 16 + g) * pitch + u_off + k16 * 16 + 2 * c;
                    ua[0] = t0 ? *reinterpret_cast<const uint32_t*>(ur) : 0u;
                    ua[2] = t0 ? *reinterpret_cast<const uint32_t*>(ur + 8) : 0u;
                    ua[1] = t1 ? *reinterpret_cast<const uint32_t*>(ur + 8 * pitch) : 0u;
                    ua[3] = t1 ? *reinterpret_cast<const uint32_t*>(ur + 8 * pitch + 8) : 0u;
                  }
                  mma16816(acc[i + e][m], ua, b[2 * e], b[2 * e + 1]);
                }
              }
            }
          }
          leave();
        }
      }
#pragma unroll
      for (int q = 0; q < G; q += 4) {
        if (q < ng) {
          named_sync<1, kRwProducts * 32>();  // the four groups before have been read
#pragma unroll
          for (int i = 0; i < 4 && q + i < G; ++i) {
#pragma unroll
            for (int m = 0; m < MT; ++m) {
              float* d = s_red + ((warp * 4 + i) * XR + m * 16 + g) * 8 + 2 * c;
              *reinterpret_cast<float2*>(d) = make_float2(acc[q + i][m][0], acc[q + i][m][1]);
              *reinterpret_cast<float2*>(d + 64) = make_float2(acc[q + i][m][2], acc[q + i][m][3]);
            }
          }
          named_sync<1, kRwProducts * 32>();
          auto sum4 = [&](int i, int t, int h, float (&o)[4]) {  // four rows of one token, in warp order
            float4 s = *reinterpret_cast<const float4*>(s_red + (i * XR + t) * 8 + h * 4);
#pragma unroll
            for (int w = 1; w < kRwProducts; ++w) {
              const float4 v = *reinterpret_cast<const float4*>(s_red + ((w * 4 + i) * XR + t) * 8 + h * 4);
              s.x += v.x, s.y += v.y, s.z += v.z, s.w += v.w;
            }
            o[0] = s.x, o[1] = s.y, o[2] = s.z, o[3] = s.w;
          };
          const int h = tid & 1, t = (tid >> 1) % XR, i = (tid >> 1) / XR;
          float o[4];
          if (silu) {
            if (i < 2 && q + 2 * i < ng && t < a.T) {
              float up[4];
              sum4(2 * i, t, h, o);
              sum4(2 * i + 1, t, h, up);
#pragma unroll
              for (int e = 0; e < 4; ++e) o[e] = silu_mul(o[e], up[e]);
              store(t, (g0 + q + 2 * i) * 4 + h * 4, o);
            }
          } else if (i < 4 && q + i < ng && t < a.T) {
            sum4(i, t, h, o);
            if constexpr (!LORA) {
              const int act = a.flags & (MLORA_ACT_RELU2 | MLORA_ACT_GELU);
#pragma unroll
              for (int e = 0; e < 4; ++e) o[e] = act == MLORA_ACT_RELU2 ? act_one(o[e], MLORA_ACT_RELU2) : act == MLORA_ACT_GELU ? gelu_fast(o[e]) : o[e];
            }
            store(t, (g0 + q + i) * 8 + h * 4, o);
          }
        }
      }
    }
  } else if constexpr (LORA) {
    // ---- the adapters' side: list, scale * u ------------------------------------------------------------
    const int lw = warp - kRwProducts - kRwCopies, r_tot = a.r_max * a.n_mod, pitch = r_tot + 8;
    pdl_wait();
    if (lw == 0) {
      const int n = distinct_slots_n(a, 0, a.T, 32, s_tok, s_list);
      if (lane == 0) {
        s_nseg = n;
        mbar_arrive(list_bar);
      }
    }
    for (int i = lw * 32 + lane; i < XR * (r_tot >> 3); i += kRwExpand * 32) {
      const int t = i / (r_tot >> 3), j = (i - t * (r_tot >> 3)) * 8;
      uint4 v = make_uint4(0u, 0u, 0u, 0u);
      const int s = t < a.T ? a.slots[t] : -1;
      if (s >= 0 && s < a.n_adapters) {
        const float sc = a.scales[s];
        const float* ur = a.u + (size_t)t * r_tot + j;
        const float4 lo = *reinterpret_cast<const float4*>(ur), hi = *reinterpret_cast<const float4*>(ur + 4);
        const float f[8] = {lo.x * sc, lo.y * sc, lo.z * sc, lo.w * sc, hi.x * sc, hi.y * sc, hi.z * sc, hi.w * sc};
        v = pack8(f);
      }
      *reinterpret_cast<uint4*>(s_u + t * pitch + j) = v;
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(u_bar);
  }
  __syncwarp();
  __syncthreads();
  if (s_abort) {
    // give copies that may still be in flight a bounded time to land before the CTA exits
    for (int i = 0; i < 64; ++i) __nanosleep(1000);
  }
}

template <int XR, int NP, bool LORA>
int launch_rows(const CUtensorMap& mx, const RwParams& p, int grid, cudaStream_t st) {
  using C = RwCfg<XR>;
  static std::atomic<unsigned long long> attr_done{0};  // the shared-memory opt-in is a per-device attribute of each instantiation
  int dev = 0;
  cudaGetDevice(&dev);
  if (!((attr_done.load(std::memory_order_acquire) >> (dev & 63)) & 1ull)) {
    const cudaError_t e = cudaFuncSetAttribute(linear_rows_kernel<XR, NP, LORA>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::smem(LORA));
    if (e != cudaSuccess) return fail(MLORA_ECUDA, "linear: cudaFuncSetAttribute: %s", cudaGetErrorString(e));
    attr_done.fetch_or(1ull << (dev & 63), std::memory_order_release);
  }
  launch_pdl_if(pdl_enabled_gemm(), linear_rows_kernel<XR, NP, LORA>, grid, rw_threads(LORA), C::smem(LORA), st, mx, p);
  count_launch();
  MLORA_CHECK_LAUNCH("linear_rows_kernel");
  return MLORA_OK;
}

struct RowsPlan {
  int units, unit, grid, passes;
  int groups, pairs;  // row groups of the widest pass; half of those that are multiplied (NP)
  int kj, slot_bytes, slots;
};

// Row groups of a pass -> NP.  A pass multiplies 2 NP groups whatever it has, so the steps lie at widths that occur: over 148 SMs 4096
// outputs have 4 groups, 5120 5, 12288 11, 15360 13, 22016 behind SiLU 20 (in two passes beyond 16 rows: 10).  A width in between
// multiplies up to five groups for nothing.
template <int XR>
int np_for(int groups) {
  constexpr int steps16[] = {2, 4, 6, 7, 10}, steps32[] = {2, 4, 5, 6};
  if constexpr (XR > 16) {
    for (int np : steps32)
      if (groups <= 2 * np) return np;
  } else {
    for (int np : steps16)
      if (groups <= 2 * np) return np;
  }
  return 0;
}

template <int XR>
RowsPlan rows_plan(const LinearArgs& a, bool lora) {
  using C = RwCfg<XR>;
  RowsPlan q{};
  const int k_blocks = (a.in + BK - 1) / BK;
  q.unit = (a.flags & MLORA_SILU_MUL) ? 2 : 1;
  q.units = (a.out + 8 * q.unit - 1) / (8 * q.unit);
  q.grid = q.units < sm_count() ? q.units : sm_count();
  const int most = (q.units + q.grid - 1) / q.grid, cap = C::kMaxG / q.unit;
  q.passes = (most + cap - 1) / cap;
  q.groups = (most + q.passes - 1) / q.passes * q.unit;
  q.pairs = np_for<XR>(q.groups);
  const int kb_bytes = q.groups * 1024 + C::kXBytes, ring = C::ring(lora);
  // As many k-blocks per slot as leave four slots: a slot's hand-over costs its warps about 0.15 us whatever it holds (1 row,
  // 11008 -> 4096: 27.6 us with two k-blocks per slot, 22 with eight).
  q.kj = 4;
  while (q.kj > 1 && (ring / (2 * q.kj * kb_bytes) < 4 || q.kj >= k_blocks)) q.kj >>= 1;
  q.slot_bytes = 2 * q.kj * kb_bytes;
  q.slots = ring / q.slot_bytes;
  if (q.slots > kRwMaxSlots) q.slots = kRwMaxSlots;
  return q;
}

template <int XR, bool LORA>
int plan_rows(const LinearArgs& a, void* work, cudaStream_t st) {
  CUtensorMap mx;
  const int rc = make_map(&mx, a.x, a.T, a.in, a.ldx, XR);
  if (rc) return rc;
  const RowsPlan q = rows_plan<XR>(a, LORA);
  RwParams p;
  p.a = a;
  p.k_blocks = (a.in + BK - 1) / BK;
  p.row_tiles = (a.out + BM - 1) / BM;
  p.unit = q.unit;
  p.units = q.units;
  p.passes = q.passes;
  p.kj = q.kj;
  p.slot_bytes = q.slot_bytes;
  p.slots = q.slots;
  p.lora_sub = a.r_max > 0 && a.r_max < 64 ? a.r_max : 64;
  p.n_sub = a.r_max > 64 ? a.r_max / 64 : 1;
  const int es = (a.flags & MLORA_OUT_F32) ? 4 : 2;
  p.vec = (reinterpret_cast<uintptr_t>(a.y) % (4 * es)) == 0 && a.ldy % 4 == 0;
  p.status = (int32_t*)work;
  if (q.pairs == 2) return launch_rows<XR, 2, LORA>(mx, p, q.grid, st);
  if (q.pairs == 4) return launch_rows<XR, 4, LORA>(mx, p, q.grid, st);
  if (q.pairs == 6) return launch_rows<XR, 6, LORA>(mx, p, q.grid, st);
  if constexpr (XR > 16) {
    return launch_rows<XR, 5, LORA>(mx, p, q.grid, st);
  } else {
    if (q.pairs == 7) return launch_rows<XR, 7, LORA>(mx, p, q.grid, st);
    return launch_rows<XR, 10, LORA>(mx, p, q.grid, st);
  }
}

// Up to which `in` a call is faster here than on stream-K, by rows and by the row groups of the widest CTA.  A k-block takes 0.11 us
// however few groups a CTA has (two k16 steps of a product warp), stream-K's share of it falls with them: narrow projections of
// great length lose what the missing hand-over gained.  Five groups multiply eight.  Above 16 rows x weighs as much as the weights.
// Time here over stream-K's (CUDA events behind a norm, 148 SMs):
//   in               1 row: 4096 8192 11008     4 rows: 2048 4096 8192     16 rows: 2048 4096 8192     32 rows: 2048 4096 6144
//    2 groups (2048)        .89  1.06 1.09              .87  .97  1.21               .83  .96  1.16               .75  .84  .92
//    4 groups (4096)        .89  .94  .94               .84  .98  1.05               .82  .89  .98                .82  .94  .99
//    5 groups (5120)        .96  1.01 1.01              .99  1.06 1.10               .95  1.02 1.10               .88  .96  1.02
//    6 groups (6144)        .90  .91  .91               .87  .95  .99                .89  .95  .98                .83  .91  .95
//    7 groups (8192)        .86  .89  .89               .79  .92  .94                .85  .91  .93                .83  .87  .89
//   11 groups (12288)       .87  .90  .91               .84  .91  .92                .87  .89  .91                .91  .93  .93
// With rank-16 adapters 4 groups .92 at 4096 but 1.05 at 8192 with 1 row, .89 and .92 with 16, .93 at 4096 with 32; 6 groups 1.01 at 6144 with
// 32; wider ranks gain more.  Within a column the limits lie where the slowest width of that many groups stays at 1.01 or below.
int rows_in_limit(int T, int groups, bool lora) {
  constexpr int any = 1 << 30;
  static constexpr int plain[6][7] = {
      // 1 group   2     3     4     5     6     7 and more
      {5120, 6144, 6144, any, 6144, any, any},       // 1 row
      {4096, 4096, 4096, 6144, 4096, any, any},      // 2
      {3072, 3072, 3072, 4096, 2048, 8192, any},     // 3, 4
      {3072, 3072, 3072, 4096, 2048, 8192, 8192},    // 5 to 7
      {3072, 3072, 3072, 6144, 2048, 8192, 8192},    // 8 to 16
      {6144, 6144, 4096, 4096, 5120, 6144, 6144}};   // 17 to 32
  static constexpr int adapters[6][7] = {
      {4096, 4096, 4096, 4096, 4096, any, any},
      {4096, 4096, 4096, 8192, 4096, 8192, any},
      {4096, 4096, 4096, 8192, 4096, 8192, any},
      {4096, 4096, 4096, 8192, 4096, 8192, 8192},
      {4096, 4096, 4096, 8192, 4096, 8192, 8192},
      {3072, 3072, 3072, 4096, 4096, 4096, 6144}};
  const int t = T <= 1 ? 0 : T <= 2 ? 1 : T <= 4 ? 2 : T <= 7 ? 3 : T <= 16 ? 4 : 5, g = groups < 7 ? groups - 1 : 6;
  return lora ? adapters[t][g] : plain[t][g];
}

}  // namespace

bool linear_rows_chosen(const LinearArgs& a) {
  if ((a.flags & (MLORA_ANY_SUMS | MLORA_STABLE_SUMS | MLORA_W_PACKED)) != (MLORA_ANY_SUMS | MLORA_W_PACKED) || a.T < 1 || a.T > 32) return false;
  // Fewer row groups than SMs leave SMs idle; stream-K cuts `in` for all of them (and has the shorter sums).
  if ((a.out + 7) / 8 < sm_count()) return false;
  const int unit = (a.flags & MLORA_SILU_MUL) ? 16 : 8;
  if (a.T > 16 && (a.out + unit - 1) / unit > 2 * (RwCfg<32>::kMaxG * 8 / unit) * sm_count()) return false;  // three passes over x
  const int units = (a.out + unit - 1) / unit, grid = units < sm_count() ? units : sm_count();
  if (a.in > rows_in_limit(a.T, (units + grid - 1) / grid * (unit / 8), a.u != nullptr)) return false;
  if (a.u == nullptr) return true;
  if (!(a.flags & MLORA_B_PACKED) || !aligned16(a.u) || a.r_max * a.n_mod > RwCfg<32>::kMaxRank) return false;
  if (!(a.r_max == 16 || a.r_max == 32 || a.r_max == 64 || a.r_max == 128)) return false;
  for (int m = 1; m < a.n_mod; ++m)
    if (a.mod_off[m] % BM != 0) return false;
  return true;
}

int launch_linear_rows(const LinearArgs& a, void* work, cudaStream_t st) {
  if (a.u == nullptr) return a.T <= 16 ? plan_rows<16, false>(a, work, st) : plan_rows<32, false>(a, work, st);
  return a.T <= 16 ? plan_rows<16, true>(a, work, st) : plan_rows<32, true>(a, work, st);
}

void linear_rows_plan(const LinearArgs& a, int32_t* v6) {
  const RowsPlan q = a.T <= 16 ? rows_plan<16>(a, a.u != nullptr) : rows_plan<32>(a, a.u != nullptr);
  v6[0] = q.passes;
  v6[1] = q.grid;
  v6[2] = q.groups;
  v6[3] = 2 * q.pairs;
  v6[4] = 2 * q.kj;
  v6[5] = q.slots;
}

}  // namespace mlora
