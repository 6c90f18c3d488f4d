// Triangle attention core for sm_100a: flash-style, head_dim 32, bf16 in, fp32 softmax.
//
// For every pair row (b, r), head h and query s:
//   o[s,:] = softmax_t( scale * (q[s]·k[t] + bias[b,h,s,t]) ; t < len[b,r] ) · v[t,:]   (* gate[s,:])
// where `bias` is the triangle bias already divided by `scale` and `gate` holds sigmoid(gate logits) (the
// prologue writes both that way).
//
// The N x N x N logits never exist in memory.  A CTA owns four units of work at a time; a unit is 128 queries of one
// (b, r, h), belongs to one softmax warpgroup and walks the keys in tiles of 64:
//   TMA      K and V tiles of the item's rows, bias tiles of its 128-query blocks -> shared memory (three stages)
//   tcgen05  S = Q·Kᵀ   (128x64x32, K-major operands in smem, accumulator in TMEM)
//   softmax  one thread per query row: S from TMEM -> registers, + bias from shared memory, exp2 relative to the
//            row's first score, row sum; the bf16 probabilities go straight back to TMEM
//   tcgen05  O += P·V   (128x32x64: P is the A operand from TMEM, V the MN-major B operand from its [key][d] tile);
//            O is only rescaled when a tile's sum would leave the safe fp32 range
//
// The floor is the special-function unit: 16 exponentials a clock and SM, one per score, 512 clocks of a scheduler for
// a warp's part of a tile.  Around its exponentials a warp has some 1000 clocks of hand-overs (barrier, TMEM load, P
// store, barrier), so the unit only stays busy when other warps of the scheduler have exponentials to do meanwhile:
// four independent units per CTA, i.e. four softmax warps on every scheduler.  Their S, P and O columns have to fit
// the 512 of TMEM, which is why a key tile has 64 keys, and they would be one S, P and O each (128 columns a unit); but
// scores only pass through S, while a warpgroup's four warps sit on four schedulers and finish a tile up to 1000
// clocks apart, and the early ones may not overwrite P before the last one's P·V.  So two units share an S buffer and
// every unit has two P buffers.
// The four units of an item are two pair rows x two 128-query blocks (or four rows x one block) of the same head:
// the bias does not depend on the pair row, so one bias tile in shared memory serves two (four) units, and a K/V
// tile two.  The bias is added by the softmax threads: on the tensor core (an identity MMA) it would need 64 more
// columns and four times the operations of Q·Kᵀ, which cost clock rate under the power cap.
//
// Measured against two halves of 256 queries x 128 keys per CTA and the bias on the tensor core (one launch, all tokens
// valid, back to back, with the median SM clock sampled meanwhile; the clock is below 1965 MHz under the power cap):
//   512 tokens            426 -> 383 thousand clocks    250 us at 1702 MHz -> 204 at 1875
//   768 tokens            1.293 -> 1.220 million        775 us at 1668     -> 643 at 1897
//   1024 tokens           2.937 -> 2.763 million        1.757 ms at 1672   -> 1.453 at 1901
//   2048 tokens           21.48 -> 20.96 million        13.08 ms at 1642   -> 10.90 at 1924
//   512 rows, 4096 keys   20.36 -> 20.65 million        12.45 ms at 1635   -> 10.67 at 1935
// So short rows need fewer clocks, because the units' hand-overs fill one another and the items are smaller; long rows need
// as many as before, and what they gain is clock rate, presumably because the bias does not go through the tensor cores.
// A launch takes about (items per SM, rounded up) x (2790 x tiles + 5000) clocks, at 2048 tokens 11.1 of 16 exponentials a
// clock and SM.  The masked form takes 105 us at 333 tokens, the unmasked one 84.
//
// A pair row without a valid key takes a constant path in "uniform" mode (probabilities all 1: the output is the
// mean of V, as the eager reference computes it) and is skipped in "zeros" mode.
//
// Warp roles (640 threads): warps 0-15 softmax (warpgroup w = unit w), warp 16 TMA producer, warp 17 score MMAs / TMEM
// owner, warps 18 and 19 P·V MMAs of units 0-1 and 2-3.  The fifth warpgroup gives most of its registers to the softmax
// warpgroups (setmaxnreg).
#include "attention_items.h"
#include "common.cuh"
#include "layout.h"

namespace b200ta {
namespace {

constexpr int kThreads = 640;
constexpr int kKTile = 64;  // keys per tile
constexpr int kStages = 3;
constexpr float kRebaseSum = 1.2676506e30f;  // 2^100: a tile sum at or above this moves the reference point

struct AttnParams {
  int B, R, S, S_pad;
  ItemPlan plan;
  const int32_t* lengths;
  long long ls_b, ls_r;
  const uint32_t* key_mask;  // masked form: bit k of word [b][r][k / 32] = key k takes part (0 at and past the length)
  long long km_b, km_r;      // strides of key_mask in words
  const __nv_bfloat16* gate;
  long long g_br, g_h, g_s;
  __nv_bfloat16* out;
  long long o_br, o_s, o_h;
  float* lse;
  float scale_log2;  // softmax_scale * log2(e)
  int empty_uniform;
  int wide_store;  // out is 32-byte aligned and its strides are multiples of 16 elements
  int* status;
};

// 32-byte store; the address must be 32-byte aligned.
__device__ __forceinline__ void stg256(void* p, const uint32_t* v) {
  asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]),
               "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
               : "memory");
}

// shared-memory map (bytes, relative to the 1024-aligned base)
constexpr int kSmQ = 0;                             // 2 item buffers x 4 units x 8 KiB
constexpr int kSmStage = kSmQ + 2 * kUnits * 8192;  // kStages x 48 KiB, laid out by the three functions below
constexpr int kStageBytes = 49152;
constexpr int kSmMask = kSmStage + kStages * kStageBytes;  // masked form: 16 warps x 64 floats, 0 or -inf per key
constexpr int kSmInfo = kSmMask + 16 * 256;  // ItemInfo of the two item buffers
constexpr int kSmBars = kSmInfo + 2 * 80;
constexpr int kSmTotal = kSmBars + 320;
constexpr int kSmDynamic = kSmTotal + 1024;

// A stage holds the bias tile of block 0 (16 KiB), then either the bias tile of block 1 or the K and V tiles of rows
// 2 and 3 (4 KiB each), then the K and V tiles of rows 0 and 1.
__device__ __forceinline__ uint32_t stage_bias(int block) { return block * 16384; }
__device__ __forceinline__ uint32_t stage_k(int row) { return (row < 2 ? 32768 : 16384) + (row & 1) * 4096; }
__device__ __forceinline__ uint32_t stage_v(int row) { return stage_k(row) + 8192; }

enum Bar {
  Q_FULL = 0,     // [2] item buffer
  Q_EMPTY = 2,    // [2]
  KV_FULL = 4,    // [kStages] K, V and bias of a tile
  KV_EMPTY = 7,   // [kStages]
  S_FULL = 10,    // [4] per unit
  S_FREE = 14,    // [2] per S buffer
  P_FULL = 16,    // [4][2] per unit and P buffer
  O_FULL = 24,    // [4][2]
  NUM_BARS = 32
};

// TMEM columns: two S buffers (units w and w + 2 take turns on buffer w % 2: scores only wait there until the
// warpgroup reads them), two P buffers (bf16 pairs) per unit, O of each unit.
constexpr uint32_t kTmemS = 0, kTmemP = 128, kTmemO = 384, kTmemCols = 512;
__device__ __forceinline__ uint32_t p_column(int unit, int buffer) { return kTmemP + unit * 64 + buffer * 32; }

// What the other warps need to know about an item, written by the TMA warp into the item's slot (released by Q_FULL).
struct __align__(16) UnitInfo {
  int br;     // b * R + r of the unit's pair row; of the item's last row where the item has no such unit
  int q0;     // first query; S, past the last one, where the item has no such unit
  int len;    // keys that take part (S for a uniform row)
  int tiles;  // key tiles; 0: no valid key and "zeros" semantics; -1: the item has no such unit
};
struct __align__(16) ItemInfo {
  UnitInfo unit[kUnits];
  int tiles;       // of the item: the longest row's
  int two_blocks;  // unit w = row w / 2, block w % 2; otherwise unit w = row w, block 0
  int h;
  uint32_t uniform;  // bit per unit: no valid key and "uniform" semantics, every logit equal
};
static_assert(sizeof(ItemInfo) == 80, "layout of kSmInfo");

// Row length as stored of the pair row of unit `lane` (clamped to the item's rows).
__device__ __forceinline__ int raw_length(const AttnParams& p, const Item& it, int lane) {
  if (p.lengths == nullptr) return p.S;
  return p.lengths[it.b * p.ls_b + (it.r0 + existing_row(it, lane & 3)) * p.ls_r];
}

template <bool kMasked>
__global__ void __launch_bounds__(kThreads, 1)
attention_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                 const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_bias,
                 const AttnParams p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* gen = smem_raw + (base - smem_u32(smem_raw));
  const uint32_t bars = base + kSmBars;
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(gen + kSmBars + NUM_BARS * 8);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(gen + kSmBars + NUM_BARS * 8 + 8);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    abort_flag[0] = 0;
    abort_flag[1] = 0;
    for (int i = 0; i < 2; ++i) {
      mbar_init(bars + (Q_FULL + i) * 8, 1);
      mbar_init(bars + (Q_EMPTY + i) * 8, 2 + 1 + 16);  // P·V warps, score warp, softmax warps (read the item's info)
    }
    for (int i = 0; i < kStages; ++i) {
      mbar_init(bars + (KV_FULL + i) * 8, 1);
      mbar_init(bars + (KV_EMPTY + i) * 8, 2);  // one arrival per P·V warp
    }
    for (int i = 0; i < kUnits; ++i) mbar_init(bars + (S_FULL + i) * 8, 1);
    for (int i = 0; i < 2; ++i) mbar_init(bars + (S_FREE + i) * 8, 4);
    for (int i = 0; i < 2 * kUnits; ++i) {
      mbar_init(bars + (P_FULL + i) * 8, 4);
      mbar_init(bars + (O_FULL + i) * 8, 1);
    }
    fence_mbar_init();
  }
  if (warp == 17) {
    tmem_alloc(smem_u32(const_cast<uint32_t*>(tmem_slot)), kTmemCols);
    pdl_trigger();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  const int my_items = (p.plan.num_items - 1 - int(blockIdx.x)) / int(gridDim.x) + 1;

  // Register budget: 640 threads start with 96 registers; setmaxnreg only moves registers inside that allocation,
  // and an increase blocks until a decrease has freed enough: the fifth warpgroup drops to 64 (frees 128 x 32) and
  // the softmax warpgroups rise to 104 (need 512 x 8, the same number).
  if (warp >= 16) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 64;");
  }
  if (warp == 16) {
    // ------------------------------------------------------------------ TMA producer (whole warp, one lane issues)
    if (lane == 0) {
      tma_prefetch_desc(&tm_q);
      tma_prefetch_desc(&tm_k);
      tma_prefetch_desc(&tm_v);
      tma_prefetch_desc(&tm_bias);
    }
    int g = 0, i = 0;  // tiles and items loaded
    bool ok = true;
    Item it = decode_item(p.plan, blockIdx.x);
    pdl_wait();  // (the MMA warps touch no global memory)
    int raw = raw_length(p, it, lane);
    while (i < my_items) {
      // lane u: unit u
      const int blocks = it.two_blocks ? 2 : 1;
      const int row = unit_row(it, lane & 3);
      int len = raw < 0 ? 0 : (raw > p.S ? p.S : raw);
      const bool exists = row < it.rows;
      const bool uni = exists && len == 0 && p.empty_uniform;
      if (uni) len = p.S;
      const int nt = exists ? (len + kKTile - 1) / kKTile : -1;
      const int tiles = max(0, __reduce_max_sync(0xffffffffu, nt));
      const uint32_t uniform = __ballot_sync(0xffffffffu, uni) & 15u;
      const int ib = i & 1;
      ok = mbar_wait_warp(bars + (Q_EMPTY + ib) * 8, ((i >> 1) & 1) ^ 1, abort_flag);
      if (!ok) break;
      ItemInfo* info = reinterpret_cast<ItemInfo*>(gen + kSmInfo) + ib;
      const int br = it.b * p.R + it.r0;
      if (lane < kUnits) {
        *reinterpret_cast<int4*>(&info->unit[lane]) =
            make_int4(br + existing_row(it, lane), exists ? it.q0 + (it.two_blocks ? lane & 1 : 0) * kQTile : p.S, len, nt);
      } else if (lane == kUnits) {
        *reinterpret_cast<int4*>(&info->tiles) = make_int4(tiles, it.two_blocks, it.h, int(uniform));
      }
      __syncwarp();
      if (lane == 0) {
        mbar_expect_tx(bars + (Q_FULL + ib) * 8, tiles > 0 ? it.rows * blocks * 8192 : 0);
        if (tiles > 0)
          for (int r = 0; r < it.rows; ++r)
            for (int w = 0; w < blocks; ++w)
              tma_load_4d(base + kSmQ + (ib * kUnits + r * blocks + w) * 8192, &tm_q, bars + (Q_FULL + ib) * 8, 0,
                          it.q0 + w * kQTile, it.h, br + r);
      }
      __syncwarp();
      ++i;
      const Item cur = it;
      if (i < my_items) {  // the next item's row lengths arrive while this item's tiles are loaded
        it = decode_item(p.plan, blockIdx.x + i * gridDim.x);
        raw = raw_length(p, it, lane);
      }
      for (int kt = 0; kt < tiles; ++kt, ++g) {
        const int stage = g % kStages;
        ok = mbar_wait_warp(bars + (KV_EMPTY + stage) * 8, ((g / kStages) & 1) ^ 1, abort_flag);
        if (!ok) break;
        // rows with this tile (a bit per row), and those of them that need the bias
        const bool first = !cur.two_blocks || (lane & 1) == 0;
        const uint32_t units = __ballot_sync(0xffffffffu, lane < kUnits && kt < nt);
        const uint32_t loads = __ballot_sync(0xffffffffu, lane < kUnits && first && kt < nt);
        if (lane == 0) {
          const uint32_t full = bars + (KV_FULL + stage) * 8;
          const uint32_t sbase = base + kSmStage + stage * kStageBytes;
          const bool with_bias = (units & ~uniform) != 0;
          mbar_expect_tx(full, __popc(loads) * 8192 + (with_bias ? blocks * 16384 : 0));
          if (with_bias)
            for (int w = 0; w < blocks; ++w)
              tma_load_4d(sbase + stage_bias(w), &tm_bias, full, kt * kKTile, cur.q0 + w * kQTile, cur.h, cur.b);
          for (uint32_t left = loads; left; left &= left - 1) {
            const int u = __ffs(left) - 1, r = cur.two_blocks ? u >> 1 : u;
            tma_load_4d(sbase + stage_k(r), &tm_k, full, 0, kt * kKTile, cur.h, br + r);
            tma_load_4d(sbase + stage_v(r), &tm_v, full, 0, kt * kKTile, cur.h, br + r);
          }
        }
        __syncwarp();
      }
      if (!ok) break;
    }
    // If the loop was abandoned, give copies still in flight a bounded chance to land.
    if (*abort_flag && lane == 0) {
      for (int j = g > kStages ? g - kStages : 0; j < g; ++j)
        mbar_wait(bars + (KV_FULL + j % kStages) * 8, (j / kStages) & 1, abort_flag + 1);
      for (int j = i > 2 ? i - 2 : 0; j < i; ++j) mbar_wait(bars + (Q_FULL + (j & 1)) * 8, (j >> 1) & 1, abort_flag + 1);
    }
    __syncwarp();
  } else if (warp == 17) {
    // ------------------------------------------------------------------ score MMAs (S = Q·Kᵀ) of the four units
    // All 32 lanes run the loop with the same values and one elected lane issues (umma_*_warp).  The warp runs a
    // tile ahead of the softmax, also across items: all it waits for besides the loads is that a unit's S columns
    // have been read.
    constexpr uint32_t idesc_s = make_idesc_bf16(kQTile, kKTile);  // both operands K-major
    const uint32_t tb = __shfl_sync(0xffffffffu, tmem_base, 0);
    int stage = 0, stage_phase = 0;
    uint32_t ns = 0;  // bit b: parity of the tiles issued into S buffer b
    bool ok = true;
    for (int i = 0; ok && i < my_items; ++i) {
      const int ib = i & 1;
      ok = mbar_wait_warp(bars + (Q_FULL + ib) * 8, (i >> 1) & 1, abort_flag);
      if (!ok) break;
      const ItemInfo* info = reinterpret_cast<const ItemInfo*>(gen + kSmInfo) + ib;
      const int tiles = info->tiles, two_blocks = info->two_blocks;
      const uint32_t uniform = info->uniform;
      int nt[kUnits];
#pragma unroll
      for (int u = 0; u < kUnits; ++u) nt[u] = info->unit[u].tiles;
      mbar_arrive_warp_after_reads(bars + (Q_EMPTY + ib) * 8);  // the info has been read (Q itself: see the P·V warps)
      const uint32_t q0 = base + kSmQ + ib * (kUnits * 8192);
      for (int kt = 0; ok && kt < tiles; ++kt) {
        ok = mbar_wait_warp(bars + (KV_FULL + stage) * 8, stage_phase, abort_flag);
        const uint32_t sbase = base + kSmStage + stage * kStageBytes;
#pragma unroll
        for (int u = 0; u < kUnits; ++u) {
          if (!ok || kt >= nt[u]) continue;
          const int sb = u & 1;
          ok = mbar_wait_warp(bars + (S_FREE + sb) * 8, ((ns >> sb) & 1u) ^ 1u, abort_flag);
          if (!ok) continue;
          ns ^= 1u << sb;
          tc_fence_after();
          if (!((uniform >> u) & 1u)) {  // a uniform row has equal logits: the softmax warps need no scores
            const uint64_t dq = smem_desc<16, 512, kLayoutSw64>(q0 + u * 8192);
            const uint64_t dk = smem_desc<16, 512, kLayoutSw64>(sbase + stage_k(two_blocks ? u >> 1 : u));
            umma_ss_warp(tb + kTmemS + sb * 64, dq, dk, idesc_s, 0u);
            umma_ss_warp(tb + kTmemS + sb * 64, dq + 2, dk + 2, idesc_s, 1u);  // second 16 channels: +32 bytes
          }
          umma_commit_warp(bars + (S_FULL + u) * 8);
        }
        if (++stage == kStages) stage = 0, stage_phase ^= 1;
      }
    }
  } else if (warp == 18 || warp == 19) {
    // ------------------------------------------------------------------ P·V MMAs of units 2j and 2j + 1
    constexpr uint32_t idesc_o = make_idesc_bf16(kQTile, kHeadDim, false, true);  // B is MN-major
    const int j = __shfl_sync(0xffffffffu, warp - 18, 0);
    const uint32_t tb = __shfl_sync(0xffffffffu, tmem_base, 0);
    int stage = 0, stage_phase = 0;
    uint32_t np[2] = {0, 0};  // P tiles consumed of the two units
    bool ok = true;
    for (int i = 0; ok && i < my_items; ++i) {
      const int ib = i & 1;
      ok = mbar_wait_warp(bars + (Q_FULL + ib) * 8, (i >> 1) & 1, abort_flag);
      if (!ok) break;
      const ItemInfo* info = reinterpret_cast<const ItemInfo*>(gen + kSmInfo) + ib;
      const int tiles = info->tiles, two_blocks = info->two_blocks;
      const int row_tiles[2] = {info->unit[2 * j].tiles, info->unit[2 * j + 1].tiles};
      const int row[2] = {two_blocks ? j : 2 * j, two_blocks ? j : 2 * j + 1};
      for (int kt = 0; ok && kt < tiles; ++kt) {
        ok = mbar_wait_warp(bars + (KV_FULL + stage) * 8, stage_phase, abort_flag);
        const uint32_t sbase = base + kSmStage + stage * kStageBytes;
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          if (!ok || kt >= row_tiles[u]) continue;
          const int w = 2 * j + u, pb = np[u] & 1;
          ok = mbar_wait_warp(bars + (P_FULL + 2 * w + pb) * 8, (np[u] >> 1) & 1u, abort_flag);
          if (!ok) continue;
          ++np[u];
          tc_fence_after();
          const uint32_t d = tb + kTmemO + w * 32, tp = tb + p_column(w, pb);
          const uint64_t dv = smem_desc<16, 512, kLayoutSw64>(sbase + stage_v(row[u]));
          umma_ts_warp(d, tp, dv, idesc_o, kt > 0 ? 1u : 0u);
#pragma unroll
          for (int k = 1; k < 4; ++k) umma_ts_warp(d, tp + k * 8, dv + k * 64, idesc_o, 1u);  // 16 keys = 1 KiB per step
          umma_commit_warp(bars + (O_FULL + 2 * w + pb) * 8);
        }
        if (!ok) break;
        // The probabilities these MMAs waited for say that the scores' MMAs have read K (and Q), and the
        // warpgroups the bias: the stage, and after the last tile the Q buffer, are free once the MMAs ran.
        umma_commit_warp(bars + (KV_EMPTY + stage) * 8);
        if (kt == tiles - 1) umma_commit_warp(bars + (Q_EMPTY + ib) * 8);
        if (++stage == kStages) stage = 0, stage_phase ^= 1;
      }
      if (tiles == 0) mbar_arrive_warp(bars + (Q_EMPTY + ib) * 8);
    }
  } else if (warp < 16) {
    // ------------------------------------------------------------------ softmax warpgroups
    asm volatile("setmaxnreg.inc.sync.aligned.u32 104;");
    pdl_wait();
    // keep_in_register: the compiler otherwise derives these from the thread index again in every tile, waiting for the
    // special register each time (2048 tokens 10.95 -> 10.66 ms)
    const int w = keep_in_register(warp >> 2);               // unit
    const int m = keep_in_register((warp & 3) * 32 + lane);  // query row inside the unit == TMEM lane
    const uint32_t lane_taddr = keep_in_register(tmem_base + (uint32_t((warp & 3) * 32) << 16));
    const uint32_t s_addr = lane_taddr + kTmemS + (w & 1) * 64;
    const uint32_t o_addr = lane_taddr + kTmemO + w * 32;
    const float c = p.scale_log2;  // raw score -> log2-domain logit
    const uint64_t c2 = pack_f32x2(c, c);
    int ct = 0;  // tiles this unit has processed (phase of S_FULL / O_FULL)
    int stage = 0, stage_phase = 0;  // ring position
    bool ok = true;
    for (int i = 0; ok && i < my_items; ++i) {
      const int ib = i & 1;
      ok = mbar_wait_warp(bars + (Q_FULL + ib) * 8, (i >> 1) & 1, abort_flag);
      if (!ok) break;
      const ItemInfo* info = reinterpret_cast<const ItemInfo*>(gen + kSmInfo) + ib;
      const int4 unit = *reinterpret_cast<const int4*>(&info->unit[w]);
      const int4 common = *reinterpret_cast<const int4*>(&info->tiles);
      const int my_tiles = unit.w, len = unit.z;
      const bool uniform = (common.w >> w) & 1;
      const uint32_t block_off = stage_bias(common.y ? w & 1 : 0) + sw128_offset(m, 0);
      if (p.gate != nullptr && unit.y + m < p.S)  // read at the end; (a missing unit has no query below S)
        asm volatile("prefetch.global.L2 [%0];" ::"l"(p.gate + unit.x * p.g_br + common.z * p.g_h + (long long)(unit.y + m) * p.g_s));
      float row_max = 0.f, row_sum = 0.f;  // row_max: reference point of the exponentials, in raw score units
      const uint32_t* mask_row = nullptr;
      if (kMasked) {
        const int b = unit.x / p.R;
        mask_row = p.key_mask + b * p.km_b + (unit.x - b * p.R) * p.km_r;
      }
      bool have_anchor = false;            // masked form: a key tile with a valid key has been seen

      for (int kt = 0; kt < my_tiles; ++kt) {
        // Scores ready; K, V and bias of the tile loaded (they are, or it would have no scores: the wait makes the
        // copies' writes visible to this thread); P·V of the tile before the previous one complete, so that this
        // tile's P buffer may be overwritten.
        const int pb = ct & 1;
        ok = mbar_wait2_warp(bars + (S_FULL + w) * 8, pb, bars + (KV_FULL + stage) * 8, stage_phase, abort_flag);
        if (!ok) break;
        tc_fence_after();
        const uint32_t o_done = bars + (O_FULL + 2 * w + pb) * 8;
        const uint32_t o_parity = ((ct >> 1) & 1) ^ 1;
        const uint32_t p_addr = lane_taddr + p_column(w, pb);
        ++ct;
        const uint32_t bias0 = base + kSmStage + stage * kStageBytes + block_off;
        if (++stage == kStages) stage = 0, stage_phase ^= 1;
        const int rem = len - kt * kKTile;  // valid keys in this tile
        if (uniform) {
          // No valid key, eager semantics: every logit is the same, so every probability of the tile is 1 (0 past
          // the last key) and the output becomes the mean of V.  No scores are read, no exponentials taken.
          __syncwarp();
          mbar_arrive_warp(bars + (S_FREE + (w & 1)) * 8);
          ok = mbar_wait_warp(o_done, o_parity, abort_flag);
          if (!ok) break;
          tc_fence_after();
#pragma unroll
          for (int half = 0; half < 2; ++half) {
            uint32_t pk[16];
#pragma unroll
            for (int e = 0; e < 16; ++e) {
              const int j0 = half * 32 + 2 * e;
              pk[e] = j0 + 1 < rem ? 0x3F803F80u : (j0 < rem ? 0x00003F80u : 0u);  // bf16 pairs of 1.0
            }
            tmem_st16(p_addr + half * 16, pk);
          }
          row_sum += float(rem < kKTile ? rem : kKTile);
          tmem_st_wait();
          tc_fence_before();
          __syncwarp();
          mbar_arrive_warp(bars + (P_FULL + 2 * w + pb) * 8);
          continue;
        }
        float s2[64];  // raw scores of this row against the tile's 64 keys
        tmem_ld64(s_addr, s2);
        tmem_ld_wait();
        tc_fence_before();
        __syncwarp();
        mbar_arrive_warp(bars + (S_FREE + (w & 1)) * 8);  // the S buffer can take the next tile's scores

        // p = 2^(c * (s + bias - row_max)); bf16 pairs go back to TMEM as the A operand of P·V.  16 keys at a time,
        // the bias of the next 16 requested before the exponentials of these, so that its latency and unpacking
        // hide behind the special-function unit.
        // The reference point of the exponentials is the row's first valid score.  No maximum is searched: the
        // largest probability is at least 1, fp32 sums, fp32 O and bf16 P share the fp32 exponent range, so
        // probabilities far above 1 lose nothing, and a tile whose sum leaves the safe range is redone below.
        const bool plain = !kMasked && rem >= kKTile;
        uint64_t sum2[2] = {0ull, 0ull};  // independent packed partial sums
        if (plain) {
          uint4 x[2][2];
          x[0][0] = lds128(bias0), x[0][1] = lds128(bias0 ^ 16);
          if (kt == 0) row_max = s2[0] + bf16_lo(x[0][0].x);
          const float nmc = -row_max * c;
          const uint64_t nmc2 = pack_f32x2(nmc, nmc);
#pragma unroll
          for (int ch = 0; ch < 4; ++ch) {
            if (ch < 3) {
              x[(ch + 1) & 1][0] = lds128(bias0 ^ ((2 * ch + 2) << 4));
              x[(ch + 1) & 1][1] = lds128(bias0 ^ ((2 * ch + 3) << 4));
            }
            uint32_t pk[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) {
              const int j0 = ch * 16 + 2 * e;
              const uint4& xx = x[ch & 1][e >> 2];
              const uint32_t bw = (e & 3) == 0 ? xx.x : (e & 3) == 1 ? xx.y : (e & 3) == 2 ? xx.z : xx.w;
              const uint64_t t2 = fma_f32x2(pack_f32x2(bf16_lo(bw), bf16_hi(bw)), c2, nmc2);
              float d0, d1;
              unpack_f32x2(fma_f32x2(pack_f32x2(s2[j0], s2[j0 + 1]), c2, t2), d0, d1);
              const float p0 = ex2_approx(d0), p1 = ex2_approx(d1);
              sum2[e & 1] = add_f32x2(sum2[e & 1], pack_f32x2(p0, p1));
              pk[e] = pack_bf16x2(p0, p1);
            }
            if (ch == 0) {
              ok = mbar_wait_warp(o_done, o_parity, abort_flag);
              tc_fence_after();
            }
            tmem_st8(p_addr + ch * 8, pk);
          }
        } else {
          // last tile (keys past the row length) and masked form
#pragma unroll
          for (int ch = 0; ch < 8; ++ch) {
            const uint4 x = lds128(bias0 ^ (ch << 4));
            const uint32_t xw[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const int j0 = ch * 8 + 2 * e;
              unpack_f32x2(add_f32x2(pack_f32x2(s2[j0], s2[j0 + 1]), pack_f32x2(bf16_lo(xw[e]), bf16_hi(xw[e]))), s2[j0],
                           s2[j0 + 1]);
            }
          }
          bool find_anchor = false;
          if (kMasked) {
            // Keys may be switched off anywhere in the row (the same bits for every query of the unit): the warp
            // expands the tile's bits to 0 / -inf in its own scratch and adds them.  Keys past the row length have
            // their bit clear.  A tile without any valid key yields zeros (the reference point stays 0 until a tile
            // with a valid key comes).
            const uint32_t* mrow = mask_row + kt * 2;
            const int words = (p.S + 31) >> 5;
            const uint32_t m0 = __ldg(mrow), m1 = kt * 2 + 1 < words ? __ldg(mrow + 1) : 0u;
            const uint32_t scratch = base + kSmMask + warp * 256;
            {
              const uint32_t pair = (lane < 16 ? m0 : m1) >> ((2 * lane) & 31);
              __syncwarp();  // the previous tile's reads are done
              asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(scratch + lane * 8),
                           "r"((pair & 1u) ? 0u : 0xFF800000u), "r"((pair & 2u) ? 0u : 0xFF800000u)
                           : "memory");
              __syncwarp();
            }
#pragma unroll
            for (int ch = 0; ch < 16; ++ch) {
              const uint4 x = lds128(scratch + ch * 16);
              unpack_f32x2(add_f32x2(pack_f32x2(s2[ch * 4], s2[ch * 4 + 1]),
                                     pack_f32x2(__uint_as_float(x.x), __uint_as_float(x.y))), s2[ch * 4], s2[ch * 4 + 1]);
              unpack_f32x2(add_f32x2(pack_f32x2(s2[ch * 4 + 2], s2[ch * 4 + 3]),
                                     pack_f32x2(__uint_as_float(x.z), __uint_as_float(x.w))), s2[ch * 4 + 2], s2[ch * 4 + 3]);
            }
            find_anchor = !have_anchor && (m0 | m1) != 0u;
            have_anchor = have_anchor || find_anchor;
          }
          if (rem < kKTile) {
#pragma unroll
            for (int j = 0; j < 64; ++j)
              if (j >= rem) s2[j] = -INFINITY;
          }
          if (!kMasked && kt == 0) {
            row_max = s2[0];
          } else if (kMasked && find_anchor) {
            float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};  // four independent chains
#pragma unroll
            for (int j = 0; j < 32; ++j) mx[j & 3] = max3_f32(mx[j & 3], s2[2 * j], s2[2 * j + 1]);
            row_max = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));  // finite: the tile holds a valid key
          }
          const float nmc = -row_max * c;
          const uint64_t nmc2 = pack_f32x2(nmc, nmc);
#pragma unroll
          for (int ch = 0; ch < 4; ++ch) {
            uint32_t pk[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) {
              const int j0 = ch * 16 + 2 * e;
              float d0, d1;
              unpack_f32x2(fma_f32x2(pack_f32x2(s2[j0], s2[j0 + 1]), c2, nmc2), d0, d1);
              const float p0 = ex2_approx(d0), p1 = ex2_approx(d1);
              sum2[e & 1] = add_f32x2(sum2[e & 1], pack_f32x2(p0, p1));
              pk[e] = pack_bf16x2(p0, p1);
            }
            if (ch == 0) {
              ok = mbar_wait_warp(o_done, o_parity, abort_flag);
              tc_fence_after();
            }
            tmem_st8(p_addr + ch * 8, pk);
          }
        }
        if (!ok) break;
        float tile_sum;
        {
          float a0, a1;
          unpack_f32x2(add_f32x2(sum2[0], sum2[1]), a0, a1);
          tile_sum = a0 + a1;
        }
        // Rare: some score lies so far above the reference point that the tile's sum leaves the safe range (or
        // overflowed).  Move the reference point of the affected rows to the tile's maximum, rescale what has
        // been accumulated (once the previous tile's P·V is complete) and redo the tile.  The scores are gone by now
        // (keeping them would cost the usual path 64 registers), so they are computed again from Q, K and the bias
        // in shared memory, which the MMA warps hand back only after this tile's P·V.
        if (__any_sync(0xffffffffu, !(tile_sum < kRebaseSum))) {
          // (ct counts this tile already: the previous one has number ct - 2)
          if (ct > 1) ok = mbar_wait_warp(bars + (O_FULL + 2 * w + (ct & 1)) * 8, ((ct - 2) >> 1) & 1, abort_flag);
          if (!ok) break;
          tc_fence_after();
          uint4 qv[4];
#pragma unroll
          for (int ch = 0; ch < 4; ++ch) qv[ch] = lds128(base + kSmQ + (ib * kUnits + w) * 8192 + sw64_offset(m, ch));
          const uint32_t k0 = bias0 - block_off + stage_k(info->two_blocks ? w >> 1 : w);
          auto score = [&](int key) {
            float d = -INFINITY;
            bool valid = key < rem;
            if (kMasked) {
              const int word = kt * 2 + (key >> 5);
              valid = word < ((p.S + 31) >> 5) &&
                      ((__ldg(mask_row + word) >> (key & 31)) & 1u);
            }
            if (valid) {
              uint32_t b16;
              asm volatile("{\n.reg .b16 h;\nld.shared.b16 h, [%1];\ncvt.u32.u16 %0, h;\n}"
                           : "=r"(b16)
                           : "r"((bias0 ^ ((key >> 3) << 4)) + (key & 7) * 2));
              d = bf16_lo(b16);
#pragma unroll
              for (int ch = 0; ch < 4; ++ch) {
                const uint4 kv = lds128(k0 + sw64_offset(key, ch));
                d = fmaf(bf16_lo(qv[ch].x), bf16_lo(kv.x), fmaf(bf16_hi(qv[ch].x), bf16_hi(kv.x), d));
                d = fmaf(bf16_lo(qv[ch].y), bf16_lo(kv.y), fmaf(bf16_hi(qv[ch].y), bf16_hi(kv.y), d));
                d = fmaf(bf16_lo(qv[ch].z), bf16_lo(kv.z), fmaf(bf16_hi(qv[ch].z), bf16_hi(kv.z), d));
                d = fmaf(bf16_lo(qv[ch].w), bf16_lo(kv.w), fmaf(bf16_hi(qv[ch].w), bf16_hi(kv.w), d));
              }
            }
            return d;
          };
          float cm = -INFINITY;
#pragma unroll 1
          for (int key = 0; key < kKTile; ++key) cm = fmaxf(cm, score(key));
          const float new_max = (tile_sum < kRebaseSum) ? row_max : cm;
          const float alpha = ex2_approx((row_max - new_max) * c);  // 1 for rows that keep their reference point
          tmem_st_wait();
          if (kt > 0) {
#pragma unroll
            for (int part = 0; part < 2; ++part) {
              uint32_t t[16];
              tmem_ld16(o_addr + part * 16, t);
              tmem_ld_wait();
#pragma unroll
              for (int j = 0; j < 16; ++j) t[j] = __float_as_uint(__uint_as_float(t[j]) * alpha);
              tmem_st16(o_addr + part * 16, t);
            }
          }
          row_sum *= alpha;
          row_max = new_max;
          tile_sum = 0.f;
#pragma unroll 1
          for (int pair = 0; pair < kKTile / 2; ++pair) {
            const float p0 = ex2_approx((score(2 * pair) - row_max) * c), p1 = ex2_approx((score(2 * pair + 1) - row_max) * c);
            tile_sum += p0 + p1;
            __syncwarp();
            tmem_st1(p_addr + pair, pack_bf16x2(p0, p1));
          }
        }
        row_sum += tile_sum;
        tmem_st_wait();
        tc_fence_before();
        __syncwarp();
        mbar_arrive_warp(bars + (P_FULL + 2 * w + pb) * 8);
      }
      if (!ok) break;
      // tiles of the item that only longer rows have
      for (int kt = max(my_tiles, 0), all = info->tiles; kt < all; ++kt)
        if (++stage == kStages) stage = 0, stage_phase ^= 1;
      // The info is read again here: kept over the tiles it cost registers that the tile loop spilled (512 tokens 204 ->
      // 199 us, the masked form at 333 tokens 136 -> 106; the unmasked form still spills two registers).
      const int br = info->unit[w].br, q = info->unit[w].q0 + m, h = info->h;  // pair row, query position
      mbar_arrive_warp_after_reads(bars + (Q_EMPTY + ib) * 8);
      if (my_tiles < 0) continue;  // the item has no such unit
      __nv_bfloat16* out_row = p.out + br * p.o_br + (long long)q * p.o_s + h * p.o_h;
      if (my_tiles == 0) {  // no valid key and "zeros" semantics
        if (q < p.S) {
#pragma unroll
          for (int j = 0; j < 4; ++j) reinterpret_cast<uint4*>(out_row)[j] = make_uint4(0, 0, 0, 0);
          if (p.lse) p.lse[((long long)br * p.S + q) * kHeads + h] = -INFINITY;
        }
        continue;
      }
      const __nv_bfloat16* gate_row = p.gate + br * p.g_br + h * p.g_h + (long long)q * p.g_s;
      // the unit's output: O (in TMEM) / row_sum * gate; the gate row is fetched while the last P·V runs
      uint4 gv[4];
      if (p.gate != nullptr && q < p.S) {
#pragma unroll
        for (int j = 0; j < 4; ++j) gv[j] = __ldg(reinterpret_cast<const uint4*>(gate_row) + j);
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) gv[j] = make_uint4(0x3F803F80u, 0x3F803F80u, 0x3F803F80u, 0x3F803F80u);  // 1.0
      }
      const float inv = 1.f / row_sum;
      ok = mbar_wait_warp(bars + (O_FULL + 2 * w + ((ct - 1) & 1)) * 8, ((ct - 1) >> 1) & 1, abort_flag);
      if (!ok) break;
      tc_fence_after();
      uint32_t pk[16];
      {
        uint32_t t[32];
        tmem_ld32(o_addr, t);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const uint32_t gw[4] = {gv[j].x, gv[j].y, gv[j].z, gv[j].w};
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int k = j * 8 + 2 * e;
            pk[j * 4 + e] = pack_bf16x2(__uint_as_float(t[k]) * (bf16_lo(gw[e]) * inv),
                                        __uint_as_float(t[k + 1]) * (bf16_hi(gw[e]) * inv));
          }
        }
      }
      tc_fence_before();
      if (q < p.S) {
        if (p.wide_store) {  // two full 32-byte sectors per row instead of four half sectors
          stg256(out_row, pk);
          stg256(out_row + 16, pk + 8);
        } else {
#pragma unroll
          for (int j = 0; j < 4; ++j)
            reinterpret_cast<uint4*>(out_row)[j] = make_uint4(pk[j * 4], pk[j * 4 + 1], pk[j * 4 + 2], pk[j * 4 + 3]);
        }
        if (p.lse)
          p.lse[((long long)br * p.S + q) * kHeads + h] =
              uniform ? -INFINITY : 0.6931471805599453f * (row_max * c + __log2f(row_sum));
      }
    }
  }

  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (warp == 17) {
    tc_fence_after();
    tmem_dealloc(tmem_base, kTmemCols);
  }
  if (threadIdx.x == 0 && *abort_flag) *p.status = B200TA_ERR_DEVICE_WAIT;
}

int launch_attention(const void* q, const void* k, const void* v, const void* gate, int64_t s_br, int64_t s_h,
                     int64_t s_s, const void* bias, int64_t bs_b, int64_t bs_h, int64_t bs_q,
                     const int32_t* lengths, int64_t ls_b, int64_t ls_r, const uint32_t* key_mask, int64_t km_b,
                     int64_t km_r, void* out, int64_t os_br, int64_t os_s, int64_t os_h, float* lse,
                     float softmax_scale, int empty_row_mode, int B, int R, int S, int S_pad, void* stream) {
  using namespace b200ta;
  B200TA_REQUIRE(q && k && v && bias && out, "attention: NULL pointer");
  B200TA_REQUIRE(B > 0 && R > 0 && S > 0, "attention: bad sizes B=%d R=%d S=%d", B, R, S);
  B200TA_REQUIRE(S_pad >= S && S_pad % 8 == 0, "attention: S_pad=%d must be a multiple of 8 and >= S=%d", S_pad, S);
  B200TA_REQUIRE(softmax_scale > 0.f, "attention: softmax_scale must be positive");
  B200TA_REQUIRE(s_br % 8 == 0 && s_h % 8 == 0 && s_s % 8 == 0 && s_s > 0, "attention: q/k/v strides must be multiples of 8 elements");
  B200TA_REQUIRE(bs_b % 8 == 0 && bs_h % 8 == 0 && bs_q % 8 == 0 && bs_q > 0, "attention: bias strides must be multiples of 8 elements");
  B200TA_REQUIRE(os_br % 8 == 0 && os_s % 8 == 0 && os_h % 8 == 0, "attention: out strides must be multiples of 8 elements");
  B200TA_REQUIRE((reinterpret_cast<uintptr_t>(out) & 15u) == 0 && (gate == nullptr || (reinterpret_cast<uintptr_t>(gate) & 15u) == 0),
                 "attention: out and gate must be 16-byte aligned");
  B200TA_REQUIRE(empty_row_mode == B200TA_EMPTY_ROW_ZEROS || empty_row_mode == B200TA_EMPTY_ROW_UNIFORM,
                 "attention: unknown empty_row_mode %d", empty_row_mode);
  DeviceState* st = nullptr;
  int rc = get_device_state(&st);
  if (rc != B200TA_OK) return rc;
  B200TA_REQUIRE(int64_t(B) * kHeads * R * ((S + kQTile - 1) / kQTile) < (int64_t(1) << 31), "attention: too many work items");
  AttnParams p{};
  p.plan = split_items(B, R, S, st->num_sms);

  CUtensorMap tm_q, tm_k, tm_v, tm_bias;
  {
    uint64_t dims[4] = {uint64_t(kHeadDim), uint64_t(S), uint64_t(kHeads), uint64_t(B) * R};
    uint64_t strides[3] = {uint64_t(s_s) * 2, uint64_t(s_h) * 2, B * R == 1 ? 64u : uint64_t(s_br) * 2};
    uint32_t box[4] = {32, kQTile, 1, 1};
    rc = encode_tensor_map(&tm_q, q, 2, 4, dims, strides, box, SWZ_64, "attention q");
    box[1] = kKTile;
    if (rc == B200TA_OK) rc = encode_tensor_map(&tm_k, k, 2, 4, dims, strides, box, SWZ_64, "attention k");
    if (rc == B200TA_OK) rc = encode_tensor_map(&tm_v, v, 2, 4, dims, strides, box, SWZ_64, "attention v");
    if (rc != B200TA_OK) return rc;
  }
  {
    uint64_t dims[4] = {uint64_t(S_pad), uint64_t(S), uint64_t(kHeads), uint64_t(B)};
    uint64_t strides[3] = {uint64_t(bs_q) * 2, uint64_t(bs_h) * 2, B == 1 ? 64u : uint64_t(bs_b) * 2};
    uint32_t box[4] = {kKTile, kQTile, 1, 1};
    rc = encode_tensor_map(&tm_bias, bias, 2, 4, dims, strides, box, SWZ_128, "attention bias");
    if (rc != B200TA_OK) return rc;
  }

  p.B = B, p.R = R, p.S = S, p.S_pad = S_pad;
  p.lengths = lengths;
  p.ls_b = ls_b, p.ls_r = ls_r;
  p.key_mask = key_mask;
  p.km_b = km_b, p.km_r = km_r;
  p.gate = static_cast<const __nv_bfloat16*>(gate);
  p.g_br = s_br, p.g_h = s_h, p.g_s = s_s;
  p.out = static_cast<__nv_bfloat16*>(out);
  p.o_br = os_br, p.o_s = os_s, p.o_h = os_h;
  p.lse = lse;
  p.scale_log2 = softmax_scale * 1.4426950408889634f;
  p.empty_uniform = empty_row_mode == B200TA_EMPTY_ROW_UNIFORM ? 1 : 0;
  p.wide_store = (reinterpret_cast<uintptr_t>(out) & 31u) == 0 && os_br % 16 == 0 && os_s % 16 == 0 && os_h % 16 == 0;
  p.status = st->status_dev;

  const int grid = p.plan.num_items < st->num_sms ? p.plan.num_items : st->num_sms;
  if (key_mask != nullptr) {
    B200TA_REQUIRE(lengths != nullptr, "attention: the masked form needs the row lengths (last valid key + 1) as well");
    return launch_kernel(st, kKernelAttentionMasked, attention_kernel<true>, dim3(grid), kThreads, kSmDynamic, stream, tm_q,
                         tm_k, tm_v, tm_bias, p);
  }
  return launch_kernel(st, kKernelAttention, attention_kernel<false>, dim3(grid), kThreads, kSmDynamic, stream, tm_q, tm_k,
                       tm_v, tm_bias, p);
}

}  // namespace
}  // namespace b200ta

extern "C" {

int b200ta_attention(const void* q, const void* k, const void* v, const void* gate, int64_t s_br, int64_t s_h,
                     int64_t s_s, const void* bias, int64_t bs_b, int64_t bs_h, int64_t bs_q,
                     const int32_t* lengths, int64_t ls_b, int64_t ls_r, void* out, int64_t os_br, int64_t os_s,
                     int64_t os_h, float* lse, float softmax_scale, int empty_row_mode, int B, int R, int S,
                     int S_pad, void* stream) {
  return b200ta::launch_attention(q, k, v, gate, s_br, s_h, s_s, bias, bs_b, bs_h, bs_q, lengths, ls_b, ls_r, nullptr, 0,
                                  0, out, os_br, os_s, os_h, lse, softmax_scale, empty_row_mode, B, R, S, S_pad, stream);
}

int b200ta_attention_masked(const void* q, const void* k, const void* v, const void* gate, int64_t s_br, int64_t s_h,
                            int64_t s_s, const void* bias, int64_t bs_b, int64_t bs_h, int64_t bs_q,
                            const int32_t* lengths, int64_t ls_b, int64_t ls_r, const uint32_t* key_mask,
                            int64_t km_b, int64_t km_r, void* out, int64_t os_br, int64_t os_s, int64_t os_h,
                            float* lse, float softmax_scale, int empty_row_mode, int B, int R, int S, int S_pad,
                            void* stream) {
  if (key_mask == nullptr) return b200ta::fail(B200TA_ERR_INVALID, "attention_masked: key_mask must not be NULL");
  return b200ta::launch_attention(q, k, v, gate, s_br, s_h, s_s, bias, bs_b, bs_h, bs_q, lengths, ls_b, ls_r, key_mask,
                                  km_b, km_r, out, os_br, os_s, os_h, lse, softmax_scale, empty_row_mode, B, R, S, S_pad,
                                  stream);
}

}  // extern "C"
