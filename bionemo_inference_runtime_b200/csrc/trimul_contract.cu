// Triangle-multiplication contraction for sm_100a: per batch item b and hidden channel d
//   x[b, d, i, j] = sum_k a[b, d, i, k] * b[b, d, j, k]
// i.e. 128 * B independent [N x N] = [N x N] · [N x N]ᵀ bf16 GEMMs with fp32 accumulation.  The projection kernel
// writes a and b channel-major with the contraction index k contiguous (for the incoming node it walks the pair
// tensor through swapped strides, so the same layout serves both directions), so both operands are K-major.
//
// Bound: the operand tiles' way from L2 (12.8 TB/s reached).  A CTA computes [256 x 256] tiles, two accumulators of 128 rows
// side by side in all of tensor memory: 64 KiB per 64-wide K step of 1096 clocks of MMAs, its epilogue behind the next
// tile's loads.  [128 x 256] tiles with two accumulators, the epilogue of one beside the MMAs of the other, ask for 48 KiB
// per 548 clocks, which L2 does not deliver: 106 us at 768 tokens, now 98 (1180 TFLOP/s).  Column tiles are as wide as the
// token count needs (a multiple of 32), a lower half without rows is left out.  At 512 tokens (45 us) and 64 x 256
// (522 us) the bytes from HBM bound it.
//
// TMA loads [256 x 64] operand tiles into a three-stage ring, one warp issues tcgen05.mma (M 128, N up to 256, K 16), and
// eight epilogue warps (TMEM lane = output row) convert the finished accumulators to bf16, stage 32 rows of 64 bytes each
// and store them by TMA (a lane's own 32-byte stores of 32 rows occupy the load-store unit for some 56 clocks).
//
// Warp roles (320 threads): warps 0-7 epilogue, warp 8 TMA producer, warp 9 MMA issuer / TMEM owner.
#include "common.cuh"
#include "layout.h"

namespace b200ta {
namespace {

constexpr int kThreads = 320;
constexpr int kBM = 256, kBN = 256, kBK = 64;
constexpr int kStages = 3;
constexpr int kStageBytes = (kBM + kBN) * kBK * 2;  // 64 KiB
constexpr int kSmOut = kStages * kStageBytes;       // 8 warps x 2 slabs x 2 KiB: 32 rows of 64 bytes
constexpr int kSmBars = kSmOut + 8 * 2 * 2048;
enum Bar { FULL = 0, EMPTY = kStages, ACC_FULL = 2 * kStages, ACC_EMPTY = 2 * kStages + 2, NUM_BARS = 2 * kStages + 4 };
constexpr int kSmTotal = kSmBars + 128;
constexpr int kSmDynamic = kSmTotal + 1024;

struct ContractParams {
  int N;          // tokens
  int planes;     // B * hidden
  int hidden;     // channels per batch item (a planes first, b planes next)
  int tiles_m, tiles_n, num_tiles;
  int width;  // columns of a tile, a multiple of 32
  int* status;
};

struct Tile {
  int plane, a_plane, b_plane, m0, n0;
};
__device__ __forceinline__ Tile decode_tile(const ContractParams& p, int t) {
  Tile r;
  const int nt = t % p.tiles_n;
  t /= p.tiles_n;
  const int mt = t % p.tiles_m;
  r.plane = t / p.tiles_m;
  const int b = r.plane / p.hidden, d = r.plane - b * p.hidden;
  r.a_plane = b * 2 * p.hidden + d;
  r.b_plane = r.a_plane + p.hidden;
  r.m0 = mt * kBM, r.n0 = nt * p.width;
  return r;
}

__global__ void __launch_bounds__(kThreads, 1)
trimul_contract_kernel(const __grid_constant__ CUtensorMap tm_ab, const __grid_constant__ CUtensorMap tm_x,
                       const ContractParams p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* gen = smem_raw + (base - smem_u32(smem_raw));
  const uint32_t bars = base + kSmBars;
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(gen + kSmBars + NUM_BARS * 8);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(gen + kSmBars + NUM_BARS * 8 + 8);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    abort_flag[0] = 0, abort_flag[1] = 0;
    for (int i = 0; i < kStages; ++i) {
      mbar_init(bars + (FULL + i) * 8, 1);
      mbar_init(bars + (EMPTY + i) * 8, 1);
    }
    for (int i = 0; i < 2; ++i) {
      mbar_init(bars + (ACC_FULL + i) * 8, 1);
      mbar_init(bars + (ACC_EMPTY + i) * 8, 4);
    }
    fence_mbar_init();
  }
  if (warp == 9) {
    tmem_alloc(smem_u32(const_cast<uint32_t*>(tmem_slot)), 512);
    pdl_trigger();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  const int my_tiles = (p.num_tiles - 1 - int(blockIdx.x)) / int(gridDim.x) + 1;
  const int ksteps = (p.N + kBK - 1) / kBK;

  if (warp == 8) {
    // ------------------------------------------------------------------ TMA producer
    if (lane == 0) {
      tma_prefetch_desc(&tm_ab);
      pdl_wait();  // (for the whole block: the epilogue stores only what came of these loads)
      int g = 0;  // ring position
      bool ok = true;
      const bool wide = p.width > 128;
      for (int i = 0; ok && i < my_tiles; ++i) {
        const Tile t = decode_tile(p, blockIdx.x + i * gridDim.x);
        const bool lower = t.m0 + 128 < p.N;
        for (int ks = 0; ks < ksteps; ++ks, ++g) {
          const int stage = g % kStages;
          ok = mbar_wait(bars + (EMPTY + stage) * 8, ((g / kStages) & 1) ^ 1, abort_flag);
          if (!ok) break;
          const uint32_t full = bars + (FULL + stage) * 8;
          const uint32_t sa = base + stage * kStageBytes, sb = sa + kBM * kBK * 2;
          mbar_expect_tx(full, (2 + lower + wide) * 128 * kBK * 2);
          tma_load_3d(sa, &tm_ab, full, ks * kBK, t.m0, t.a_plane);
          if (lower) tma_load_3d(sa + 128 * kBK * 2, &tm_ab, full, ks * kBK, t.m0 + 128, t.a_plane);
          tma_load_3d(sb, &tm_ab, full, ks * kBK, t.n0, t.b_plane);
          if (wide) tma_load_3d(sb + 128 * kBK * 2, &tm_ab, full, ks * kBK, t.n0 + 128, t.b_plane);
        }
      }
      // If the loop was abandoned, give copies still in flight a bounded chance to land.
      if (*abort_flag)
        for (int j = g > kStages ? g - kStages : 0; j < g; ++j)
          mbar_wait(bars + (FULL + j % kStages) * 8, (j / kStages) & 1, abort_flag + 1);
    }
  } else if (warp == 9) {
    // ------------------------------------------------------------------ MMA issuer (whole warp, one lane issues)
    const uint32_t idesc = make_idesc_bf16(128, p.width);
    const uint32_t tb = __shfl_sync(0xffffffffu, tmem_base, 0);
    int g = 0;
    bool ok = true;
    for (int i = 0; ok && i < my_tiles; ++i) {
      const Tile t = decode_tile(p, blockIdx.x + i * gridDim.x);
      const bool lower = t.m0 + 128 < p.N;
      for (int ks = 0; ks < ksteps; ++ks, ++g) {
        const int stage = g % kStages;
        ok = mbar_wait_warp(bars + (FULL + stage) * 8, (g / kStages) & 1, abort_flag);
        // each accumulator is handed over on its own, so that a tile's first half starts while the second half of the
        // tile before is still being stored (both are handed over each tile, also when the lower half was left out)
        if (ok && ks == 0) ok = mbar_wait_warp(bars + ACC_EMPTY * 8, (i & 1) ^ 1, abort_flag);
        if (!ok) break;
        tc_fence_after();
        const uint32_t sa = base + stage * kStageBytes;
        // [rows][64 k] tiles with 128-byte swizzle: 8-row groups 1 KiB apart; a K step of 16 = 32 bytes
        const uint64_t da = smem_desc<16, 1024, kLayoutSw128>(sa);
        const uint64_t db = smem_desc<16, 1024, kLayoutSw128>(sa + kBM * kBK * 2);
#pragma unroll
        for (int k = 0; k < kBK / 16; ++k) umma_ss_warp(tb, da + k * 2, db + k * 2, idesc, (ks > 0 || k > 0) ? 1u : 0u);
        if (ks == ksteps - 1) umma_commit_warp(bars + ACC_FULL * 8);
        if (ks == 0) {
          ok = mbar_wait_warp(bars + (ACC_EMPTY + 1) * 8, (i & 1) ^ 1, abort_flag);
          if (!ok) break;
          tc_fence_after();
        }
        if (lower) {
#pragma unroll
          for (int k = 0; k < kBK / 16; ++k)
            umma_ss_warp(tb + kBN, da + (16384 >> 4) + k * 2, db + k * 2, idesc, (ks > 0 || k > 0) ? 1u : 0u);
        }
        umma_commit_warp(bars + (EMPTY + stage) * 8);  // the stage is free once these MMAs have read it
      }
      if (!ok) break;
      umma_commit_warp(bars + (ACC_FULL + 1) * 8);
    }
  } else {
    // ------------------------------------------------------------------ epilogue warps
    const int half = warp >> 2;             // which accumulator
    const int m = (warp & 3) * 32;          // first output row of the warp == TMEM lane
    const uint32_t acc = tmem_base + (uint32_t(m) << 16) + half * kBN;
    const uint32_t slab0 = base + kSmOut + warp * 4096;
    uint32_t stores = 0;  // the slabs take turns over all stores, whatever the number of a tile's
    bool ok = true;
    for (int i = 0; ok && i < my_tiles; ++i) {
      const Tile t = decode_tile(p, blockIdx.x + i * gridDim.x);
      ok = mbar_wait_warp(bars + (ACC_FULL + half) * 8, i & 1, abort_flag);
      if (!ok) break;
      tc_fence_after();
      const int row0 = t.m0 + half * 128 + m;
      if (row0 < p.N) {
        const int columns = p.width < p.N - t.n0 ? p.width : p.N - t.n0;
        for (int c = 0; c < columns; c += 32, ++stores) {
          uint32_t a[32];
          tmem_ld32(acc + c, a);
          const uint32_t slab = slab0 + (stores & 1) * 2048;
          if (lane == 0) tma_store_wait_read<1>();  // the store before the previous one has read this slab
          __syncwarp();
          tmem_ld_wait();
          uint32_t packed[16];
#pragma unroll
          for (int j = 0; j < 16; ++j) packed[j] = pack_bf16x2(__uint_as_float(a[2 * j]), __uint_as_float(a[2 * j + 1]));
#pragma unroll
          for (int j = 0; j < 4; ++j)
            sts128(slab + sw64_offset(lane, j), make_uint4(packed[j * 4], packed[j * 4 + 1], packed[j * 4 + 2], packed[j * 4 + 3]));
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            // rows past the token count and columns past the row pitch are not written; columns between the token count
            // and the pitch receive zeros (the operand rows past the token count are zero-filled by the loads)
            tma_store_3d(&tm_x, slab, t.n0 + c, row0, t.plane);
            tma_store_commit();
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      mbar_arrive_warp(bars + (ACC_EMPTY + half) * 8);
    }
    if (lane == 0) tma_store_wait_all();
  }

  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (warp == 9) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
  if (threadIdx.x == 0 && *abort_flag) *p.status = B200TA_ERR_DEVICE_WAIT;
}

}  // namespace
}  // namespace b200ta

extern "C" {

int b200ta_trimul_contract(const void* ab, void* x, int B, int N, int64_t pitch, void* stream) {
  using namespace b200ta;
  B200TA_REQUIRE(ab && x, "trimul_contract: NULL pointer");
  B200TA_REQUIRE(B > 0 && N > 0, "trimul_contract: bad sizes B=%d N=%d", B, N);
  B200TA_REQUIRE(pitch >= N && pitch % 16 == 0, "trimul_contract: pitch=%lld must be a multiple of 16 and >= N=%d",
                 (long long)pitch, N);
  B200TA_REQUIRE((reinterpret_cast<uintptr_t>(ab) & 31u) == 0 && (reinterpret_cast<uintptr_t>(x) & 31u) == 0,
                 "trimul_contract: buffers must be 32-byte aligned");
  DeviceState* st = nullptr;
  int rc = get_device_state(&st);
  if (rc != B200TA_OK) return rc;

  constexpr int kHidden = kC;
  CUtensorMap tm_ab;
  {
    // (k, row, plane): rows and k past N read as zero
    uint64_t dims[3] = {uint64_t(N), uint64_t(N), uint64_t(B) * 2 * kHidden};
    uint64_t strides[2] = {uint64_t(pitch) * 2, uint64_t(pitch) * N * 2};
    uint32_t box[3] = {kBK, 128, 1};
    rc = encode_tensor_map(&tm_ab, ab, 2, 3, dims, strides, box, SWZ_128, "trimul a/b planes");
    if (rc != B200TA_OK) return rc;
  }
  CUtensorMap tm_x;
  {
    // (column, row, plane): an epilogue warp's slab
    uint64_t dims[3] = {uint64_t(pitch), uint64_t(N), uint64_t(B) * kHidden};
    uint64_t strides[2] = {uint64_t(pitch) * 2, uint64_t(pitch) * N * 2};
    uint32_t box[3] = {32, 32, 1};
    rc = encode_tensor_map(&tm_x, x, 2, 3, dims, strides, box, SWZ_64, "trimul x planes");
    if (rc != B200TA_OK) return rc;
  }
  ContractParams p{};
  p.N = N, p.planes = B * kHidden, p.hidden = kHidden;
  p.tiles_m = (N + kBM - 1) / kBM, p.tiles_n = (N + kBN - 1) / kBN;
  const int64_t tiles = int64_t(p.planes) * p.tiles_m * p.tiles_n;
  B200TA_REQUIRE(tiles < (int64_t(1) << 31), "trimul_contract: too many tiles");
  p.num_tiles = int(tiles);
  p.width = ((N + p.tiles_n - 1) / p.tiles_n + 31) / 32 * 32;
  p.status = st->status_dev;

  const int grid = p.num_tiles < st->num_sms ? p.num_tiles : st->num_sms;
  return launch_kernel(st, kKernelContract, trimul_contract_kernel, dim3(grid), kThreads, kSmDynamic, stream, tm_ab, tm_x, p);
}

}  // extern "C"
