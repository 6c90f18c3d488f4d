// Triangle-multiplication input stage for sm_100a:
//   x̂        = LayerNorm_in(z)
//   ab[ch]   = sigmoid(x̂·W_g[ch] + b_g) * (x̂·W_p[ch] + b_p) * mask          ch = a(0..127) | b(128..255)
// written channel-major, ab[b][ch][r][s], so that the contraction kernel finds the index it sums over (s)
// contiguous.  The incoming node calls this with the pair strides swapped (rows r = pair columns).
//
// The GEMM is computed transposed, D[channel, position] = W'[channel, :] · z[position, :]ᵀ: a TMEM lane is a channel, so
// that every epilogue thread owns one channel of consecutive positions - one contiguous run of the channel-major output.
// The folded weight rows (four blocks of 128: gate and value of the a and of the b channels) stay in tensor memory as the
// A operand for the whole kernel (256 columns), the raw tile of 128 positions is the B operand.
//
// Bound: first the writes, 512 of 768 bytes per position: at 768 tokens the kernel takes 100 us, a plain fill of 512 bytes per
// position 82.  No other unit is near its limit (issue slots 58 %, special functions 44 %, tensor pipe 39 % busy).
// With the weights in tensor memory an MMA takes 36 clocks for 64 positions (as shared-memory operand 69 for 128), so that
// accumulators of 64 positions cost nothing, two of them (a, b) are in turn filled and read, and shared memory is a ring
// of four tiles.  A warp stages its 32 channels x 32 positions in shared memory and hands them to a TMA store, because a
// 32-byte store of 32 lanes to 32 channels' runs occupies the load-store unit for some 56 clocks.  Without the two
// (weights in shared memory, two tiles in flight, direct stores): 131 us.
//
// LayerNorm is folded into the weights (rows centred, per-row sum kept; gamma, beta and the biases included): the
// MMAs run on the raw tile as soon as it has landed, four statistics warps (one thread per position) compute mean
// and rstd of every position meanwhile, and the epilogue applies rstd[pos]·(D − mean[pos]·rowsum[ch]) + const[ch].
//
// Warp roles (704 threads): warps 0-15 epilogue - warps 0-7 finish the a, 8-15 the b channels; of each eight, two warps
// share a quarter of the channels, for 32 of the accumulator's 64 positions each -, warps 16-19 statistics, warp 20 TMA
// producer, warp 21 MMA issuer / TMEM owner.
#include "common.cuh"
#include "layout.h"

namespace b200ta {
namespace {

constexpr int kThreads = 704;
constexpr int kTileM = 128;                 // positions per tile
constexpr int kHalf = 64;                   // positions per accumulator
constexpr int kStages = 4;                  // tiles in flight (at first: the four weight blocks)
constexpr int kSmZ = 0;                     // kStages x 32 KiB
constexpr int kSmStats = kSmZ + kStages * 32768;  // 8 slots (tile i uses slot i & 7) x 4 x 128 floats
constexpr int kStatsSlot = 4 * 512;         // rstd, -mean*rstd, mask/2, mask/2 * b_scale
constexpr int kSmOut = kSmStats + 8 * kStatsSlot;  // 16 warps x 2 slabs x 2 KiB: 32 channels x 32 positions
constexpr int kSmBars = kSmOut + 16 * 2 * 2048;
enum Bar { W_FULL = 0, W_READY = 1, Z_FULL = 2, Z_EMPTY = Z_FULL + kStages, STATS_READY = Z_EMPTY + kStages, ACC_FULL = STATS_READY + 8,
           ACC_EMPTY = ACC_FULL + 2, NUM_BARS = ACC_EMPTY + 2 };
constexpr int kSmTotal = kSmBars + 256;
constexpr int kSmDynamic = kSmTotal + 1024;
// TMEM: the two accumulators (gate 64 | value 64 columns each), then the four weight blocks (64 columns each)
constexpr uint32_t kTmemW = 256;

struct ProjectParams {
  int B, R, S;
  int tiles_s, num_tiles;
  const float2* sc;  // {rowsum, const} per folded row
  float eps;
  const float* mask;  // may be NULL
  long long ms_b, ms_r, ms_s;
  const float* b_scale;  // per batch item, multiplies the b channels; may be NULL
  int* status;
};

__global__ void __launch_bounds__(kThreads, 1)
trimul_project_kernel(const __grid_constant__ CUtensorMap tm_z, const __grid_constant__ CUtensorMap tm_w,
                      const __grid_constant__ CUtensorMap tm_ab, const ProjectParams p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* gen = smem_raw + (base - smem_u32(smem_raw));
  const uint32_t bars = base + kSmBars;
  volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(gen + kSmBars + NUM_BARS * 8);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(gen + kSmBars + NUM_BARS * 8 + 8);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    abort_flag[0] = 0, abort_flag[1] = 0;
    mbar_init(bars + W_FULL * 8, 1);
    mbar_init(bars + W_READY * 8, 16);
    for (int i = 0; i < kStages; ++i) {
      mbar_init(bars + (Z_FULL + i) * 8, 1);
      mbar_init(bars + (Z_EMPTY + i) * 8, 5);  // the MMA commit + the four statistics warps have read the tile
    }
    for (int i = 0; i < 8; ++i) mbar_init(bars + (STATS_READY + i) * 8, 4);
    for (int i = 0; i < 2; ++i) {
      mbar_init(bars + (ACC_FULL + i) * 8, 1);
      mbar_init(bars + (ACC_EMPTY + i) * 8, 8);
    }
    fence_mbar_init();
  }
  if (warp == 21) {
    tmem_alloc(smem_u32(const_cast<uint32_t*>(tmem_slot)), 512);
    pdl_trigger();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const int my_tiles = (p.num_tiles - 1 - int(blockIdx.x)) / int(gridDim.x) + 1;

  if (warp == 20) {
    // ------------------------------------------------------------------ TMA producer
    if (lane == 0) {
      tma_prefetch_desc(&tm_z);
      // the weights pass through the ring on their way to tensor memory: block k in stage k
      mbar_expect_tx(bars + W_FULL * 8, kStages * 32768);
      for (int k = 0; k < kStages; ++k)
        for (int kh = 0; kh < 2; ++kh)
          tma_load_2d(base + kSmZ + k * 32768 + kh * 16384, &tm_w, bars + W_FULL * 8, kh * 64, k * 128);
      mbar_wait(bars + W_READY * 8, 0, abort_flag);
      pdl_wait();
      int issued = 0;
      for (int i = 0, stage = 0, phase = 1; i < my_tiles; ++i) {
        const int tile = blockIdx.x + i * gridDim.x;
        const int st = tile % p.tiles_s, br = tile / p.tiles_s;
        const int r = br % p.R, b = br / p.R;
        if (!mbar_wait(bars + (Z_EMPTY + stage) * 8, phase, abort_flag)) break;
        const uint32_t full = bars + (Z_FULL + stage) * 8;
        mbar_expect_tx(full, 32768);
        tma_load_4d(base + kSmZ + stage * 32768, &tm_z, full, 0, st * kTileM, r, b);
        tma_load_4d(base + kSmZ + stage * 32768 + 16384, &tm_z, full, 64, st * kTileM, r, b);
        ++issued;
        if (++stage == kStages) stage = 0, phase ^= 1;
      }
      // If the loop was abandoned, give copies still in flight a bounded chance to land.
      if (*abort_flag)
        for (int j = issued > kStages ? issued - kStages : 0; j < issued; ++j)
          mbar_wait(bars + (Z_FULL + j % kStages) * 8, (j / kStages) & 1, abort_flag + 1);
    }
  } else if (warp == 21) {
    // ------------------------------------------------------------------ MMA issuer (whole warp, one lane issues)
    constexpr uint32_t idesc = make_idesc_bf16(128, kHalf);
    const uint32_t tb = __shfl_sync(0xffffffffu, tmem_base, 0);
    bool ok = mbar_wait_warp(bars + W_READY * 8, 0, abort_flag);
    uint32_t uses = 0;  // accumulators filled, of each kind
    for (int i = 0, stage = 0, phase = 0; ok && i < my_tiles; ++i) {
      ok = mbar_wait_warp(bars + (Z_FULL + stage) * 8, phase, abort_flag);
      const uint64_t dz = smem_desc<16, 1024, kLayoutSw128>(base + kSmZ + stage * 32768);
      for (int half = 0; ok && half < 2; ++half, ++uses) {
#pragma unroll
        for (int g = 0; g < 2; ++g) {  // a channels, b channels
          if (!ok) break;
          ok = mbar_wait_warp(bars + (ACC_EMPTY + g) * 8, (uses & 1) ^ 1, abort_flag);
          if (!ok) break;
          tc_fence_after();
#pragma unroll
          for (int acc = 0; acc < 2; ++acc) {  // gate rows, then value rows
            const uint32_t d = tb + g * 128 + acc * 64, w = tb + kTmemW + (g * 2 + acc) * 64;
#pragma unroll
            for (int k = 0; k < 8; ++k)
              umma_ts_warp(d, w + k * 8, dz + (half * (8192 >> 4) + (k >> 2) * (16384 >> 4) + (k & 3) * 2), idesc,
                           k > 0 ? 1u : 0u);
          }
          umma_commit_warp(bars + (ACC_FULL + g) * 8);
        }
      }
      if (!ok) break;
      umma_commit_warp(bars + (Z_EMPTY + stage) * 8);
      if (++stage == kStages) stage = 0, phase ^= 1;
    }
  } else if (warp >= 16) {
    // ------------------------------------------------------------------ statistics: one thread per position
    pdl_wait();
    const int m = (warp - 16) * 32 + lane;
    for (int i = 0, stage = 0, phase = 0; i < my_tiles; ++i) {
      const int tile = blockIdx.x + i * gridDim.x;
      const int st = tile % p.tiles_s, br = tile / p.tiles_s;
      const int r = br % p.R, b = br / p.R;
      const int s = st * kTileM + m;
      float mval = 0.f;
      if (s < p.S) mval = p.mask ? __ldg(p.mask + b * p.ms_b + r * p.ms_r + (long long)s * p.ms_s) : 1.f;
      const float scale = p.b_scale ? __ldg(p.b_scale + b) : 1.f;
      if (!mbar_wait(bars + (Z_FULL + stage) * 8, phase, abort_flag)) break;
      const float2 v = row_stats_128(base + kSmZ + stage * 32768, m, p.eps);
      // Eight slots: a slot is rewritten eight tiles later, after the MMAs of the tile two later, whose accumulators the
      // epilogue has handed back only after it was done with this tile.
      float* slot = reinterpret_cast<float*>(gen + kSmStats + (i & 7) * kStatsSlot);
      slot[m] = v.x;
      slot[128 + m] = v.y;
      slot[256 + m] = 0.5f * mval;  // sigmoid(g) * v * mask = tanh(g/2) * h + h with h = v * mask / 2
      slot[384 + m] = 0.5f * mval * scale;
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(bars + (STATS_READY + (i & 7)) * 8);
        mbar_arrive(bars + (Z_EMPTY + stage) * 8);  // done reading the tile
      }
      if (++stage == kStages) stage = 0, phase ^= 1;
    }
  } else {
    // ------------------------------------------------------------------ epilogue warps: one thread per channel
    const int g = warp >> 3;           // 0: a channels, 1: b channels
    const int part = (warp >> 2) & 1;  // which 32 positions of the accumulator
    const int ch = (warp & 3) * 32 + lane;  // channel inside the 128 == TMEM lane
    const uint32_t lane_taddr = tmem_base + (uint32_t((warp & 3) * 32) << 16);
    {
      // this warp's 32 rows of weight block 2 g + part, as bf16 pairs
      mbar_wait_warp(bars + W_FULL * 8, 0, abort_flag);
      const uint32_t src = base + kSmZ + (g * 2 + part) * 32768;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        uint32_t v[16];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const uint4 x = lds128(src + (k >> 1) * 16384 + sw128_offset(ch, (k & 1) * 4 + j));
          v[j * 4] = x.x, v[j * 4 + 1] = x.y, v[j * 4 + 2] = x.z, v[j * 4 + 3] = x.w;
        }
        tmem_st16(lane_taddr + kTmemW + (g * 2 + part) * 64 + k * 16, v);
      }
      tmem_st_wait();
      tc_fence_before();
      __syncwarp();
      mbar_arrive_warp(bars + W_READY * 8);
    }
    const uint32_t acc = lane_taddr + g * 128 + part * 32;  // the value columns lie 64 further
    const float2 kg = p.sc[g * 256 + ch], kp = p.sc[g * 256 + 128 + ch];  // {rowsum, const} of the gate / value row
    const uint64_t cg2 = pack_f32x2(kg.y, kg.y), cp2 = pack_f32x2(kp.y, kp.y);
    const uint64_t rg2 = pack_f32x2(kg.x, kg.x), rp2 = pack_f32x2(kp.x, kp.x);
    pdl_wait();
    bool ok = true;
    uint32_t uses = 0;
    for (int i = 0; ok && i < my_tiles; ++i) {
      const int tile = blockIdx.x + i * gridDim.x;
      const int st = tile % p.tiles_s, br = tile / p.tiles_s;
      const int r = br % p.R, b = br / p.R;
      const uint32_t stats = base + kSmStats + (i & 7) * kStatsSlot;
      for (int half = 0; half < 2; ++half, ++uses) {
        ok = mbar_wait2_warp(bars + (STATS_READY + (i & 7)) * 8, (i >> 3) & 1, bars + (ACC_FULL + g) * 8, uses & 1, abort_flag);
        if (!ok) break;
        tc_fence_after();
        const int pos = half * kHalf + part * 32;
        const uint32_t slab = base + kSmOut + (warp * 2 + (uses & 1)) * 2048;
        if (lane == 0) tma_store_wait_read<1>();  // the store before the previous one has read this slab
        __syncwarp();
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          uint32_t gg[16], vv[16];
          tmem_ld16(acc + q * 16, gg);
          tmem_ld16(acc + 64 + q * 16, vv);
          tmem_ld_wait();
          if (q == 1) {  // the accumulator is in registers: the next MMAs may have it
            tc_fence_before();
            __syncwarp();
            mbar_arrive_warp(bars + (ACC_EMPTY + g) * 8);
          }
          uint32_t packed[8];
#pragma unroll
          for (int e = 0; e < 4; ++e) {  // four positions, as two packed pairs
            const uint32_t at = stats + (pos + q * 16 + e * 4) * 4;
            uint64_t rs[2], nm[2], mh[2];
            lds_f32x2(at, rs[0], rs[1]);
            lds_f32x2(at + 512, nm[0], nm[1]);
            lds_f32x2(at + 1024 + g * 512, mh[0], mh[1]);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              const int j = e * 4 + h * 2;
              const uint64_t rs2 = rs[h], nm2 = nm[h];
              float a0, a1;
              unpack_f32x2(fma_f32x2(rs2, pack_f32x2(__uint_as_float(gg[j]), __uint_as_float(gg[j + 1])),
                                     fma_f32x2(nm2, rg2, cg2)), a0, a1);
              const uint64_t val2 = fma_f32x2(rs2, pack_f32x2(__uint_as_float(vv[j]), __uint_as_float(vv[j + 1])),
                                              fma_f32x2(nm2, rp2, cp2));
              const uint64_t h2 = mul_f32x2(val2, mh[h]);
              float o0, o1;  // gate rows are pre-halved
              unpack_f32x2(fma_f32x2(pack_f32x2(tanh_approx(a0), tanh_approx(a1)), h2, h2), o0, o1);
              packed[e * 2 + h] = pack_bf16x2(o0, o1);
            }
          }
#pragma unroll
          for (int c = 0; c < 2; ++c)
            sts128(slab + sw64_offset(lane, q * 2 + c), make_uint4(packed[c * 4], packed[c * 4 + 1], packed[c * 4 + 2], packed[c * 4 + 3]));
        }
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
          // (positions past the row pitch are not written; between the token count and the pitch they are zero)
          tma_store_3d(&tm_ab, slab, st * kTileM + pos, r, (b * 2 + g) * kTriHidden + (warp & 3) * 32);
          tma_store_commit();
        }
      }
    }
    if (lane == 0) tma_store_wait_all();
  }

  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (warp == 21) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
  if (threadIdx.x == 0 && *abort_flag) *p.status = B200TA_ERR_DEVICE_WAIT;
}

}  // namespace
}  // namespace b200ta

extern "C" {

int b200ta_trimul_project(const void* z, int64_t zs_b, int64_t zs_r, int64_t zs_s, const float* mask, int64_t ms_b,
                          int64_t ms_r, int64_t ms_s, const float* b_scale, const void* packed, float eps, void* ab,
                          int64_t pitch, int B, int R, int S, void* stream) {
  using namespace b200ta;
  B200TA_REQUIRE(z && packed && ab, "trimul_project: NULL pointer");
  B200TA_REQUIRE(B > 0 && R > 0 && S > 0, "trimul_project: bad sizes B=%d R=%d S=%d", B, R, S);
  B200TA_REQUIRE(pitch >= S && pitch % 16 == 0, "trimul_project: pitch=%lld must be a multiple of 16 and >= S=%d",
                 (long long)pitch, S);
  B200TA_REQUIRE(zs_b % 8 == 0 && zs_r % 8 == 0 && zs_s % 8 == 0 && zs_b >= 0 && zs_r >= 0 && zs_s >= 0,
                 "trimul_project: z element strides must be non-negative multiples of 8 (16 bytes)");
  B200TA_REQUIRE((reinterpret_cast<uintptr_t>(packed) & 255u) == 0, "trimul_project: packed must be 256-byte aligned");
  B200TA_REQUIRE((reinterpret_cast<uintptr_t>(ab) & 31u) == 0, "trimul_project: ab must be 32-byte aligned");
  B200TA_REQUIRE(int64_t(B) * R < (int64_t(1) << 31), "trimul_project: B*R too large");
  DeviceState* st = nullptr;
  int rc = get_device_state(&st);
  if (rc != B200TA_OK) return rc;

  CUtensorMap tm_z, tm_w, tm_ab;
  {
    // (c, s, r, b); a size-1 dimension may carry any stride: give it a valid one
    auto fix = [](int64_t stride, int extent) -> uint64_t { return extent == 1 ? 256u : uint64_t(stride) * 2u; };
    uint64_t dims[4] = {uint64_t(kC), uint64_t(S), uint64_t(R), uint64_t(B)};
    uint64_t strides[3] = {fix(zs_s, S), fix(zs_r, R), fix(zs_b, B)};
    uint32_t box[4] = {64, kTileM, 1, 1};
    rc = encode_tensor_map(&tm_z, z, 2, 4, dims, strides, box, SWZ_128, "trimul_project z");
    if (rc != B200TA_OK) return rc;
  }
  const char* pk = static_cast<const char*>(packed);
  {
    uint64_t dims[2] = {uint64_t(kC), uint64_t(kTriRows)};
    uint64_t strides[1] = {uint64_t(kC) * 2};
    uint32_t box[2] = {64, 128};
    rc = encode_tensor_map(&tm_w, pk + kTriWOff, 2, 2, dims, strides, box, SWZ_128, "trimul_project weights");
    if (rc != B200TA_OK) return rc;
  }
  {
    // (position, row, plane): a warp's slab of 32 channels
    uint64_t dims[3] = {uint64_t(pitch), uint64_t(R), uint64_t(B) * 2 * kTriHidden};
    uint64_t strides[2] = {uint64_t(pitch) * 2, uint64_t(pitch) * R * 2};
    uint32_t box[3] = {32, 1, 32};
    rc = encode_tensor_map(&tm_ab, ab, 2, 3, dims, strides, box, SWZ_64, "trimul_project ab");
    if (rc != B200TA_OK) return rc;
  }
  ProjectParams p{};
  p.B = B, p.R = R, p.S = S;
  p.tiles_s = (S + kTileM - 1) / kTileM;
  p.num_tiles = B * R * p.tiles_s;
  p.sc = reinterpret_cast<const float2*>(pk + kTriScOff);
  p.eps = eps;
  p.mask = mask;
  p.ms_b = ms_b, p.ms_r = ms_r, p.ms_s = ms_s;
  p.b_scale = b_scale;
  p.status = st->status_dev;

  const int grid = p.num_tiles < st->num_sms ? p.num_tiles : st->num_sms;
  return launch_kernel(st, kKernelProject, trimul_project_kernel, dim3(grid), kThreads, kSmDynamic, stream, tm_z, tm_w, tm_ab, p);
}

}  // extern "C"
