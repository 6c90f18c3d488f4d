// Triangle-multiplication output stage for sm_100a:
//   out[b,i,j,:] = sigmoid(LN_in(z[b,i,j,:])·W_goᵀ + b_go) ⊙ (LN_out(x[b,:,i,j])·W_poᵀ + b_po)   [+ z]   [* mask]
// x is the contraction result, channel-major x[b][d][i][j] (bf16).  One tile = 128 consecutive positions j of one
// pair row (b, i); per tile two tcgen05 GEMMs share one accumulator slot (256 TMEM columns, double-buffered):
//   D_g[pos, ch] = z[pos, :] · W_go'[ch, :]ᵀ    A = the raw z tile (K-major)
//   D_p[pos, ch] = x[:, pos]ᵀ · W_po'[ch, :]ᵀ   A = the x tile as it lies in memory, [d][pos] = MN-major
// Both LayerNorms are folded into the weights (rows centred, per-row sum kept): the epilogue, one thread per
// position, applies rstd·(D − mean·rowsum) + const with the statistics the statistics warps computed from the two
// tiles while the MMAs ran - neither tile is rewritten and the MMAs wait for nothing but the loads.
//
// The residual is read from the z tile in shared memory, and the result leaves through a slab per warp (32 positions of
// 64 bytes) and TMA: with a thread per position, 32-byte global accesses of a warp go to 32 rows and occupy the load-store
// unit for some 56 clocks each, which bounded the kernel (148 us at 768 tokens, 3.1 TB/s of the 768 bytes per position).
// What bounds it now is the time from a tile's load to the reuse of its stage, with room for two (the weights take 64
// KiB): some 3600 clocks of latency, 1900 of statistics, then the epilogue copies the residual and hands the stage back.
//
// Warp roles (576 threads): warps 0-7 epilogue (thread = position; the two warpgroups take alternate groups of 32
// output channels), warps 8-11 statistics of the z rows (one thread per position), warps 12-15 of the x columns (a thread
// takes two neighbouring positions over half of the channels), warp 16 TMA producer, warp 17 MMA issuer / TMEM owner.
#include "common.cuh"
#include "layout.h"

namespace b200ta {
namespace {

constexpr int kThreads = 576;
constexpr int kTileM = 128;
constexpr int kSmW = 0;                      // W_go' and W_po': 2 matrices x 2 K-halves x 128 rows x 128 B
constexpr int kSmZ = kSmW + 65536;           // 2 stages x 32 KiB
constexpr int kSmX = kSmZ + 2 * 32768;       // 2 stages x 32 KiB
constexpr int kSmConst = kSmX + 2 * 32768;   // per channel pair: float4 [64] {c_gate0, c_gate1, rowsum_g0, rowsum_g1}, float4 [64] {c_p0, c_p1, rowsum_p0, rowsum_p1}
constexpr int kSmStats = kSmConst + 2048;    // 4 slots (tile i uses slot i & 3) x { float4 [128] {rstd_o, -mean_o*rstd_o, rstd_i, -mean_i*rstd_i}, float [128] mask }
constexpr int kStatsSlot = 2048 + 512;
constexpr int kSmOut = kSmStats + 4 * kStatsSlot;  // 8 warps x 2 KiB: 32 positions x 64 bytes
constexpr int kSmBars = kSmOut + 8 * 2048;
enum Bar { W_FULL = 0, IN_FULL = 1, READY = 3, IN_EMPTY = 7, ACC_FULL = 9, ACC_EMPTY = 11, NUM_BARS = 13 };
constexpr int kSmTotal = kSmBars + 256;
constexpr int kSmDynamic = kSmTotal + 1024;

struct OutputParams {
  int B, N;  // pair tensor [B, N, N, 128]
  int tiles_j, num_tiles;
  const float2* sc;  // folded {rowsum, const} of the output gate rows, then of the output projection rows
  float eps;
  int add_residual;
  const float* mask;  // [B, N, N] via strides; NULL = no output mask
  long long ms_b, ms_i, ms_j;
  int* status;
};

__device__ __forceinline__ uint32_t lds32(uint32_t addr) {
  uint32_t v;
  asm volatile("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(addr));
  return v;
}

template <bool kF32>
__global__ void __launch_bounds__(kThreads, 1)
trimul_output_kernel(const __grid_constant__ CUtensorMap tm_z, const __grid_constant__ CUtensorMap tm_x,
                     const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_out,
                     const OutputParams p) {
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
    // statistics written (the four statistics warps): one barrier per statistics slot, because the statistics of
    // tile t + 2 may be complete before the epilogue of tile t has looked at its barrier
    for (int i = 0; i < 4; ++i) mbar_init(bars + (READY + i) * 8, 8);
    for (int i = 0; i < 2; ++i) {
      mbar_init(bars + (IN_FULL + i) * 8, 1);
      mbar_init(bars + (IN_EMPTY + i) * 8, 1 + 8 + 8);  // MMA commit, statistics, epilogue (residual) have read the tiles
      mbar_init(bars + (ACC_FULL + i) * 8, 1);
      mbar_init(bars + (ACC_EMPTY + i) * 8, 8);
    }
    fence_mbar_init();
  }
  if (warp == 17) {
    tmem_alloc(smem_u32(const_cast<uint32_t*>(tmem_slot)), 512);
    pdl_trigger();
  }
  // per-channel constants of the epilogue
  if (threadIdx.x < kC / 2) {
    const int c = 2 * threadIdx.x;
    const float2 g0 = p.sc[c], g1 = p.sc[c + 1], q0 = p.sc[kC + c], q1 = p.sc[kC + c + 1];
    reinterpret_cast<float4*>(gen + kSmConst)[threadIdx.x] = make_float4(g0.y, g1.y, g0.x, g1.x);
    reinterpret_cast<float4*>(gen + kSmConst + 1024)[threadIdx.x] = make_float4(q0.y, q1.y, q0.x, q1.x);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const int my_tiles = (p.num_tiles - 1 - int(blockIdx.x)) / int(gridDim.x) + 1;

  if (warp == 16) {
    // ------------------------------------------------------------------ TMA producer
    if (lane == 0) {
      tma_prefetch_desc(&tm_z);
      tma_prefetch_desc(&tm_x);
      tma_prefetch_desc(&tm_w);
      mbar_expect_tx(bars + W_FULL * 8, 65536);
      for (int mat = 0; mat < 2; ++mat)
        for (int kh = 0; kh < 2; ++kh)
          tma_load_2d(base + kSmW + mat * 32768 + kh * 16384, &tm_w, bars + W_FULL * 8, kh * 64, kTriInRows + mat * kC);
      pdl_wait();
      int issued = 0;
      for (int it = 0; it < my_tiles; ++it) {
        const int tile = blockIdx.x + it * gridDim.x;
        const int jt = tile % p.tiles_j, bi = tile / p.tiles_j;
        const int i = bi % p.N, b = bi / p.N;
        const int stage = it & 1;
        if (!mbar_wait(bars + (IN_EMPTY + stage) * 8, ((it >> 1) & 1) ^ 1, abort_flag)) break;
        const uint32_t full = bars + (IN_FULL + stage) * 8;
        mbar_expect_tx(full, 65536);
        tma_load_4d(base + kSmZ + stage * 32768, &tm_z, full, 0, jt * kTileM, i, b);
        tma_load_4d(base + kSmZ + stage * 32768 + 16384, &tm_z, full, 64, jt * kTileM, i, b);
        tma_load_3d(base + kSmX + stage * 32768, &tm_x, full, jt * kTileM, i, b * kTriHidden);
        tma_load_3d(base + kSmX + stage * 32768 + 16384, &tm_x, full, jt * kTileM + 64, i, b * kTriHidden);
        ++issued;
      }
      if (*abort_flag && issued > 0) {
        const int last = issued - 1;
        mbar_wait(bars + (IN_FULL + (last & 1)) * 8, (last >> 1) & 1, abort_flag + 1);
      }
    }
  } else if (warp == 17) {
    // ------------------------------------------------------------------ MMA issuer (whole warp, one lane issues)
    constexpr uint32_t idesc_g = make_idesc_bf16(kTileM, kC);               // both operands K-major
    constexpr uint32_t idesc_p = make_idesc_bf16(kTileM, kC, true, false);  // A (the x tile) MN-major
    const uint32_t tb = __shfl_sync(0xffffffffu, tmem_base, 0);
    bool ok = mbar_wait_warp(bars + W_FULL * 8, 0, abort_flag);
    for (int it = 0; ok && it < my_tiles; ++it) {
      const int stage = it & 1, slot = it & 1;
      ok = mbar_wait2_warp(bars + (IN_FULL + stage) * 8, (it >> 1) & 1, bars + (ACC_EMPTY + slot) * 8, ((it >> 1) & 1) ^ 1,
                           abort_flag);
      if (!ok) break;
      tc_fence_after();
      const uint32_t d = tb + slot * 256;
      const uint64_t dz = smem_desc<16, 1024, kLayoutSw128>(base + kSmZ + stage * 32768);
      const uint64_t dwg = smem_desc<16, 1024, kLayoutSw128>(base + kSmW);
      const uint64_t dwp = smem_desc<16, 1024, kLayoutSw128>(base + kSmW + 32768);
      // x tile: [128 d][64 j] blocks of 128-byte rows, the two 64-position blocks 16 KiB apart; as A[pos][d] this
      // is MN-major, a K step of 16 channels is 16 rows = 2 KiB
      const uint64_t dx = smem_desc<16384, 1024, kLayoutSw128>(base + kSmX + stage * 32768);
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const uint32_t koff = (k >> 2) * (16384 >> 4) + (k & 3) * 2;
        umma_ss_warp(d, dz + koff, dwg + koff, idesc_g, k > 0 ? 1u : 0u);
      }
#pragma unroll
      for (int k = 0; k < 8; ++k)
        umma_ss_warp(d + 128, dx + k * 128, dwp + ((k >> 2) * (16384 >> 4) + (k & 3) * 2), idesc_p, k > 0 ? 1u : 0u);
      umma_commit_warp(bars + (ACC_FULL + slot) * 8);
      umma_commit_warp(bars + (IN_EMPTY + stage) * 8);
    }
  } else if (warp >= 8 && warp < 12) {
    // ------------------------------------------------------------------ statistics of the z rows
    pdl_wait();
    const int t = (warp - 8) * 32 + lane;
    for (int it = 0; it < my_tiles; ++it) {
      const int tile = blockIdx.x + it * gridDim.x;
      const int jt = tile % p.tiles_j, bi = tile / p.tiles_j;
      const int i = bi % p.N, b = bi / p.N;
      const int stage = it & 1;
      const int j = jt * kTileM + t;
      float mval = 1.f;
      if (p.mask != nullptr) mval = j < p.N ? __ldg(p.mask + b * p.ms_b + i * p.ms_i + (long long)j * p.ms_j) : 0.f;
      if (!mbar_wait(bars + (IN_FULL + stage) * 8, (it >> 1) & 1, abort_flag)) break;
      const float2 v = row_stats_128(base + kSmZ + stage * 32768, t, p.eps);
      // Statistics and mask go to one of four slots: the epilogue of a tile may still read its slot while the
      // next two tiles' statistics are written.
      uint8_t* slot = gen + kSmStats + (it & 3) * kStatsSlot;
      reinterpret_cast<float2*>(slot)[2 * t + 1] = v;
      reinterpret_cast<float*>(slot + 2048)[t] = mval;
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(bars + (READY + (it & 3)) * 8);
        mbar_arrive(bars + (IN_EMPTY + stage) * 8);  // done reading the tile
      }
    }
  } else if (warp >= 12 && warp < 16) {
    // ------------------------------------------------------------------ statistics of the x columns
    pdl_wait();
    for (int it = 0; it < my_tiles; ++it) {
      const int stage = it & 1;
      if (!mbar_wait(bars + (IN_FULL + stage) * 8, (it >> 1) & 1, abort_flag)) break;
      // ---- x columns: this thread takes positions 2q, 2q+1 over channels [64 h, 64 h + 64), in one pass of packed sums
      // shifted by the first channel (as row_stats_128)
      {
        const int q = (warp - 12) * 16 + (lane & 15), h = lane >> 4;
        const int jj = (2 * q) & 63;
        const uint32_t x0 = base + kSmX + stage * 32768 + ((2 * q) >> 6) * 16384 + h * 8192 + (jj & 7) * 2;
        const uint32_t chunk = uint32_t(jj >> 3);
        const uint32_t first = lds32(x0 + (chunk << 4));
        const float k0 = bf16_lo(first), k1 = bf16_hi(first);
        const uint64_t nk2 = pack_f32x2(-k0, -k1);
        uint64_t sa[2] = {0ull, 0ull}, sq[2] = {0ull, 0ull};
#pragma unroll 16
        for (int d = 0; d < 64; ++d) {
          const uint32_t w = lds32(x0 + d * 128 + ((chunk ^ (d & 7)) << 4));
          const uint64_t v = add_f32x2(pack_f32x2(bf16_lo(w), bf16_hi(w)), nk2);
          sa[d & 1] = add_f32x2(sa[d & 1], v);
          sq[d & 1] = fma_f32x2(v, v, sq[d & 1]);
        }
        float s0, s1, q0, q1;
        unpack_f32x2(add_f32x2(sa[0], sa[1]), s0, s1);
        unpack_f32x2(add_f32x2(sq[0], sq[1]), q0, q1);
        // Mean and sum of squared deviations of the 64 channels, combined with those of the other half of the channels
        // in lane ^ 16; lanes 0-15 write position 2q, lanes 16-31 position 2q + 1.
        const float m0 = s0 * (1.f / 64) + k0, m1 = s1 * (1.f / 64) + k1;
        const float d0 = fmaxf(q0 - s0 * s0 * (1.f / 64), 0.f), d1 = fmaxf(q1 - s1 * s1 * (1.f / 64), 0.f);
        const float mo = __shfl_xor_sync(0xffffffffu, h ? m0 : m1, 16), qo = __shfl_xor_sync(0xffffffffu, h ? d0 : d1, 16);
        const float mm = h ? m1 : m0, qm = h ? d1 : d0;
        const float mean = 0.5f * (mm + mo);
        const float var = (qm + qo + (mm - mo) * (mm - mo) * 32.f) * (1.f / kTriHidden);
        const float rstd = rsqrtf(var + p.eps);
        reinterpret_cast<float2*>(gen + kSmStats + (it & 3) * kStatsSlot)[2 * (2 * q + h)] = make_float2(rstd, -mean * rstd);
      }
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(bars + (READY + (it & 3)) * 8);
        mbar_arrive(bars + (IN_EMPTY + stage) * 8);  // done reading the tile
      }
    }
  } else if (warp < 8) {
    // ------------------------------------------------------------------ epilogue warps: one thread per position
    pdl_wait();
    const int e = warp >> 2;
    const int m = (warp & 3) * 32 + lane;
    const uint32_t lane_taddr = tmem_base + (uint32_t((warp & 3) * 32) << 16);
    const float4* c4 = reinterpret_cast<const float4*>(gen + kSmConst);         // per channel pair
    const float4* c4b = reinterpret_cast<const float4*>(gen + kSmConst + 1024);  // per channel pair
    const uint32_t slab = base + kSmOut + warp * 2048;
    bool ok = true;
    for (int it = 0; ok && it < my_tiles; ++it) {
      const int tile = blockIdx.x + it * gridDim.x;
      const int jt = tile % p.tiles_j, bi = tile / p.tiles_j;
      const int i = bi % p.N, b = bi / p.N;
      const int j0 = jt * kTileM + (warp & 3) * 32;  // the warp's first position
      const int slot = it & 1;
      // (IN_FULL is complete, or there would be no statistics: it makes the copies' writes visible to this thread)
      ok = mbar_wait2_warp(bars + (READY + (it & 3)) * 8, (it >> 2) & 1, bars + (ACC_FULL + slot) * 8, (it >> 1) & 1, abort_flag) &&
           mbar_wait_warp(bars + (IN_FULL + slot) * 8, (it >> 1) & 1, abort_flag);
      if (!ok) break;
      tc_fence_after();
      const uint32_t row = base + kSmZ + slot * 32768 + sw128_offset(m, 0);  // chunk c of a row lies at chunk c ^ (row % 8)
      uint32_t res[2][16];  // the residual of this thread's channel groups e and e + 2
#pragma unroll
      for (int gi = 0; gi < 2; ++gi)
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const uint4 x = lds128((row + gi * 16384) ^ ((e * 4 + c) << 4));
          res[gi][c * 4 + 0] = x.x, res[gi][c * 4 + 1] = x.y, res[gi][c * 4 + 2] = x.z, res[gi][c * 4 + 3] = x.w;
        }
      mbar_arrive_warp_after_reads(bars + (IN_EMPTY + slot) * 8);
      const uint8_t* stats = gen + kSmStats + (it & 3) * kStatsSlot;
      const float4 stv = reinterpret_cast<const float4*>(stats)[m];
      const float mval = reinterpret_cast<const float*>(stats + 2048)[m];
      const uint64_t rstd2 = pack_f32x2(stv.x, stv.x), nmr2 = pack_f32x2(stv.y, stv.y), mval2 = pack_f32x2(mval, mval);
      const uint64_t rstdg2 = pack_f32x2(stv.z, stv.z), nmrg2 = pack_f32x2(stv.w, stv.w);
      const uint64_t half2 = pack_f32x2(0.5f, 0.5f);
      // four chunks of 16 output channels: [32 g + 16 h, +16) for this warpgroup's groups g = e, e + 2
      const uint32_t acc = lane_taddr + slot * 256;
#pragma unroll
      for (int ck = 0; ck < 4; ++ck) {
        const int g = e + 2 * (ck >> 1), h = ck & 1;
        const int ch0 = g * 32 + h * 16;
        uint32_t xg[16], xp[16];
        tmem_ld16(acc + ch0, xg);
        tmem_ld16(acc + 128 + ch0, xp);
        tmem_ld_wait();
        // a slab holds 32 bf16 or 16 float channels of the warp's 32 positions
        if (kF32 || h == 0) {
          if (lane == 0) tma_store_wait_read<0>();
          __syncwarp();
        }
        uint32_t packed[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          // two channels at a time, packed fp32x2 math; constants per channel pair: {const0, const1, rowsum0,
          // rowsum1} of the gate rows and of the projection rows
          const float4 ka = c4[(ch0 >> 1) + c];
          const float4 kb = c4b[(ch0 >> 1) + c];
          float a0, a1;
          unpack_f32x2(fma_f32x2(rstdg2, pack_f32x2(__uint_as_float(xg[2 * c]), __uint_as_float(xg[2 * c + 1])),
                                 fma_f32x2(nmrg2, pack_f32x2(ka.z, ka.w), pack_f32x2(ka.x, ka.y))),
                       a0, a1);
          // gate rows are pre-halved: sigmoid(x) = 0.5 * tanh(x / 2) + 0.5
          const uint64_t s2 = fma_f32x2(pack_f32x2(tanh_approx(a0), tanh_approx(a1)), half2, half2);
          const uint64_t v2 = fma_f32x2(rstd2, pack_f32x2(__uint_as_float(xp[2 * c]), __uint_as_float(xp[2 * c + 1])),
                                        fma_f32x2(nmr2, pack_f32x2(kb.z, kb.w), pack_f32x2(kb.x, kb.y)));
          const uint32_t r = p.add_residual ? res[ck >> 1][h * 8 + c] : 0u;
          float o0, o1;
          unpack_f32x2(mul_f32x2(fma_f32x2(s2, v2, pack_f32x2(bf16_lo(r), bf16_hi(r))), mval2), o0, o1);
          if (kF32) {
            packed[(2 * c) & 7] = __float_as_uint(o0), packed[(2 * c + 1) & 7] = __float_as_uint(o1);
            if ((c & 3) == 3) {
#pragma unroll
              for (int q = 0; q < 2; ++q)
                sts128(slab + sw64_offset(lane, (c - 3) / 2 + q), make_uint4(packed[q * 4], packed[q * 4 + 1], packed[q * 4 + 2], packed[q * 4 + 3]));
            }
          } else {
            packed[c] = pack_bf16x2(o0, o1);
          }
        }
        if (!kF32) {
#pragma unroll
          for (int c = 0; c < 2; ++c)
            sts128(slab + sw64_offset(lane, h * 2 + c), make_uint4(packed[c * 4], packed[c * 4 + 1], packed[c * 4 + 2], packed[c * 4 + 3]));
        }
        if (kF32 || h == 1) {
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0 && j0 < p.N) {
            tma_store_4d(&tm_out, slab, kF32 ? ch0 : g * 32, j0, i, b);
            tma_store_commit();
          }
        }
      }
      tc_fence_before();
      __syncwarp();
      mbar_arrive_warp(bars + (ACC_EMPTY + slot) * 8);
    }
    if (lane == 0) tma_store_wait_all();
  }

  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (warp == 17) {
    tc_fence_after();
    tmem_dealloc(tmem_base, 512);
  }
  if (threadIdx.x == 0 && *abort_flag) *p.status = B200TA_ERR_DEVICE_WAIT;
}

}  // namespace
}  // namespace b200ta

namespace b200ta {
namespace {

template <bool kF32>
int launch_output(const void* z, int64_t zs_b, int64_t zs_i, int64_t zs_j, const void* x, int64_t pitch, const float* mask,
                  int64_t ms_b, int64_t ms_i, int64_t ms_j, const void* packed, float eps, int add_residual, void* out,
                  int64_t os_b, int64_t os_i, int64_t os_j, int B, int N, void* stream) {
  B200TA_REQUIRE(z && x && packed && out, "trimul_output: NULL pointer");
  B200TA_REQUIRE(B > 0 && N > 0, "trimul_output: bad sizes B=%d N=%d", B, N);
  B200TA_REQUIRE(pitch >= N && pitch % 16 == 0, "trimul_output: pitch=%lld must be a multiple of 16 and >= N=%d",
                 (long long)pitch, N);
  for (int64_t s : {zs_b, zs_i, zs_j, os_b, os_i, os_j})
    B200TA_REQUIRE(s >= 0 && s % 16 == 0, "trimul_output: z/out element strides must be non-negative multiples of 16");
  B200TA_REQUIRE((reinterpret_cast<uintptr_t>(packed) & 255u) == 0, "trimul_output: packed must be 256-byte aligned");
  B200TA_REQUIRE((reinterpret_cast<uintptr_t>(z) & 31u) == 0 && (reinterpret_cast<uintptr_t>(out) & 31u) == 0 &&
                     (reinterpret_cast<uintptr_t>(x) & 31u) == 0,
                 "trimul_output: z, x and out must be 32-byte aligned");
  B200TA_REQUIRE(int64_t(B) * N < (int64_t(1) << 31), "trimul_output: B*N too large");
  DeviceState* st = nullptr;
  int rc = get_device_state(&st);
  if (rc != B200TA_OK) return rc;

  CUtensorMap tm_z, tm_x, tm_w, tm_out;
  {
    auto fix = [](int64_t stride, int extent) -> uint64_t { return extent == 1 ? 256u : uint64_t(stride) * 2u; };
    uint64_t dims[4] = {uint64_t(kC), uint64_t(N), uint64_t(N), uint64_t(B)};
    uint64_t strides[3] = {fix(zs_j, N), fix(zs_i, N), fix(zs_b, B)};
    uint32_t box[4] = {64, kTileM, 1, 1};
    rc = encode_tensor_map(&tm_z, z, 2, 4, dims, strides, box, SWZ_128, "trimul_output z");
    if (rc != B200TA_OK) return rc;
    constexpr int kBytes = kF32 ? 4 : 2;
    auto fix_out = [](int64_t stride, int extent) -> uint64_t { return uint64_t(extent == 1 ? 128 : stride) * kBytes; };
    uint64_t ostrides[3] = {fix_out(os_j, N), fix_out(os_i, N), fix_out(os_b, B)};
    uint32_t obox[4] = {64 / kBytes, 32, 1, 1};
    rc = encode_tensor_map(&tm_out, out, kBytes, 4, dims, ostrides, obox, SWZ_64, "trimul_output out");
    if (rc != B200TA_OK) return rc;
  }
  {
    // (j, i, plane): one load = 64 positions x 128 channels of one pair row
    uint64_t dims[3] = {uint64_t(N), uint64_t(N), uint64_t(B) * kTriHidden};
    uint64_t strides[2] = {uint64_t(pitch) * 2, uint64_t(pitch) * N * 2};
    uint32_t box[3] = {64, 1, kTriHidden};
    rc = encode_tensor_map(&tm_x, x, 2, 3, dims, strides, box, SWZ_128, "trimul_output x");
    if (rc != B200TA_OK) return rc;
  }
  const char* pk = static_cast<const char*>(packed);
  {
    uint64_t dims[2] = {uint64_t(kC), uint64_t(kTriRows)};
    uint64_t strides[1] = {uint64_t(kC) * 2};
    uint32_t box[2] = {64, 128};
    rc = encode_tensor_map(&tm_w, pk + kTriWOff, 2, 2, dims, strides, box, SWZ_128, "trimul_output weights");
    if (rc != B200TA_OK) return rc;
  }
  OutputParams p{};
  p.B = B, p.N = N;
  p.tiles_j = (N + kTileM - 1) / kTileM;
  p.num_tiles = B * N * p.tiles_j;
  p.sc = reinterpret_cast<const float2*>(pk + kTriScOff) + kTriInRows;
  p.eps = eps;
  p.add_residual = add_residual ? 1 : 0;
  p.mask = mask;
  p.ms_b = ms_b, p.ms_i = ms_i, p.ms_j = ms_j;
  p.status = st->status_dev;

  const int grid = p.num_tiles < st->num_sms ? p.num_tiles : st->num_sms;
  return launch_kernel(st, kF32 ? kKernelOutputF32 : kKernelOutput, trimul_output_kernel<kF32>, dim3(grid), kThreads, kSmDynamic, stream, tm_z, tm_x, tm_w, tm_out, p);
}

}  // namespace
}  // namespace b200ta

extern "C" {

int b200ta_trimul_output(const void* z, int64_t zs_b, int64_t zs_i, int64_t zs_j, const void* x, int64_t pitch,
                         const float* mask, int64_t ms_b, int64_t ms_i, int64_t ms_j, const void* packed, float eps,
                         int add_residual, void* out, int64_t os_b, int64_t os_i, int64_t os_j, int B, int N,
                         void* stream) {
  return b200ta::launch_output<false>(z, zs_b, zs_i, zs_j, x, pitch, mask, ms_b, ms_i, ms_j, packed, eps, add_residual, out,
                                      os_b, os_i, os_j, B, N, stream);
}

int b200ta_trimul_output_f32(const void* z, int64_t zs_b, int64_t zs_i, int64_t zs_j, const void* x, int64_t pitch,
                             const float* mask, int64_t ms_b, int64_t ms_i, int64_t ms_j, const void* packed, float eps,
                             int add_residual, void* out, int64_t os_b, int64_t os_i, int64_t os_j, int B, int N,
                             void* stream) {
  return b200ta::launch_output<true>(z, zs_b, zs_i, zs_j, x, pitch, mask, ms_b, ms_i, ms_j, packed, eps, add_residual, out,
                                     os_b, os_i, os_j, B, N, stream);
}

}  // extern "C"
