// Row payloads of pair masks in one pass each (bound by launch latency at the sizes of a mask: a warp takes a row, reads
// it once, and ballots say which keys take part).  As torch operations the same payloads took 5 (lengths) and 13
// (key bits) launches of 2-10 us.
#include "common.cuh"

namespace b200ta {
namespace {

constexpr int kWarps = 8;

struct MaskParams {
  const float* mask;
  long long s_b, s_r, s_s;  // element strides of [B, rows, keys]
  float threshold;          // a key takes part if mask >= threshold (inclusive) or mask > threshold
  int inclusive;
  int B, R, S;
  int32_t* lengths;    // [B, R]
  int32_t* lengths_t;  // [B, S] of the transposed mask, or NULL (R == S)
  uint32_t* bits;      // [B, R, ceil(S / 32)], or NULL
};

// lengths: number of keys that take part; with bits: last key that takes part + 1.
__global__ void __launch_bounds__(kWarps * 32) mask_rows_kernel(const MaskParams p) {
  pdl_trigger();
  pdl_wait();
  int row = blockIdx.x * kWarps + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  const bool transposed = row >= p.B * p.R;
  if (transposed) row -= p.B * p.R;
  if (row >= p.B * (transposed ? p.S : p.R) || (transposed && p.lengths_t == nullptr)) return;
  const int rows = transposed ? p.S : p.R, keys = transposed ? p.R : p.S;
  const int b = row / rows, r = row - b * rows;
  const float* src = p.mask + b * p.s_b + r * (transposed ? p.s_s : p.s_r);
  const long long step = transposed ? p.s_r : p.s_s;
  const int words = (keys + 31) >> 5;
  int count = 0, last = 0;
  for (int w = 0; w < words; ++w) {
    const int k = w * 32 + lane;
    bool valid = false;
    if (k < keys) {
      const float v = __ldg(src + k * step);
      valid = p.inclusive ? v >= p.threshold : v > p.threshold;
    }
    const uint32_t word = __ballot_sync(0xffffffffu, valid);
    count += __popc(word);
    if (word) last = w * 32 + 32 - __clz(word);
    if (p.bits != nullptr && lane == 0) p.bits[(long long)row * words + w] = word;
  }
  if (lane == 0) (transposed ? p.lengths_t : p.lengths)[row] = p.bits != nullptr ? last : count;
}

int launch(const MaskParams& p, void* stream) {
  B200TA_REQUIRE(p.mask && p.lengths, "mask: NULL pointer");
  B200TA_REQUIRE(p.B > 0 && p.R > 0 && p.S > 0, "mask: bad sizes B=%d R=%d S=%d", p.B, p.R, p.S);
  const int64_t rows = int64_t(p.B) * (p.R + (p.lengths_t ? p.S : 0));
  B200TA_REQUIRE(rows < (int64_t(1) << 30), "mask: too many rows");
  DeviceState* st = nullptr;
  const int rc = get_device_state(&st);
  if (rc != B200TA_OK) return rc;
  return launch_kernel(st, kKernelMaskRows, mask_rows_kernel, dim3(unsigned((rows + kWarps - 1) / kWarps)), kWarps * 32, 0,
                       stream, p);
}

}  // namespace
}  // namespace b200ta

extern "C" {

int b200ta_mask_lengths(const float* mask, int64_t s_b, int64_t s_r, int64_t s_s, int32_t* lengths, int32_t* lengths_t,
                        int B, int R, int S, void* stream) {
  return b200ta::launch({mask, s_b, s_r, s_s, 0.5f, 0, B, R, S, lengths, lengths_t, nullptr}, stream);
}

int b200ta_mask_bits(const float* mask, int64_t s_b, int64_t s_r, int64_t s_s, int additive, int32_t* lengths,
                     uint32_t* bits, int B, int R, int S, void* stream) {
  if (bits == nullptr) return b200ta::fail(B200TA_ERR_INVALID, "mask_bits: bits must not be NULL");
  return b200ta::launch({mask, s_b, s_r, s_s, additive ? 0.f : 0.5f, additive ? 1 : 0, B, R, S, lengths, nullptr, bits}, stream);
}

}  // extern "C"
