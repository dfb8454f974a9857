// The FP8 activation quantisation of one 1 x 128 group, shared by the stand-alone kernels and the
// fused decode prologue: scale = max(amax/448, FLT_MIN), code = e4m3(x / scale), both true
// divisions, as the reference's _fp8_input does
// (aklr/plugins/sglang/models/qwen3_moe/reference.py:44-54).
#pragma once
#include <cfloat>

#include "common.cuh"
#include "kernels.h"

namespace aklr {

__device__ __forceinline__ void unpack8(const uint4& raw, float (&v)[8]) {
  const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    v[2 * i] = __uint_as_float(w[i] << 16);
    v[2 * i + 1] = __uint_as_float(w[i] & 0xFFFF0000u);
  }
}

__device__ __forceinline__ float amax8(const float (&v)[8]) {
  float m = 0.0f;
#pragma unroll
  for (int i = 0; i < 8; ++i) m = fmaxf(m, fabsf(v[i]));
  return m;
}

__device__ __forceinline__ uint2 pack8_e4m3(const float (&v)[8]) {
  uint2 out;
  out.x = cvt_e4m3x2(v[0], v[1]) | (static_cast<uint32_t>(cvt_e4m3x2(v[2], v[3])) << 16);
  out.y = cvt_e4m3x2(v[4], v[5]) | (static_cast<uint32_t>(cvt_e4m3x2(v[6], v[7])) << 16);
  return out;
}

// x / scale rounded to nearest, as the reference's true division gives it, without eight IEEE divisions per
// lane: with y = RN(1/scale), q = RN(x*y), r = x - q*scale (exact in one fma) the quotient RN(q + r*y) is the
// correctly rounded x/scale whenever nothing under- or overflows on the way and scale's significand is not all
// ones (Markstein's theorem).  |x/scale| <= 448 here; the groups where the shortcut is not proven -- an all-ones
// significand, or a scale so small that its reciprocal or the residual leaves the normal range -- take the
// division itself (uniform over a group's lanes, rare).
struct ExactDivider {
  float scale, recip;
  bool slow;
  __device__ __forceinline__ explicit ExactDivider(float s) {
    scale = s;
    recip = __fdiv_rn(1.0f, s);  // correctly rounded
    const uint32_t bits = __float_as_uint(s);
    slow = (bits & 0x7FFFFFu) == 0x7FFFFFu || s < 1.0e-30f || s > 1.0e30f;
  }
  __device__ __forceinline__ float operator()(float x) const {
    if (slow) return __fdiv_rn(x, scale);
    const float q = __fmul_rn(x, recip);
    return __fmaf_rn(__fmaf_rn(-q, scale, x), recip, q);
  }
};

// LANES lanes x 128 / LANES consecutive values per 1 x 128 group.  Once the loads are wide these passes are bound by
// instructions, not by bytes: a group's reduction and its two true divisions cost the same whatever a lane holds, so
// 16 lanes x 8 values pay them twice as often as 8 x 16 (once per token at 16384 x 7168: 122 -> 93 us, the stand-alone op
// at 2048 x 7168 9.7 -> 7.8).  A few rows are the other way round: the chip is not full, a lane's chain of loads, maxima,
// quotients and conversions is all there is, and it is half as long with 8 values (64 x 7168: 1.94 us with 16 lanes, 2.15
// with 8; 512 x 1024, 4096 groups, 1.90 / 2.15).  The line: 100 x 7168, 5600 groups, 2.12 / 2.34; 1024 x 1024, 8192 groups,
// 2.76 / 2.36.  The codes and scales are the same either way.
constexpr int kWideGroupsFrom = 8192;  // groups of a launch from which eight lanes take each
inline int quant_lanes(int64_t groups) { return groups < kWideGroupsFrom ? 16 : 8; }

template <int LANES>
struct GroupValues {
  static constexpr int N = 128 / LANES;
  static_assert(N == 8 || N == 16, "a lane stores its codes in one or two 8-byte words");
  float v[N];
  __device__ __forceinline__ static int sub() { return threadIdx.x & (LANES - 1); }
  __device__ __forceinline__ static uint32_t mask() {  // this group's lanes
    return ((1u << LANES) - 1u) << (threadIdx.x & (32 - LANES));
  }
  __device__ __forceinline__ void load(const uint16_t* __restrict__ x) {  // this lane's values
    uint4 raw[N / 8];
#pragma unroll
    for (int h = 0; h < N / 8; ++h) raw[h] = reinterpret_cast<const uint4*>(x)[h];
#pragma unroll
    for (int h = 0; h < N / 8; ++h) {
      const uint32_t w[4] = {raw[h].x, raw[h].y, raw[h].z, raw[h].w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        v[h * 8 + 2 * i] = __uint_as_float(w[i] << 16);
        v[h * 8 + 2 * i + 1] = __uint_as_float(w[i] & 0xFFFF0000u);
      }
    }
  }
  __device__ __forceinline__ float group_amax(uint32_t group_mask) const {
    float m = 0.0f;
#pragma unroll
    for (int i = 0; i < N; ++i) m = fmaxf(m, fabsf(v[i]));
#pragma unroll
    for (int off = LANES / 2; off >= 1; off >>= 1) m = fmaxf(m, __shfl_xor_sync(group_mask, m, off, LANES));
    return m;
  }
  // Sixteen codes in one store where the caller's buffer allows it (``wide``; eight-byte alignment is all that is asked of it).
  static __device__ __forceinline__ void store(uint8_t* dst, const uint32_t (&codes)[N / 4], bool wide) {
    if (N == 16 && wide) {
      *reinterpret_cast<uint4*>(dst) = make_uint4(codes[0], codes[1], codes[N / 4 - 2], codes[N / 4 - 1]);
    } else {
#pragma unroll
      for (int h = 0; h < N / 8; ++h) reinterpret_cast<uint2*>(dst)[h] = make_uint2(codes[2 * h], codes[2 * h + 1]);
    }
  }
  __device__ __forceinline__ void pack(uint32_t (&codes)[N / 4]) const {
#pragma unroll
    for (int i = 0; i < N / 4; ++i)
      codes[i] = cvt_e4m3x2(v[4 * i], v[4 * i + 1]) | (static_cast<uint32_t>(cvt_e4m3x2(v[4 * i + 2], v[4 * i + 3])) << 16);
  }
};

// This group of lanes takes groups ``first``, ``first + stride``, ... of the row table (the caller's grid-stride).
template <int LANES>
__device__ __forceinline__ void gather_quant_fp8_groups(const GatherQuantParams& p, int64_t first, int64_t stride) {
  using Values = GroupValues<LANES>;
  const int groups_per_row = p.hidden >> 7;
  const int n_rows = p.num_rows ? min(*p.num_rows, p.n_rows) : p.n_rows;
  const int64_t total = static_cast<int64_t>(n_rows) * groups_per_row;
  const int sub = Values::sub();
  const uint32_t group_mask = Values::mask();
  const bool wide = reinterpret_cast<uintptr_t>(p.q) % 16 == 0;
  for (int64_t g = first; g < total; g += stride) {
    // 32-bit division: a 64-bit one is a subroutine of a hundred instructions, per group and lane
    const int row = static_cast<int>(static_cast<uint32_t>(g) / static_cast<uint32_t>(groups_per_row));
    const int grp = static_cast<int>(static_cast<uint32_t>(g) - static_cast<uint32_t>(row) * static_cast<uint32_t>(groups_per_row));
    int token = row;
    if (p.sorted_ids) {
      const int rid = p.sorted_ids[row];
      token = rid < 0 ? -1 : rid / p.routes_per_token;
    }
    uint8_t* dst = p.q + static_cast<size_t>(row) * p.hidden + grp * 128 + sub * Values::N;
    uint32_t codes[Values::N / 4] = {};
    if (token < 0) {  // padding rows are never read back; uniform over the group's lanes
      if (p.zero_padding) Values::store(dst, codes, wide);  // but multiplied: zero codes cost the tensor core least
      continue;
    }
    Values x;
    x.load(reinterpret_cast<const uint16_t*>(p.x) + static_cast<size_t>(token) * p.hidden + grp * 128 + sub * Values::N);
    const float scale = fmaxf(__fdiv_rn(x.group_amax(group_mask), 448.0f), FLT_MIN);
    const ExactDivider divide(scale);
#pragma unroll
    for (int i = 0; i < Values::N; ++i) x.v[i] = divide(x.v[i]);
    x.pack(codes);
    Values::store(dst, codes, wide);
    if (sub == 0) {
      if (p.block_m > 0)  // [block][group][row in block]: what the grouped GEMM stages per tile
        p.scales[(static_cast<size_t>(row / p.block_m) * groups_per_row + grp) * p.block_m + row % p.block_m] = scale;
      else
        p.scales[static_cast<size_t>(row) * groups_per_row + grp] = scale;
    }
  }
}

}  // namespace aklr
