// Router projection on the tensor cores, sm_100a: logits[T, E] = bf16( x[T, H] . W[E, H]^T ) with
// float32 accumulation in TMEM, the rounding point of the reference's _router_logits
// (aklr/plugins/sglang/models/qwen3_moe/reference.py:24-31).  One CTA per 128 tokens x 16..256
// experts: TMA (SWIZZLE_128B, 64 bf16 = 128 bytes of K per box, one or two boxes per stage) feeds
// tcgen05.mma kind::f16 (M128, N = experts of the tile, K16); rows and experts past the end are zero-filled by the
// TMA.  192 threads: warp 0 TMA, warp 1 MMA + TMEM, warps 2..5 epilogue (one TMEM lane quarter each).
//
// A tile's time is the latency of its loads, not their bytes or its arithmetic: with one CTA per 128 tokens and all
// experts (four stages of 48 KB) 64 tokens on 7168 x 256 took 43 us on ONE SM.  So the experts are spread over as
// many CTAs as the chip has SMs, which makes the stages small and the ring deep; every logit is still one
// accumulation over K in the same order, so no bit of it changes (splitting K over CTAs would be faster still and
// change roundings, and with them picks).
#include "common.cuh"
#include "kernels.h"

namespace aklr {

namespace {

constexpr int kThreads = 192;
constexpr int kMaxStages = 10;
constexpr int kABytes = 128 * 128;
constexpr int kSmemBudget = 222 * 1024;  // stages; barriers and alignment slack fit in the rest of 227 KB

struct RouterParams {
  CUtensorMap map_x;  // bf16 [T, H], box 64 x 128
  CUtensorMap map_w;  // bf16 [E, H], box 64 x n_tile
  uint16_t* logits;   // bf16 [T, E]
  int32_t* status;    // optional [2]
  int32_t* host_status;  // the device's host-visible copy of a failure (or null)
  int n_tokens, hidden, n_routed, n_tile, stages;
};

__device__ __forceinline__ void umma_bf16(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc,
                                          uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
      : "memory");
}

// BOXES: 64-wide boxes of K per stage, two where hidden allows and the tile leaves room for three such stages and more
// (256 experts do not: two of 96 KB, at which 16384 tokens on 7168 x 256 took 69-71 us, 62-65 with four stages of one box).
// LONE_LANE: one lane of the producer and of the MMA warp waits and issues, the others stand by, in place of the whole warp
// waiting and an elected lane issuing.  Cheap issue does not matter where an MMA of 256 columns outlasts it, and the vote
// after every wait then is one hand-off more in a ring of four stages: 9600 / 16384 / 32768 tokens on 7168 x 256 51 / 62 /
// 121 us by the warp, 48 / 58 / 115 by the lane; below 256 columns the lane is the slower (300 tokens: 19 / 27).
template <int BOXES, bool LONE_LANE>
__global__ void __launch_bounds__(kThreads, 1) router_gemm_tc_kernel(const __grid_constant__ RouterParams p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int box_bytes = kABytes + p.n_tile * 128, stage_bytes = BOXES * box_bytes;
  const int kStages = p.stages;
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + kStages * stage_bytes);
  uint64_t* empty = full + kStages;
  uint64_t* acc_full = empty + kStages;
  uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(acc_full + 1);
  // everything lives in the dynamic allocation: a static __shared__ variable on top of the 227 KB
  // opt-in would exceed the per-CTA limit
  int* abort_word = reinterpret_cast<int*>(tmem_ptr + 1);
  int* local_status = abort_word + 1;
  volatile int* abort_flag = abort_word;
  int* status = p.status ? p.status : local_status;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int k_steps = (p.hidden >> 6) / BOXES;
  const int tok0 = blockIdx.x * 128, exp0 = blockIdx.y * p.n_tile;
  uint32_t tmem_cols = 32;
  while (tmem_cols < static_cast<uint32_t>(p.n_tile)) tmem_cols <<= 1;

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(acc_full, 1);
    *abort_word = 0;
    local_status[0] = local_status[1] = 0;
    fence_mbar_init();
    tma_prefetch_desc(&p.map_x);
    tma_prefetch_desc(&p.map_w);
  }
  if (warp == 1) {
    tmem_alloc(tmem_ptr, tmem_cols);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_ptr;
  griddep_wait();
  griddep_launch();
  auto wait = [&](uint64_t* bar, uint32_t parity, int where) {
    return LONE_LANE ? mbar_wait(bar, parity, abort_flag, status, where) : mbar_wait_warp(bar, parity, abort_flag, status, where);
  };
  const bool stands_by = LONE_LANE && warp < 2 && lane != 0;

  if (warp == 0) {
    const bool leader = LONE_LANE || elect_one();
    int s = 0;
    uint32_t ph = 0;
    for (int it = stands_by ? k_steps : 0; it < k_steps; ++it) {
      if (!wait(&empty[s], ph ^ 1, 31)) break;
      uint8_t* st = smem + s * stage_bytes;
      if (leader) {
        mbar_expect_tx(&full[s], stage_bytes);
#pragma unroll
        for (int b = 0; b < BOXES; ++b) {
          tma_load_2d(st + b * box_bytes, &p.map_x, &full[s], (it * BOXES + b) * 64, tok0);
          tma_load_2d(st + b * box_bytes + kABytes, &p.map_w, &full[s], (it * BOXES + b) * 64, exp0);
        }
      }
      if (++s == kStages) { s = 0; ph ^= 1; }
    }
  } else if (warp == 1) {
    const bool leader = LONE_LANE || elect_one();
    // kind::f16: f32 accumulator, bf16 A and B, K-major, M 128, N n_tile
    const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(p.n_tile >> 3) << 17) |
                           (static_cast<uint32_t>(128 >> 4) << 24);
    bool ok = !stands_by;
    int s = 0;
    uint32_t ph = 0;
    for (int it = 0; it < k_steps && ok; ++it) {
      if (!wait(&full[s], ph, 32)) { ok = false; break; }
      tc_fence_after_sync();
      if (leader) {
#pragma unroll
        for (int b = 0; b < BOXES; ++b) {
          const uint32_t a0 = smem_u32(smem + s * stage_bytes + b * box_bytes);
          const uint64_t da = umma_desc_sw128(a0), db = umma_desc_sw128(a0 + kABytes);
#pragma unroll
          for (int k = 0; k < 4; ++k) umma_bf16(tmem_base, da + 2 * k, db + 2 * k, idesc, (it > 0 || b > 0 || k > 0) ? 1u : 0u);
        }
        tc_commit(&empty[s]);
      }
      if (++s == kStages) { s = 0; ph ^= 1; }
    }
    if (ok && leader) tc_commit(acc_full);
  } else {
    const int quarter = warp & 3;
    const int token = tok0 + quarter * 32 + lane;
    const bool wide = (p.n_routed & 7) == 0 && (reinterpret_cast<uintptr_t>(p.logits) & 15) == 0;  // 16-byte stores start on their boundary
    const bool got = mbar_wait(acc_full, 0, abort_flag, status, 33);
    tc_fence_after_sync();
    const uint32_t t0 = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
    for (int c = 0; c < p.n_tile; c += 16) {
      uint32_t r[16];
      AKLR_TMEM_LD_16(t0 + c, r);
      tc_wait_ld();
      if (got && token < p.n_tokens) {
        uint16_t* dst = p.logits + static_cast<size_t>(token) * p.n_routed + exp0 + c;
        if (wide && exp0 + c + 16 <= p.n_routed) {
          uint32_t o[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const __nv_bfloat162 two = __floats2bfloat162_rn(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1]));
            o[i] = *reinterpret_cast<const uint32_t*>(&two);
          }
          *reinterpret_cast<uint4*>(dst) = make_uint4(o[0], o[1], o[2], o[3]);
          *reinterpret_cast<uint4*>(dst + 8) = make_uint4(o[4], o[5], o[6], o[7]);
        } else {
#pragma unroll
          for (int i = 0; i < 16; ++i)
            if (exp0 + c + i < p.n_routed) {
              const __nv_bfloat16 v = __float2bfloat16_rn(__uint_as_float(r[i]));
              dst[i] = *reinterpret_cast<const uint16_t*>(&v);
            }
        }
      }
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (*abort_flag) {
    if (threadIdx.x == 0) publish_wait_failure(status, p.host_status);
    const uint64_t start = global_timer_ns();
    while (global_timer_ns() - start < 200000ull) __nanosleep(1000);
  }
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, tmem_cols);
  }
}


// ---- float32 router weights ----------------------------------------------------------------------
// logits[T, E] = x[T, H] (bf16) . W[E, H]^T (float32), float32 logits, nothing rounded on the way in: a float32 weight
// is the sum of three bf16 terms (its 24 significant bits cut into 8 + 8 + 8, exact short of underflow), a product of two
// bf16 values is exact in float32, and the three products' sums are kept apart and added once, smallest first.  So the
// only roundings are those of the accumulation: one per 16 products (K = 16 per MMA), in kF32Slices accumulators of the first
// term that share K out between them, where a CUDA-core chain over H has one per product.
// An infinite activation times a low term that is zero is NaN where the product itself is infinite, so a logit whose first
// term is not finite is that term's sum alone: +-inf and NaN come out as from the CUDA-core kernels, whatever the batch
// size.  (The first term of a weight below 2^-133 is zero too: its product with an infinity is NaN here.)
//
// One CTA per 128 tokens x 32 experts, 64 of K per stage: TMA loads the bf16 token tile (16 KB, SWIZZLE_128B) and the
// raw weights (32 x 64 floats), four of eight warps turn the weights into one 96-row operand tile (32 rows of each term,
// swizzled as the MMA reads it), and two MMAs of M128 K16 per step cover the first term (N 32) and the other two (N 64).
// 320 threads: warp 0 TMA, warp 1 MMA + TMEM, warps 2..5 and 6..9 conversion of alternate stages, warps 2..5 then the
// epilogue.  2000 tokens on 3072 x 256: 194 us on the CUDA cores (bound by shared-memory
// reads of a 4 x 4 tile per thread and a memory round trip per 16 k), 30 us here; against 64 bits the relative error (2-norm) fell from 9.9e-7 to 2.4e-7, at
// 4096 x 7168 from 1.5e-6 to 5.8e-7 (with 4 accumulators it would be 1.8e-6: the MMA truncates as it accumulates).
constexpr int kF32Experts = 32;
constexpr int kF32Slices = 12;                               // accumulators of the first term along K; the other two terms share 64 columns
constexpr int kF32RawBytes = kF32Experts * 64 * 4;           // raw weights of a stage
constexpr int kF32TermBytes = 3 * kF32Experts * 128;         // their bf16 terms
constexpr int kF32StageBytes = kABytes + kF32TermBytes + kF32RawBytes;
constexpr int kF32Stages = 6;

struct RouterF32Params {
  CUtensorMap map_x;  // bf16 [T, H], box 64 x 128, SWIZZLE_128B
  CUtensorMap map_w;  // float32 [E, H], box 64 x 32, no swizzle
  float* logits;      // [T, E]
  int32_t* host_status;
  int n_tokens, hidden, n_routed;
};

constexpr int kF32Threads = 320;
__global__ void __launch_bounds__(kF32Threads, 1) router_gemm_f32_tc_kernel(const __grid_constant__ RouterF32Params p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + kF32Stages * kF32StageBytes);
  uint64_t* ready = full + kF32Stages;  // the stage's terms are written
  uint64_t* empty = ready + kF32Stages;
  uint64_t* acc_full = empty + kF32Stages;
  uint32_t* tmem_ptr = reinterpret_cast<uint32_t*>(acc_full + 1);
  int* abort_word = reinterpret_cast<int*>(tmem_ptr + 1);
  int* status = abort_word + 1;
  volatile int* abort_flag = abort_word;

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int k_steps = p.hidden >> 6;
  const int tok0 = blockIdx.x * 128, exp0 = blockIdx.y * kF32Experts;
  const int slices = k_steps < kF32Slices ? k_steps : kF32Slices;  // every accumulator is written by at least one step
  auto slice_of = [&](int it) { return it * slices / k_steps; };

  if (threadIdx.x == 0) {
    for (int s = 0; s < kF32Stages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&ready[s], 4);
      mbar_init(&empty[s], 1);
    }
    mbar_init(acc_full, 1);
    *abort_word = 0;
    status[0] = status[1] = 0;
    fence_mbar_init();
    tma_prefetch_desc(&p.map_x);
    tma_prefetch_desc(&p.map_w);
  }
  if (warp == 1) {
    tmem_alloc(tmem_ptr, 512);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_ptr;
  griddep_wait();
  griddep_launch();

  if (warp == 0) {
    const bool leader = elect_one();
    int s = 0;
    uint32_t ph = 0;
    for (int it = 0; it < k_steps; ++it) {
      if (!mbar_wait_warp(&empty[s], ph ^ 1, abort_flag, status, 34)) break;
      uint8_t* st = smem + s * kF32StageBytes;
      if (leader) {
        mbar_expect_tx(&full[s], kABytes + kF32RawBytes);
        tma_load_2d(st, &p.map_x, &full[s], it * 64, tok0);
        tma_load_2d(st + kABytes + kF32TermBytes, &p.map_w, &full[s], it * 64, exp0);
      }
      if (++s == kF32Stages) { s = 0; ph ^= 1; }
    }
  } else if (warp == 1) {
    const bool leader = elect_one();
    auto idesc_of = [](int n) {
      return (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(n >> 3) << 17) | (static_cast<uint32_t>(128 >> 4) << 24);
    };
    bool ok = true;
    int s = 0;
    uint32_t ph = 0;
    for (int it = 0; it < k_steps; ++it) {
      if (!mbar_wait_warp(&full[s], ph, abort_flag, status, 35)) { ok = false; break; }
      if (!mbar_wait_warp(&ready[s], ph, abort_flag, status, 36)) { ok = false; break; }
      tc_fence_after_sync();
      if (leader) {
        const uint32_t a0 = smem_u32(smem + s * kF32StageBytes);
        const uint64_t da = umma_desc_sw128(a0), db = umma_desc_sw128(a0 + kABytes);
        const int slice = slice_of(it);
        const bool first = it == 0 || slice_of(it - 1) != slice;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          umma_bf16(tmem_base + (2 + slice) * kF32Experts, da + 2 * k, db + 2 * k, idesc_of(kF32Experts), (!first || k > 0) ? 1u : 0u);
          umma_bf16(tmem_base, da + 2 * k, db + ((kF32Experts * 128) >> 4) + 2 * k, idesc_of(2 * kF32Experts), (it > 0 || k > 0) ? 1u : 0u);
        }
        tc_commit(&empty[s]);
      }
      if (++s == kF32Stages) { s = 0; ph ^= 1; }
    }
    if (ok && leader) tc_commit(acc_full);
  } else {
    // two groups of four warps take alternate stages; a thread turns 8 floats of rows `row` and `row + 16`
    const int group = (warp - 2) >> 2, ct = (threadIdx.x - 64) & 127;
    const int row = ct >> 3, chunk = ct & 7;
    int s = group;
    uint32_t ph = 0;
    bool got = true;
    for (int it = group; it < k_steps; it += 2) {
      if (!mbar_wait_warp(&full[s], ph, abort_flag, status, 37)) { got = false; break; }
      uint8_t* st = smem + s * kF32StageBytes;
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        const int r = row + half * 16;
        const float4* raw = reinterpret_cast<const float4*>(st + kABytes + kF32TermBytes) + r * 16 + chunk * 2;
        // eight lanes read one row: the upper four take their second 16 bytes first, so that no two meet in a bank
        const bool swap = chunk >= 4;
        const float4 f0 = raw[swap ? 1 : 0], f1 = raw[swap ? 0 : 1];
        float v[8] = {swap ? f1.x : f0.x, swap ? f1.y : f0.y, swap ? f1.z : f0.z, swap ? f1.w : f0.w,
                      swap ? f0.x : f1.x, swap ? f0.y : f1.y, swap ? f0.z : f1.z, swap ? f0.w : f1.w};
#pragma unroll
        for (int term = 0; term < 3; ++term) {
          uint32_t o[4];
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            float& a = v[2 * q];
            float& b = v[2 * q + 1];
            const float ah = __uint_as_float(__float_as_uint(a) & 0xFFFF0000u), bh = __uint_as_float(__float_as_uint(b) & 0xFFFF0000u);
            o[q] = (__float_as_uint(a) >> 16) | __float_as_uint(bh);
            a = a == ah ? 0.0f : a - ah;  // exact: what the term left over (an infinite weight leaves nothing, a NaN stays one)
            b = b == bh ? 0.0f : b - bh;
          }
          *reinterpret_cast<uint4*>(st + kABytes + (term * kF32Experts + r) * 128 + ((chunk ^ (r & 7)) << 4)) = make_uint4(o[0], o[1], o[2], o[3]);
        }
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the MMA reads these bytes through the async proxy
      __syncwarp();
      if (lane == 0) mbar_arrive(&ready[s]);
      s += 2;  // kF32Stages is even
      if (s >= kF32Stages) { s -= kF32Stages; ph ^= 1; }
    }
    const int quarter = warp & 3;
    const int token = tok0 + quarter * 32 + lane;
    got = got && group == 0 && mbar_wait_warp(acc_full, 0, abort_flag, status, 38);
    tc_fence_after_sync();
    if (got) {
      const uint32_t t0 = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16);
#pragma unroll
      for (int c = 0; c < kF32Experts; c += 16) {
        float sum[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) sum[i] = 0.0f;
#pragma unroll
        for (int low = 1; low >= 0; --low) {  // the lowest term's sum, then the middle one's
          uint32_t r[16];
          AKLR_TMEM_LD_16(t0 + low * kF32Experts + c, r);
          tc_wait_ld();
#pragma unroll
          for (int i = 0; i < 16; ++i) sum[i] += __uint_as_float(r[i]);
        }
        for (int sl = 0; sl < slices; ++sl) {
          uint32_t r[16];
          AKLR_TMEM_LD_16(t0 + (2 + sl) * kF32Experts + c, r);
          tc_wait_ld();
#pragma unroll
          for (int i = 0; i < 16; ++i) sum[i] += __uint_as_float(r[i]);
        }
        bool finite = true;
#pragma unroll
        for (int i = 0; i < 16; ++i) finite = finite && isfinite(sum[i]);
        if (!__all_sync(0xFFFFFFFFu, finite)) {  // see above: infinities meet the low terms' zeros
          float first[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) first[i] = 0.0f;
          for (int sl = 0; sl < slices; ++sl) {
            uint32_t r[16];
            AKLR_TMEM_LD_16(t0 + (2 + sl) * kF32Experts + c, r);
            tc_wait_ld();
#pragma unroll
            for (int i = 0; i < 16; ++i) first[i] += __uint_as_float(r[i]);
          }
#pragma unroll
          for (int i = 0; i < 16; ++i)
            if (!isfinite(first[i])) sum[i] = first[i];
        }
        if (token < p.n_tokens) {
          float* dst = p.logits + static_cast<size_t>(token) * p.n_routed + exp0 + c;
          if (exp0 + c + 16 <= p.n_routed && (p.n_routed & 3) == 0) {
#pragma unroll
            for (int i = 0; i < 16; i += 4) *reinterpret_cast<float4*>(dst + i) = make_float4(sum[i], sum[i + 1], sum[i + 2], sum[i + 3]);
          } else {
#pragma unroll
            for (int i = 0; i < 16; ++i)
              if (exp0 + c + i < p.n_routed) dst[i] = sum[i];
          }
        }
      }
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (*abort_flag) {
    if (threadIdx.x == 0) publish_wait_failure(status, p.host_status);
    const uint64_t start = global_timer_ns();
    while (global_timer_ns() - start < 200000ull) __nanosleep(1000);
  }
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, 512);
  }
}

}  // namespace

// Experts per CTA: the fewest (a power of two from 16, what the layout of the logits allows to be written in whole
// sectors) whose CTAs still fit the chip in one wave.
int router_gemm_tc_pick_n_tile(int n_tokens, int n_routed, int sm_count) {
  const int64_t token_tiles = (n_tokens + 127) / 128;
  int n_tile = 16;
  while (n_tile < 256 && n_tile < n_routed && token_tiles * ((n_routed + n_tile - 1) / n_tile) > sm_count) n_tile *= 2;
  return n_tile;
}

int launch_router_gemm_tc(const CUtensorMap& map_x, const CUtensorMap& map_w, void* logits, int n_tokens, int hidden,
                          int n_routed, int n_tile, int32_t* host_status, cudaStream_t stream) {
  if (hidden % 64 != 0 || n_tile % 16 != 0 || n_tile < 16 || n_tile > 256) return AKLR_ERR_UNSUPPORTED_SHAPE;
  RouterParams p{};
  p.map_x = map_x;
  p.map_w = map_w;
  p.logits = static_cast<uint16_t*>(logits);
  p.status = nullptr;
  p.host_status = host_status;
  p.n_tokens = n_tokens;
  p.hidden = hidden;
  p.n_routed = n_routed;
  p.n_tile = n_tile;
  const int boxes = hidden % 128 == 0 && n_tile < 256 ? 2 : 1;
  const int stage_bytes = boxes * (kABytes + n_tile * 128);
  p.stages = kSmemBudget / stage_bytes;
  if (p.stages > kMaxStages) p.stages = kMaxStages;
  const size_t smem = static_cast<size_t>(p.stages) * stage_bytes + (2 * p.stages + 1) * 8 + 32 + 1024;
  auto* kernel = n_tile == 256 ? router_gemm_tc_kernel<1, true> : boxes == 2 ? router_gemm_tc_kernel<2, false> : router_gemm_tc_kernel<1, false>;
  if (ensure_max_dynamic_smem(reinterpret_cast<const void*>(kernel)) != AKLR_OK) return AKLR_ERR_CUDA;
  const dim3 grid((n_tokens + 127) / 128, (n_routed + n_tile - 1) / n_tile);
  return launch_kernel(kernel, grid, dim3(kThreads), smem, stream, 1, p) == cudaSuccess ? AKLR_OK : AKLR_ERR_CUDA;
}

int launch_router_gemm_f32_tc(const CUtensorMap& map_x, const CUtensorMap& map_w, float* logits, int n_tokens, int hidden,
                              int n_routed, int32_t* host_status, cudaStream_t stream) {
  if (hidden % 64 != 0 || n_tokens < 1 || n_routed < 1) return AKLR_ERR_UNSUPPORTED_SHAPE;
  RouterF32Params p{};
  p.map_x = map_x;
  p.map_w = map_w;
  p.logits = logits;
  p.host_status = host_status;
  p.n_tokens = n_tokens;
  p.hidden = hidden;
  p.n_routed = n_routed;
  const size_t smem = static_cast<size_t>(kF32Stages) * kF32StageBytes + (3 * kF32Stages + 1) * 8 + 32 + 1024;
  if (ensure_max_dynamic_smem(reinterpret_cast<const void*>(router_gemm_f32_tc_kernel)) != AKLR_OK) return AKLR_ERR_CUDA;
  const dim3 grid((n_tokens + 127) / 128, (n_routed + kF32Experts - 1) / kF32Experts);
  return launch_kernel(router_gemm_f32_tc_kernel, grid, dim3(kF32Threads), smem, stream, 1, p) == cudaSuccess ? AKLR_OK : AKLR_ERR_CUDA;
}

}  // namespace aklr
