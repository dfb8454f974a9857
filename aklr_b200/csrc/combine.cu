// Top-k weighted combine (unpermute) and the router projection, sm_100a.
//
// combine: out[t] = bf16( sum over the token's routes of its per-route row ), summed in float32
// in slot order; the rows already carry the route weight (the down projection applies it).
// Routes to experts this rank does not hold add nothing, as in the reference's expert_mask /
// expert_offset statements (aklr/ops/fused_moe/reference.py:78-84).  HBM-bound: 16-byte loads.
//
// router: logits = bf16( x @ W^T ) with float32 accumulation, the rounding point of the
// reference's _router_logits (aklr/plugins/sglang/models/qwen3_moe/reference.py:24-31).
#include <algorithm>

#include "common.cuh"
#include "kernels.h"

namespace aklr {

// A warp takes ``chunks_per_item`` runs of 256 columns of one token: its routes are looked at once per item, one lane
// each, and are a bit mask from then on, so that a thread is left with its rows' loads (nine at a time in flight) and
// additions.  With every thread reading and testing all of its token's ids per 8 columns, 16384 tokens x 9 routes on 7168
// (2.35 GB) took 490 us, 4.8 TB/s; so 385, 6.1.  (In a capture at 4096 tokens that form issued in 45 % of its cycles at three
// CTAs per SM and used 69 % of the memory's nominal rate, this one 75 %.)
constexpr int kCombineSlots = 9;
__global__ void __launch_bounds__(256, 4) combine_kernel(CombineParams p, int chunks_per_item, int items_per_token) {
  griddep_wait();
  griddep_launch();
  const int lane = threadIdx.x & 31;
  const int warps = (gridDim.x * blockDim.x) >> 5;
  const int items = p.n_tokens * items_per_token;  // < 2^31: checked at launch
  for (int item = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; item < items; item += warps) {
    const int token = static_cast<int>(static_cast<uint32_t>(item) / static_cast<uint32_t>(items_per_token));
    const int chunk0 = (item - token * items_per_token) * chunks_per_item;
    bool mine = false;  // lane s: whether slot s of the token is added here (at most 32 slots)
    if (lane < p.routes_per_token && (!p.num_local_tokens || token < __ldg(p.num_local_tokens))) {
      const int e = __ldg(p.topk_ids + token * p.routes_per_token + lane);
      mine = e >= 0 && e < p.n_experts_global && (!p.expert_map || __ldg(p.expert_map + e) >= 0);
    }
    const uint32_t live = __ballot_sync(0xFFFFFFFFu, mine);
    const uint16_t* rows = static_cast<const uint16_t*>(p.rows) + static_cast<size_t>(token) * p.routes_per_token * p.hidden;
    uint16_t* out = static_cast<uint16_t*>(p.out) + static_cast<size_t>(token) * p.hidden;
    for (int c = 0; c < chunks_per_item; ++c) {
      const int col = (chunk0 + c) * 256 + lane * 8;
      if (col >= p.hidden) break;
      float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
      // slots are summed in order; their loads do not wait for one another
      for (int s0 = 0; s0 < p.routes_per_token; s0 += kCombineSlots) {
        uint4 raw[kCombineSlots];
#pragma unroll
        for (int d = 0; d < kCombineSlots; ++d)
          if (s0 + d < 32 && (live >> (s0 + d)) & 1u)
            raw[d] = *reinterpret_cast<const uint4*>(rows + static_cast<size_t>(s0 + d) * p.hidden + col);
#pragma unroll
        for (int d = 0; d < kCombineSlots; ++d) {
          if (s0 + d >= 32 || !((live >> (s0 + d)) & 1u)) continue;
          const uint32_t w[4] = {raw[d].x, raw[d].y, raw[d].z, raw[d].w};
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            acc[2 * q] += __uint_as_float(w[q] << 16);
            acc[2 * q + 1] += __uint_as_float(w[q] & 0xFFFF0000u);
          }
        }
      }
      uint4 packed;
      uint32_t* o = reinterpret_cast<uint32_t*>(&packed);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const __nv_bfloat162 two = __floats2bfloat162_rn(acc[2 * q], acc[2 * q + 1]);
        o[q] = *reinterpret_cast<const uint32_t*>(&two);
      }
      *reinterpret_cast<uint4*>(out + col) = packed;
    }
  }
}

int launch_combine(const CombineParams& p, cudaStream_t stream) {
  if (p.hidden % 8 != 0 || p.routes_per_token > 32) return AKLR_ERR_UNSUPPORTED_SHAPE;
  if (p.n_tokens == 0) return AKLR_OK;
  const int64_t total = static_cast<int64_t>(p.n_tokens) * (p.hidden / 8);
  if (total >= (int64_t{1} << 31)) return AKLR_ERR_TOO_LARGE;
  // One run per warp until every SM's 32 warps have several; then four, so that an item's look at its routes is shared.
  const int chunks = (p.hidden + 255) / 256;
  const int per_item = static_cast<int64_t>(p.n_tokens) * chunks >= 148 * 32 * 8 ? 4 : 1;
  const int per_token = (chunks + per_item - 1) / per_item;
  const int64_t blocks = (static_cast<int64_t>(p.n_tokens) * per_token + 7) / 8;
  const int grid = static_cast<int>(blocks < 148 * 8 ? blocks : 148 * 8);
  return launch_kernel(combine_kernel, dim3(grid), dim3(256), 0, stream, 1, p, per_item, per_token) == cudaSuccess ? AKLR_OK : AKLR_ERR_CUDA;
}

// One warp per (TOKENS tokens, EXPERTS experts): lanes stride the hidden dimension with 16-byte loads, and the loads of
// UNROLL strides are on their way before the first product.  What bounds it is the latency of those loads -- a decode
// call finds the router weight in HBM -- so a warp has 12-16 of them in flight; with the loads of one stride at a time
// (28 strides at 7168) one token on 256 experts took 16.9 us and 17 tokens on 2048 x 512 31 us.  Several tokens per warp
// share a weight load and several experts a token load.  Each dot product is the same chain of FMAs whatever the shape.
template <int TOKENS, int EXPERTS, int UNROLL>
__global__ void __launch_bounds__(256)
router_gemm_kernel(const uint16_t* __restrict__ x, const uint16_t* __restrict__ w, uint16_t* __restrict__ logits,
                   int n_tokens, int hidden, int n_routed) {
  const int lane = threadIdx.x & 31;
  const int groups = (n_routed + EXPERTS - 1) / EXPERTS;
  const int item = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int tok0 = item / groups * TOKENS, e0 = item % groups * EXPERTS;
  griddep_wait();
  griddep_launch();
  if (tok0 >= n_tokens) return;
  const uint16_t* xp[TOKENS];  // rows past the end repeat the last one and are not stored
  const uint16_t* wp[EXPERTS];
#pragma unroll
  for (int t = 0; t < TOKENS; ++t) xp[t] = x + static_cast<size_t>(min(tok0 + t, n_tokens - 1)) * hidden;
#pragma unroll
  for (int j = 0; j < EXPERTS; ++j) wp[j] = w + static_cast<size_t>(min(e0 + j, n_routed - 1)) * hidden;
  float acc[TOKENS][EXPERTS] = {};
  for (int h0 = lane * 8; h0 < hidden; h0 += 256 * UNROLL) {
    uint4 xr[UNROLL][TOKENS], wr[UNROLL][EXPERTS];
#pragma unroll
    for (int u = 0; u < UNROLL; ++u) {
      const int h = h0 + u * 256;
      if (h < hidden) {
#pragma unroll
        for (int j = 0; j < EXPERTS; ++j) wr[u][j] = __ldg(reinterpret_cast<const uint4*>(wp[j] + h));
#pragma unroll
        for (int t = 0; t < TOKENS; ++t) xr[u][t] = *reinterpret_cast<const uint4*>(xp[t] + h);
      }
    }
#pragma unroll
    for (int u = 0; u < UNROLL; ++u) {
      if (h0 + u * 256 >= hidden) continue;
#pragma unroll
      for (int t = 0; t < TOKENS; ++t) {
        const uint32_t xw[4] = {xr[u][t].x, xr[u][t].y, xr[u][t].z, xr[u][t].w};
#pragma unroll
        for (int j = 0; j < EXPERTS; ++j) {
          const uint32_t ww[4] = {wr[u][j].x, wr[u][j].y, wr[u][j].z, wr[u][j].w};
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            acc[t][j] = fmaf(__uint_as_float(xw[q] << 16), __uint_as_float(ww[q] << 16), acc[t][j]);
            acc[t][j] = fmaf(__uint_as_float(xw[q] & 0xFFFF0000u), __uint_as_float(ww[q] & 0xFFFF0000u), acc[t][j]);
          }
        }
      }
    }
  }
#pragma unroll
  for (int t = 0; t < TOKENS; ++t)
#pragma unroll
    for (int j = 0; j < EXPERTS; ++j) {
#pragma unroll
      for (int off = 16; off >= 1; off >>= 1) acc[t][j] += __shfl_xor_sync(0xFFFFFFFFu, acc[t][j], off);
      if (lane == t * EXPERTS + j && tok0 + t < n_tokens && e0 + j < n_routed) {
        const __nv_bfloat16 r = __float2bfloat16_rn(acc[t][j]);
        logits[static_cast<size_t>(tok0 + t) * n_routed + e0 + j] = *reinterpret_cast<const uint16_t*>(&r);
      }
    }
}

// Qwen2-MoE's gated shared expert (aklr/plugins/sglang/models/qwen2_moe/reference.py:84-90): the
// routing table gets one more slot per token, expert ``shared_slot`` at weight
// sigmoid(x . shared_gate).  ``ids_in`` / ``weights_in`` [T, K] given: copied into the first K
// slots of the [T, K+1] tables; null: those slots are already in place.  One warp per token.
__global__ void __launch_bounds__(256)
shared_gate_kernel(const uint16_t* __restrict__ x, const uint16_t* __restrict__ gate, const int32_t* __restrict__ ids_in,
                   const float* __restrict__ weights_in, int32_t* __restrict__ ids, float* __restrict__ weights,
                   int n_tokens, int hidden, int topk, int shared_slot) {
  const int lane = threadIdx.x & 31;
  const int token = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (token >= n_tokens) return;
  float acc = 0.0f;
  for (int h = lane * 8; h < hidden; h += 256) {
    const uint4 xr = *reinterpret_cast<const uint4*>(x + static_cast<size_t>(token) * hidden + h);
    const uint4 gr = *reinterpret_cast<const uint4*>(gate + h);
    const uint32_t xw[4] = {xr.x, xr.y, xr.z, xr.w}, gw[4] = {gr.x, gr.y, gr.z, gr.w};
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      acc = fmaf(__uint_as_float(xw[q] << 16), __uint_as_float(gw[q] << 16), acc);
      acc = fmaf(__uint_as_float(xw[q] & 0xFFFF0000u), __uint_as_float(gw[q] & 0xFFFF0000u), acc);
    }
  }
#pragma unroll
  for (int off = 16; off >= 1; off >>= 1) acc += __shfl_xor_sync(0xFFFFFFFFu, acc, off);
  const size_t row = static_cast<size_t>(token) * (topk + 1);
  if (ids_in && lane < topk) {
    ids[row + lane] = ids_in[static_cast<size_t>(token) * topk + lane];
    weights[row + lane] = weights_in[static_cast<size_t>(token) * topk + lane];
  }
  if (lane == 0) {
    ids[row + topk] = shared_slot;
    weights[row + topk] = __fdiv_rn(1.0f, 1.0f + expf(-acc));
  }
}

int launch_shared_gate(const void* x, const void* gate, const int32_t* ids_in, const float* weights_in, int32_t* ids,
                       float* weights, int n_tokens, int hidden, int topk, int shared_slot, cudaStream_t stream) {
  if (hidden % 8 != 0 || topk < 1 || topk > 31) return AKLR_ERR_UNSUPPORTED_SHAPE;
  if (n_tokens == 0) return AKLR_OK;
  shared_gate_kernel<<<(n_tokens + 7) / 8, 256, 0, stream>>>(static_cast<const uint16_t*>(x), static_cast<const uint16_t*>(gate),
                                                          ids_in, weights_in, ids, weights, n_tokens, hidden, topk, shared_slot);
  return cudaGetLastError() == cudaSuccess ? AKLR_OK : AKLR_ERR_CUDA;
}

// A shared expert kept apart from the routed ones in bf16 (qwen2_moe_mxfp4_moe,
// aklr/plugins/sglang/models/qwen2_moe/reference.py:160-185): its two projections are dense bf16
// GEMMs the caller runs; these are the two steps around them.
//  * silu_mul: h[t, i] = bf16( silu(gate_up[t, i]) * gate_up[t, I + i] ), 8 values per thread;
//  * add_gated_rows: out[t] = bf16( out[t] + sigmoid(x[t] . gate) * rows[t] ), one warp per token.
__global__ void __launch_bounds__(256)
silu_mul_bf16_kernel(const uint16_t* __restrict__ gate_up, uint16_t* __restrict__ out, int64_t n_vectors, int vec_per_row) {
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n_vectors; i += stride) {
    const int64_t row = static_cast<uint32_t>(i) / static_cast<uint32_t>(vec_per_row);  // n_vectors < 2^31: checked at launch
    const int64_t v = i - row * vec_per_row;
    const uint4 g = *reinterpret_cast<const uint4*>(gate_up + (row * 2 * vec_per_row + v) * 8);
    const uint4 u = *reinterpret_cast<const uint4*>(gate_up + (row * 2 * vec_per_row + vec_per_row + v) * 8);
    const uint32_t gw[4] = {g.x, g.y, g.z, g.w}, uw[4] = {u.x, u.y, u.z, u.w};
    uint32_t r[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const float g0 = __uint_as_float(gw[q] << 16), g1 = __uint_as_float(gw[q] & 0xFFFF0000u);
      const float u0 = __uint_as_float(uw[q] << 16), u1 = __uint_as_float(uw[q] & 0xFFFF0000u);
      const __nv_bfloat162 pair = __floats2bfloat162_rn(__fdiv_rn(g0, 1.0f + expf(-g0)) * u0, __fdiv_rn(g1, 1.0f + expf(-g1)) * u1);
      r[q] = *reinterpret_cast<const uint32_t*>(&pair);
    }
    *reinterpret_cast<uint4*>(out + i * 8) = make_uint4(r[0], r[1], r[2], r[3]);
  }
}

__global__ void __launch_bounds__(256)
add_gated_rows_kernel(const uint16_t* __restrict__ x, const uint16_t* __restrict__ gate, const uint16_t* __restrict__ rows,
                      uint16_t* __restrict__ out, int n_tokens, int hidden) {
  const int lane = threadIdx.x & 31;
  const int token = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (token >= n_tokens) return;
  const size_t base = static_cast<size_t>(token) * hidden;
  float acc = 0.0f;
  for (int h = lane * 8; h < hidden; h += 256) {
    const uint4 xr = *reinterpret_cast<const uint4*>(x + base + h);
    const uint4 gr = *reinterpret_cast<const uint4*>(gate + h);
    const uint32_t xw[4] = {xr.x, xr.y, xr.z, xr.w}, gw[4] = {gr.x, gr.y, gr.z, gr.w};
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      acc = fmaf(__uint_as_float(xw[q] << 16), __uint_as_float(gw[q] << 16), acc);
      acc = fmaf(__uint_as_float(xw[q] & 0xFFFF0000u), __uint_as_float(gw[q] & 0xFFFF0000u), acc);
    }
  }
#pragma unroll
  for (int off = 16; off >= 1; off >>= 1) acc += __shfl_xor_sync(0xFFFFFFFFu, acc, off);
  const float weight = __fdiv_rn(1.0f, 1.0f + expf(-acc));
  for (int h = lane * 8; h < hidden; h += 256) {
    const uint4 rr = *reinterpret_cast<const uint4*>(rows + base + h);
    const uint4 orr = *reinterpret_cast<const uint4*>(out + base + h);
    const uint32_t rw[4] = {rr.x, rr.y, rr.z, rr.w}, ow[4] = {orr.x, orr.y, orr.z, orr.w};
    uint32_t res[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const float lo = fmaf(weight, __uint_as_float(rw[q] << 16), __uint_as_float(ow[q] << 16));
      const float hi = fmaf(weight, __uint_as_float(rw[q] & 0xFFFF0000u), __uint_as_float(ow[q] & 0xFFFF0000u));
      const __nv_bfloat162 pair = __floats2bfloat162_rn(lo, hi);
      res[q] = *reinterpret_cast<const uint32_t*>(&pair);
    }
    *reinterpret_cast<uint4*>(out + base + h) = make_uint4(res[0], res[1], res[2], res[3]);
  }
}

int launch_silu_mul_bf16(const void* gate_up, void* out, int n_tokens, int inter, cudaStream_t stream) {
  if (inter % 8 != 0 || inter < 8) return AKLR_ERR_UNSUPPORTED_SHAPE;
  if (n_tokens == 0) return AKLR_OK;
  const int vec_per_row = inter / 8;
  const int64_t n_vectors = static_cast<int64_t>(n_tokens) * vec_per_row;
  if (n_vectors >= (int64_t{1} << 31)) return AKLR_ERR_TOO_LARGE;
  const int grid = static_cast<int>(std::min<int64_t>((n_vectors + 255) / 256, 148 * 8));
  silu_mul_bf16_kernel<<<grid, 256, 0, stream>>>(static_cast<const uint16_t*>(gate_up), static_cast<uint16_t*>(out), n_vectors, vec_per_row);
  return cudaGetLastError() == cudaSuccess ? AKLR_OK : AKLR_ERR_CUDA;
}

int launch_add_gated_rows(const void* x, const void* gate, const void* rows, void* out, int n_tokens, int hidden,
                          cudaStream_t stream) {
  if (hidden % 8 != 0) return AKLR_ERR_UNSUPPORTED_SHAPE;
  if (n_tokens == 0) return AKLR_OK;
  add_gated_rows_kernel<<<(n_tokens + 7) / 8, 256, 0, stream>>>(static_cast<const uint16_t*>(x), static_cast<const uint16_t*>(gate),
                                                             static_cast<const uint16_t*>(rows), static_cast<uint16_t*>(out), n_tokens, hidden);
  return cudaGetLastError() == cudaSuccess ? AKLR_OK : AKLR_ERR_CUDA;
}

// Router with float32 weights and float32 logits (MiniMax-M2's gate:
// aklr/plugins/sglang/models/minimax_m2/reference.py:43-50 takes x @ router^T in float32, nothing
// rounded).  CUDA cores, float32 FMAs in k order.
//  * few tokens: one warp per (token, expert) dot product, so the weight is read by many SMs;
//  * else the tensor cores (router_gemm.cu); this file keeps a 64 x 64 tile per CTA, 16 k per step, 4 x 4 outputs per
//    thread, for token rows a TMA load cannot start at and logits that 16-byte stores cannot (off a 16-byte boundary).
template <int UNROLL>  // strides whose loads are in flight together (see router_gemm_kernel)
__global__ void __launch_bounds__(256)
router_dot_f32_kernel(const uint16_t* __restrict__ x, const float* __restrict__ w, float* __restrict__ logits,
                      int n_tokens, int hidden, int n_routed) {
  const int lane = threadIdx.x & 31;
  const int64_t item = static_cast<int64_t>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5);
  griddep_wait();
  griddep_launch();
  if (item >= static_cast<int64_t>(n_tokens) * n_routed) return;
  const int token = static_cast<int>(item / n_routed), e = static_cast<int>(item - static_cast<int64_t>(token) * n_routed);
  float acc = 0.0f;
  for (int h0 = lane * 4; h0 < hidden; h0 += 128 * UNROLL) {
    uint2 xr[UNROLL];
    float4 wr[UNROLL];
#pragma unroll
    for (int u = 0; u < UNROLL; ++u)
      if (h0 + u * 128 < hidden) {
        wr[u] = __ldg(reinterpret_cast<const float4*>(w + static_cast<size_t>(e) * hidden + h0 + u * 128));
        xr[u] = *reinterpret_cast<const uint2*>(x + static_cast<size_t>(token) * hidden + h0 + u * 128);
      }
#pragma unroll
    for (int u = 0; u < UNROLL; ++u)
      if (h0 + u * 128 < hidden) {
        acc = fmaf(__uint_as_float(xr[u].x << 16), wr[u].x, acc);
        acc = fmaf(__uint_as_float(xr[u].x & 0xFFFF0000u), wr[u].y, acc);
        acc = fmaf(__uint_as_float(xr[u].y << 16), wr[u].z, acc);
        acc = fmaf(__uint_as_float(xr[u].y & 0xFFFF0000u), wr[u].w, acc);
      }
  }
#pragma unroll
  for (int off = 16; off >= 1; off >>= 1) acc += __shfl_xor_sync(0xFFFFFFFFu, acc, off);
  if (lane == 0) logits[static_cast<size_t>(token) * n_routed + e] = acc;
}

__global__ void __launch_bounds__(256)
router_tile_f32_kernel(const uint16_t* __restrict__ x, const float* __restrict__ w, float* __restrict__ logits,
                       int n_tokens, int hidden, int n_routed) {
  constexpr int BM = 64, BN = 64, BK = 16;
  __shared__ float xs[BK][BM + 4];
  __shared__ float ws[BK][BN + 4];
  const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
  const int token0 = blockIdx.x * BM, e0 = blockIdx.y * BN;
  const int lrow = tid >> 2, lk = (tid & 3) * 4;  // this thread stages 4 k of one row of each tile
  float acc[4][4] = {};
  griddep_wait();
  griddep_launch();
  for (int k0 = 0; k0 < hidden; k0 += BK) {
    uint2 xr = make_uint2(0u, 0u);
    float4 wr = make_float4(0.f, 0.f, 0.f, 0.f);
    if (token0 + lrow < n_tokens) xr = *reinterpret_cast<const uint2*>(x + static_cast<size_t>(token0 + lrow) * hidden + k0 + lk);
    if (e0 + lrow < n_routed) wr = *reinterpret_cast<const float4*>(w + static_cast<size_t>(e0 + lrow) * hidden + k0 + lk);
    __syncthreads();  // the previous step is done with the tiles
    xs[lk + 0][lrow] = __uint_as_float(xr.x << 16);
    xs[lk + 1][lrow] = __uint_as_float(xr.x & 0xFFFF0000u);
    xs[lk + 2][lrow] = __uint_as_float(xr.y << 16);
    xs[lk + 3][lrow] = __uint_as_float(xr.y & 0xFFFF0000u);
    ws[lk + 0][lrow] = wr.x;
    ws[lk + 1][lrow] = wr.y;
    ws[lk + 2][lrow] = wr.z;
    ws[lk + 3][lrow] = wr.w;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < BK; ++k) {
      const float4 a = *reinterpret_cast<const float4*>(&xs[k][ty * 4]);
      const float4 b = *reinterpret_cast<const float4*>(&ws[k][tx * 4]);
      const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int token = token0 + ty * 4 + i;
    if (token >= n_tokens) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int e = e0 + tx * 4 + j;
      if (e < n_routed) logits[static_cast<size_t>(token) * n_routed + e] = acc[i][j];
    }
  }
}

int launch_router_gemm_f32(const void* x, const float* w, float* logits, int n_tokens, int hidden, int n_routed,
                           cudaStream_t stream) {
  if (hidden % 128 != 0) return AKLR_ERR_UNSUPPORTED_SHAPE;
  if (n_tokens == 0 || n_routed == 0) return AKLR_OK;
  auto* xp = static_cast<const uint16_t*>(x);
  if (n_tokens <= 16) {
    const int64_t blocks = (static_cast<int64_t>(n_tokens) * n_routed + 7) / 8;
    // Eight strides in flight take 66 registers a thread, three CTAs per SM: from 512 CTAs on, more CTAs with four strides hide
    // as much (eight / four: 12 tokens on 7168 x 384 12.4 / 10.0 us, 16 on 3072 x 256 6.4 / 4.9; 8 on 7168 x 384 8.0 / 9.3).
    return launch_kernel(blocks < 512 ? router_dot_f32_kernel<8> : router_dot_f32_kernel<4>, dim3(static_cast<unsigned>(blocks)), dim3(256), 0, stream, 1, xp, w, logits, n_tokens,
                         hidden, n_routed) == cudaSuccess ? AKLR_OK : AKLR_ERR_CUDA;
  }
  const dim3 grid((n_tokens + 63) / 64, (n_routed + 63) / 64);
  return launch_kernel(router_tile_f32_kernel, grid, dim3(256), 0, stream, 1, xp, w, logits, n_tokens, hidden, n_routed) == cudaSuccess
             ? AKLR_OK : AKLR_ERR_CUDA;
}

int launch_router_gemm(const void* x, const void* w, void* logits, int n_tokens, int hidden, int n_routed,
                       cudaStream_t stream) {
  if (hidden % 8 != 0) return AKLR_ERR_UNSUPPORTED_SHAPE;
  if (n_tokens == 0) return AKLR_OK;
  auto* xp = static_cast<const uint16_t*>(x);
  auto* wp = static_cast<const uint16_t*>(w);
  auto* lp = static_cast<uint16_t*>(logits);
  auto run = [&](auto kernel, int tokens, int experts, int warps) {
    const int64_t items = static_cast<int64_t>((n_tokens + tokens - 1) / tokens) * ((n_routed + experts - 1) / experts);
    const int64_t blocks = (items + warps - 1) / warps;
    if (items > 0x7FFFFFFF - 32) return AKLR_ERR_TOO_LARGE;
    return launch_kernel(kernel, dim3(static_cast<unsigned>(blocks)), dim3(32 * warps), 0, stream, 1, xp, wp, lp, n_tokens, hidden,
                         n_routed) == cudaSuccess ? AKLR_OK : AKLR_ERR_CUDA;
  };
  // One token: one dot product per warp and two warps per CTA, so that the weight is read by every SM.  More tokens
  // reuse what a warp has loaded: at 17 tokens on 2048 x 512 2 x 4 products per warp read 27 MB from L2, 1 x 8 35 MB.
  if (n_tokens == 1) return run(router_gemm_kernel<1, 1, 8>, 1, 1, 2);
  if (n_tokens <= 16) return run(router_gemm_kernel<2, 2, 4>, 2, 2, 4);
  return run(router_gemm_kernel<2, 4, 2>, 2, 4, 8);
}

}  // namespace aklr
