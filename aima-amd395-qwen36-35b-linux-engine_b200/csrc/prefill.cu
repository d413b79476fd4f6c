// Prefill MoE half-layer on the GPU: router + top-8, dispatch plan, gather,
// grouped expert products, shared expert, weighted combine.
//
// Stage list and rounding points follow the reference orchestration
// (native/src/native_moe_prefill.hip.cpp:790-893):
//   router GEMM -> BF16 logits -> router_topk8_softmax_256_kernel (:234-323)
//   moe_align_block32_256_kernel (:325-382)            -> here: a deterministic
//       counting sort into a per-expert offset table (no padding rows)
//   fused_moe_kernel gate_up -> expert_silu_multiply_kernel (:384-402)
//   fused_moe_kernel down (x routing weight)           -> moe_sum8_kernel (:404-431)
//   shared expert (:210-232, 790-826), bf16_add_pair_kernel
//   (native/src/native_pointwise.hip.cpp:94-107)
#include "prefill.cuh"

#include "grouped_gemm.cuh"

#include <cstdio>
#include <math_constants.h>

namespace aima {
namespace {

// Monotone map FP32 -> uint32 (larger float <=> larger key), for redux-based maxima.
__device__ __forceinline__ uint32_t order_key(float f) {
  const uint32_t u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float key_value(uint32_t k) {
  return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}

// 8th largest of the 256 values a warp holds (8 per lane), counting repeats.  Every lane sorts its eight keys once
// (Batcher's odd-even merge network), so that a round is one warp maximum and a shift on the lane that held it.
__device__ __forceinline__ float warp_eighth_largest(const float* v, int lane) {
  uint32_t k[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) k[q] = order_key(v[q]);
  constexpr int kPairs[19][2] = {{0, 1}, {2, 3}, {4, 5}, {6, 7}, {0, 2}, {1, 3}, {4, 6}, {5, 7}, {1, 2}, {5, 6},
                                 {0, 4}, {1, 5}, {2, 6}, {3, 7}, {2, 4}, {3, 5}, {1, 2}, {3, 4}, {5, 6}};
#pragma unroll
  for (int p = 0; p < 19; ++p) {
    const uint32_t hi = max(k[kPairs[p][0]], k[kPairs[p][1]]);
    k[kPairs[p][1]] = min(k[kPairs[p][0]], k[kPairs[p][1]]);
    k[kPairs[p][0]] = hi;
  }
  uint32_t best = 0;
#pragma unroll
  for (int r = 0; r < kTopK; ++r) {
    best = __reduce_max_sync(0xffffffffu, k[0]);
    const unsigned owners = __ballot_sync(0xffffffffu, k[0] == best);
    if (lane == __ffs(owners) - 1) {
#pragma unroll
      for (int q = 0; q < 7; ++q) k[q] = k[q + 1];
      k[7] = 0u;
    }
  }
  return key_value(best);
}

// Where a value goes among the eight selected: the values above the threshold in lane order of this call, behind the
// `held` ones taken before.  Returns how many are held then.
__device__ __forceinline__ int take_values(bool take, float value, int expert, int held, int lane, float* sel_v, int* sel_i) {
  const unsigned m = __ballot_sync(0xffffffffu, take);
  const int pos = held + __popc(m & ((1u << lane) - 1u));
  if (take && pos < kTopK) {
    sel_v[pos] = value;
    sel_i[pos] = expert;
  }
  return held + __popc(m);
}

// Second half of the reference's prefill selection: lane r < 8 holds the r-th gathered value and its expert.  Fixed bitonic
// network of width 8 (a pair is exchanged when (value[left] > value[right]) equals the "ascending" flag of the left index),
// softmax summed in slot order; lane r writes slot r and returns its expert.
__device__ __forceinline__ int finish_route(float v, int expert, int lane, size_t token, int32_t* __restrict__ ids,
                                            float* __restrict__ scores, float* __restrict__ weights,
                                            __nv_bfloat16* __restrict__ dbg_weights) {
#pragma unroll
  for (int width = 2; width <= kTopK; width *= 2) {
#pragma unroll
    for (int stride = width / 2; stride > 0; stride /= 2) {
      const float other = __shfl_xor_sync(0xffffffffu, v, stride);
      const int other_expert = __shfl_xor_sync(0xffffffffu, expert, stride);
      const bool is_left = (lane & stride) == 0;
      const bool ascending = (lane & width) != 0;      // the same in both lanes of a pair
      if (((is_left ? v : other) > (is_left ? other : v)) == ascending) {
        v = other;
        expert = other_expert;
      }
    }
  }
  const float ex = det_expf(__fsub_rn(v, __shfl_sync(0xffffffffu, v, 0)));
  float denom = 0.0f;
#pragma unroll
  for (int r = 0; r < kTopK; ++r) denom = __fadd_rn(denom, __shfl_sync(0xffffffffu, ex, r));
  if (lane < kTopK) {
    const size_t o = token * kTopK + lane;
    const uint16_t wb = float_to_bf16_bits(__fdiv_rn(ex, denom));
    ids[o] = expert;
    scores[o] = v;
    weights[o] = bf16_bits_to_float(wb);
    if (dbg_weights != nullptr) reinterpret_cast<uint16_t*>(dbg_weights)[o] = wb;
  }
  return lane < kTopK ? expert : -1;
}

// The reference's prefill selection on the final (BF16-rounded) logits of one
// token held as v[q] = logit of expert 32 q + lane: threshold, gather in expert
// order, then finish_route.  `threshold` is the 8th largest of the values, none
// of which may be a NaN (selectable): then at least eight of them reach it and every slot is written.
__device__ __forceinline__ int route_token(const float* v, float threshold, int lane, float* sel_v, int* sel_i,
                                            size_t token, int32_t* __restrict__ ids,
                                            float* __restrict__ scores, float* __restrict__ weights,
                                            __nv_bfloat16* __restrict__ dbg_weights) {
  int held = 0;
#pragma unroll
  for (int q = 0; q < 8; ++q) held = take_values(v[q] > threshold, v[q], 32 * q + lane, held, lane, sel_v, sel_i);
#pragma unroll
  for (int q = 0; q < 8; ++q) held = take_values(v[q] == threshold, v[q], 32 * q + lane, held, lane, sel_v, sel_i);
  __syncwarp();
  const float chosen = sel_v[lane & (kTopK - 1)];
  const int expert = sel_i[lane & (kTopK - 1)];
  __syncwarp();
  return finish_route(chosen, expert, lane, token, ids, scores, weights, dbg_weights);
}

// logit transform shared by the router kernels: optional harness hooks, then
// the BF16 rounding the reference's router GEMM applies
__device__ __forceinline__ float finish_logit(float x, float bias, int quant_eighths) {
  x = __fadd_rn(x, bias);
  if (quant_eighths) x = __fmul_rn(rintf(__fmul_rn(x, 8.0f)), 0.125f);
  return round_bf16(x);
}

// What the selection sees of a logit.  A NaN compares false with every threshold, so route_token would leave slots
// unwritten and the plan would lose rows; counted as -inf it loses to every number, and a token with fewer than eight
// numbers still gets eight valid experts (the lowest ids among the rest).
__device__ __forceinline__ float selectable(float logit) { return logit == logit ? logit : -CUDART_INF_F; }

// ---------------------------------------------------------------------------
// Router: canonical FP32 logits of all 256 experts (+ the shared-expert gate
// row), BF16 rounding, the reference's selection rule and softmax.
// One warp per token, 16 tokens per block; router rows are staged through
// shared memory 32 at a time.
// ---------------------------------------------------------------------------
constexpr int kRouterWarps = 16;
constexpr int kRouterChunkRows = 32;
constexpr int kRouterSmemBytes = kRouterChunkRows * kHidden * 2 + kRouterWarps * 8 * 8;

__global__ void __launch_bounds__(kRouterWarps * 32, 1)
prefill_router_kernel(const __nv_bfloat16* __restrict__ h2,
                      const __nv_bfloat16* __restrict__ router,
                      const __nv_bfloat16* __restrict__ shared_gate,
                      const float* __restrict__ bias, int quant_eighths, int tokens,
                      int32_t* __restrict__ ids, float* __restrict__ scores,
                      float* __restrict__ weights, float* __restrict__ shared_sigmoid,
                      float* __restrict__ dbg_logits, __nv_bfloat16* __restrict__ dbg_weights) {
  extern __shared__ __align__(16) uint8_t smem[];
  uint4* rows_s = reinterpret_cast<uint4*>(smem);
  float* sel_v_s = reinterpret_cast<float*>(smem + kRouterChunkRows * kHidden * 2);
  int* sel_i_s = reinterpret_cast<int*>(sel_v_s + kRouterWarps * 8);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int token = blockIdx.x * kRouterWarps + warp;
  const bool valid = token < tokens;

  float xr[64];
#pragma unroll
  for (int g = 0; g < 8; ++g) {
    uint4 v = make_uint4(0, 0, 0, 0);
    if (valid) v = *(reinterpret_cast<const uint4*>(h2 + static_cast<size_t>(token) * kHidden) + g * 32 + lane);
    unpack8(v, xr + 8 * g);
  }

  float v[8];   // lane l holds the logit of expert 32 q + l in v[q]
  float gate_dot = 0.0f;
#pragma unroll
  for (int chunk = 0; chunk < 9; ++chunk) {
    const int n_rows = (chunk < 8) ? kRouterChunkRows : 1;
    const __nv_bfloat16* src = (chunk < 8) ? router + static_cast<size_t>(chunk) * kRouterChunkRows * kHidden
                                           : shared_gate;
    __syncthreads();
    for (int i = threadIdx.x; i < n_rows * (kHidden / 8); i += blockDim.x) {
      rows_s[i] = __ldg(reinterpret_cast<const uint4*>(src) + i);
    }
    __syncthreads();
    if (chunk < 8) {
      float mine = 0.0f;
      for (int r = 0; r < kRouterChunkRows; r += 2) {
        const uint4* r0 = rows_s + r * (kHidden / 8) + lane;
        const uint4* r1 = r0 + (kHidden / 8);
        float a = 0.0f, b = 0.0f;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          a = fma8(xr + 8 * i, r0[i * 32], a);
          b = fma8(xr + 8 * i, r1[i * 32], b);
        }
        a = butterfly_sum(a);
        b = butterfly_sum(b);
        if (lane == r) mine = a;
        if (lane == r + 1) mine = b;
      }
      v[chunk] = mine;
    } else {
      const uint4* r0 = rows_s + lane;
      float a = 0.0f;
#pragma unroll
      for (int i = 0; i < 8; ++i) a = fma8(xr + 8 * i, r0[i * 32], a);
      gate_dot = butterfly_sum(a);
    }
  }
  if (!valid) return;

  // harness hooks, then the BF16 rounding the reference's router GEMM applies
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    v[q] = finish_logit(v[q], bias != nullptr ? bias[32 * q + lane] : 0.0f, quant_eighths);
    if (dbg_logits != nullptr) dbg_logits[static_cast<size_t>(token) * kExperts + 32 * q + lane] = v[q];
    v[q] = selectable(v[q]);
  }
  route_token(v, warp_eighth_largest(v, lane), lane, sel_v_s + warp * 8, sel_i_s + warp * 8, static_cast<size_t>(token),
              ids, scores, weights, dbg_weights);
  if (lane == 0) {
    shared_sigmoid[token] = round_bf16(det_sigmoid(round_bf16(gate_dot)));
  }
}

// ---------------------------------------------------------------------------
// Certified router.  All 256 logits come from the tensor cores first (FP32,
// unknown accumulation order, `approx`).  Their distance to the canonical value
// is bounded by kappa * |x|_2 * |w_e|_2 (Cauchy-Schwarz on the FP32 rounding
// error of a 2048-term sum, in the spirit of the reference's certified LM head,
// native/src/native_lm_head_certificate.hip.cpp:33-39).  Only experts whose
// upper bound reaches the lower bound of the 8th-largest value can be selected;
// those few are recomputed with the canonical dot and the reference's rule runs
// on them alone, so ids, scores and weights stay bit-exact.
//
// The bound is a statement about hardware whose accumulation order is not
// published, so the kernel checks it where it can: every candidate has both
// values, and if one lies further from its tensor-core value than the bound
// allows, the whole token is recomputed with the canonical dot (all 256
// experts) and counted.  With audit_stride > 0 every audit_stride-th token is
// recomputed in full as well and its ids compared with the certified ones.
// kWays warps share a token's dots: a call whose tokens would leave the chip half empty with one warp each is bound by
// the latency of one token, which two or four warps cut.  At 8192 tokens the kernel takes 42 us (57 with candidates filed by
// expert, the selection run by every lane and the statistics added per token), at 333 8 us (14).
// ---------------------------------------------------------------------------
constexpr int kCertWarps = 8;
constexpr int kCertBlocksPerSm = 2;
constexpr float kCertKappa = 6.103515625e-05f;   // 2^-14, ~4x the summed worst-case rounding terms

// canonical 8-element step of the warp dot with BOTH operands still packed (same FMA order as fma8)
__device__ __forceinline__ float fma8_packed(const uint4& x, const uint4& w, float acc) {
  acc = __fmaf_rn(bf16_lo(x.x), bf16_lo(w.x), acc);
  acc = __fmaf_rn(bf16_hi(x.x), bf16_hi(w.x), acc);
  acc = __fmaf_rn(bf16_lo(x.y), bf16_lo(w.y), acc);
  acc = __fmaf_rn(bf16_hi(x.y), bf16_hi(w.y), acc);
  acc = __fmaf_rn(bf16_lo(x.z), bf16_lo(w.z), acc);
  acc = __fmaf_rn(bf16_hi(x.z), bf16_hi(w.z), acc);
  acc = __fmaf_rn(bf16_lo(x.w), bf16_lo(w.w), acc);
  acc = __fmaf_rn(bf16_hi(x.w), bf16_hi(w.w), acc);
  return acc;
}

// Tensor-core logits of one call: `splits` partial sums over K, each [tokens, 256], added in this order.  (The additions are
// part of the distance the bound covers: three more roundings beside the 128 of the accumulator.)
struct ApproxLogits {
  const float* partial;
  size_t stride;
  int splits;
};

// The token's row stays packed in registers, and the candidates are recomputed two at a time: a pair shares the unpacking
// of the row, and two router rows are on their way from L2 at once.  A lane keeps one candidate from then on, so that the
// check of the bound, the selection and the softmax are one pass of the warp each.
template <int kWays>
__global__ void __launch_bounds__(kCertWarps * 32, kCertBlocksPerSm)
prefill_router_certified_kernel(const __nv_bfloat16* __restrict__ h2,
                                const __nv_bfloat16* __restrict__ router,
                                const __nv_bfloat16* __restrict__ shared_gate,
                                const ApproxLogits approx,
                                const float* __restrict__ row_norms,
                                const float* __restrict__ bias, int quant_eighths, int tokens,
                                int32_t* __restrict__ ids, float* __restrict__ scores,
                                float* __restrict__ weights, float* __restrict__ shared_sigmoid,
                                __nv_bfloat16* __restrict__ dbg_weights, unsigned long long* __restrict__ stats,
                                int audit_stride, uint8_t* __restrict__ chunk_counts) {
  constexpr int kTokens = kCertWarps / kWays;
  __shared__ float exact_s[kTokens][kExperts];           // canonical dot of candidate c
  __shared__ float approx_s[kTokens][kExperts];          // tensor-core logit of expert e
  __shared__ float bound_s[kTokens][kExperts];           // and how far from it the canonical one may lie
  __shared__ uint8_t list_s[kCertWarps][kExperts];       // expert of candidate c
  __shared__ float gate_s[kTokens];
  __shared__ float sel_v_s[kTokens * kTopK];
  __shared__ int sel_i_s[kTokens * kTopK];
  __shared__ int histogram[kExperts];
  __shared__ int tally[5];
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int slot = warp / kWays;
  const int part = warp % kWays;
  const int token = blockIdx.x * kTokens + slot;
  const bool valid = token < tokens;
  histogram[threadIdx.x] = 0;
  if (threadIdx.x < 5) tally[threadIdx.x] = 0;
  __syncthreads();
  pdl_enter();

  uint4 xp[8];
  int n = 0;                        // candidates
  uint8_t* list = list_s[warp];
  // Canonical dots of the rows row_of(from), row_of(from + 1), row_of(from + step), row_of(from + step + 1), ... up to
  // row_of(last): two rows at a time share the unpacking of the token's row.  Bound by the rows coming from L2 (302 MB at
  // 8192 tokens); fetching the next half of a pair ahead costs registers that the rest of the kernel needs (43 -> 42 us
  // without it).
  auto walk = [&](int from, int step, int last, auto row_of, auto sink) {
    if (from > last) return;
    uint4 w[2][4];
    auto fetch = [&](int c, int half) {
      const uint4* row0 = reinterpret_cast<const uint4*>(row_of(c)) + lane + 128 * half;
      const uint4* row1 = reinterpret_cast<const uint4*>(row_of(c + 1)) + lane + 128 * half;
#pragma unroll
      for (int i = 0; i < 4; ++i) w[0][i] = __ldg(row0 + 32 * i);
#pragma unroll
      for (int i = 0; i < 4; ++i) w[1][i] = __ldg(row1 + 32 * i);
    };
#pragma unroll 1
    for (int c = from; c <= last; c += step) {
      fetch(c, 0);
      float acc0 = 0.0f, acc1 = 0.0f;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        acc0 = fma8_packed(xp[i], w[0][i], acc0);
        acc1 = fma8_packed(xp[i], w[1][i], acc1);
      }
      fetch(c, 1);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        acc0 = fma8_packed(xp[4 + i], w[0][i], acc0);
        acc1 = fma8_packed(xp[4 + i], w[1][i], acc1);
      }
      sink(c, butterfly_sum(acc0), butterfly_sum(acc1));
    }
  };
  if (valid) {
    float sumsq = 0.0f;
    float a[8];
#pragma unroll
    for (int g = 0; g < 8; ++g)
      xp[g] = *(reinterpret_cast<const uint4*>(h2 + static_cast<size_t>(token) * kHidden) + g * 32 + lane);
    const float* logits = approx.partial + static_cast<size_t>(token) * kExperts + lane;
#pragma unroll
    for (int q = 0; q < 8; ++q) a[q] = logits[32 * q];
#pragma unroll
    for (int g = 0; g < 8; ++g) {
      float x8[8];
      unpack8(xp[g], x8);
#pragma unroll
      for (int j = 0; j < 8; ++j) sumsq = fmaf(x8[j], x8[j], sumsq);
    }
    for (int split = 1; split < approx.splits; ++split) {      // eight loads at a time: one by one each waits for L2
      logits += approx.stride;
      float more[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) more[q] = logits[32 * q];
#pragma unroll
      for (int q = 0; q < 8; ++q) a[q] = __fadd_rn(a[q], more[q]);
    }
    float upper[8], lower[8], norm[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) norm[q] = __ldg(row_norms + 32 * q + lane);
    sumsq = butterfly_sum(sumsq);
    const float x_norm = sqrtf(sumsq) * 1.0001f;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int e = 32 * q + lane;
      const float b = bias != nullptr ? bias[e] : 0.0f;
      const float delta = kCertKappa * x_norm * norm[q] + 9.5367431640625e-07f * fabsf(a[q] + b);
      if (part == 0) {
        approx_s[slot][e] = a[q];
        bound_s[slot][e] = delta;
      }
      upper[q] = finish_logit(a[q] + delta, b, quant_eighths);
      lower[q] = selectable(finish_logit(a[q] - delta, b, quant_eighths));      // a NaN bounds nothing from below
    }
    const float floor_value = warp_eighth_largest(lower, lane);
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const bool take = upper[q] >= floor_value;
      const unsigned m = __ballot_sync(0xffffffffu, take);
      if (take) list[n + __popc(m & ((1u << lane) - 1u))] = static_cast<uint8_t>(32 * q + lane);
      n += __popc(m);
    }
    __syncwarp();
    // candidate n stands for the shared expert's gate row
    walk(2 * part, 2 * kWays, n, [&](int c) { return c < n ? router + static_cast<size_t>(list[c]) * kHidden : shared_gate; },
         [&](int c, float acc0, float acc1) {
           if (lane == 0) {
             if (c < n) exact_s[slot][c] = acc0;
             else gate_s[slot] = acc0;
             if (c + 1 < n) exact_s[slot][c + 1] = acc1;
             else if (c + 1 == n) gate_s[slot] = acc1;
           }
         });
  }
  if (kWays == 1) __syncwarp();
  else __syncthreads();

  if (valid && part == 0) {
    const float* exact = exact_s[slot];
    float* sel_v = sel_v_s + slot * kTopK;
    int* sel_i = sel_i_s + slot * kTopK;
    const size_t row = static_cast<size_t>(token);
    auto bias_of = [&](int e) { return bias != nullptr ? __ldg(bias + e) : 0.0f; };
    // is a canonical value further from the tensor-core value than the bound the filter relied on?
    bool violated = false;
    for (int c = lane; c < n; c += 32) violated = violated || fabsf(exact[c] - approx_s[slot][list[c]]) > bound_s[slot][list[c]];
    violated = __any_sync(0xffffffffu, violated);

    int chosen = -1;
    bool routed = false;
    if (n >= kTopK && n <= 32 && !violated) {
      // (nearly always) candidate c on lane c, in expert order; of exactly eight all are selected and the threshold is
      // their smallest.  A threshold at or below -inf in the order of the keys leaves room for other experts: general rule.
      const bool mine = lane < n;
      const int e = mine ? list[lane] : 0;
      const float v = mine ? selectable(finish_logit(exact[lane], bias_of(e), quant_eighths)) : 0.0f;
      const uint32_t key = mine ? order_key(v) : 0u;
      uint32_t eighth = 0u;
      if (n == kTopK) {
        eighth = __reduce_min_sync(0xffffffffu, mine ? key : 0xffffffffu);
      } else {
        uint32_t left = key;
#pragma unroll 1
        for (int r = 0; r < kTopK; ++r) {
          eighth = __reduce_max_sync(0xffffffffu, left);
          const unsigned owners = __ballot_sync(0xffffffffu, left == eighth);
          if (lane == __ffs(owners) - 1) left = 0u;
        }
      }
      if (eighth > order_key(-CUDART_INF_F)) {
        const float threshold = key_value(eighth);
        const int held = take_values(mine && v > threshold, v, e, 0, lane, sel_v, sel_i);
        take_values(mine && v == threshold, v, e, held, lane, sel_v, sel_i);
        __syncwarp();
        chosen = finish_route(sel_v[lane & (kTopK - 1)], sel_i[lane & (kTopK - 1)], lane, row, ids, scores, weights, dbg_weights);
        routed = true;
        __syncwarp();
      }
    }
    float v[8];
    auto file = [&](int e, float acc) {       // the owner lane keeps the final logit of expert e
      const float f = selectable(finish_logit(acc, bias_of(e), quant_eighths));
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        if (e == 32 * q + lane) v[q] = f;
      }
    };
    auto general = [&]() {
      return route_token(v, warp_eighth_largest(v, lane), lane, sel_v, sel_i, row, ids, scores, weights, dbg_weights);
    };
    if (!routed && !violated) {
#pragma unroll
      for (int q = 0; q < 8; ++q) v[q] = -CUDART_INF_F;
#pragma unroll 1
      for (int c = 0; c < n; ++c) file(list[c], exact[c]);
      chosen = general();
    }
    // a token whose filter's premise failed takes nothing from it; an audited one is routed both ways
    const bool audited = audit_stride > 0 && token % audit_stride == 0 && !violated;
    bool mismatch = false;
    if (violated || audited) {
      walk(0, 2, kExperts - 1, [&](int e) { return router + static_cast<size_t>(e) * kHidden; },
           [&](int e, float acc0, float acc1) {
             file(e, acc0);
             file(e + 1, acc1);
           });
      const int exact_id = general();
      mismatch = audited && __any_sync(0xffffffffu, lane < kTopK && exact_id != chosen);
      chosen = exact_id;
    }
    if (lane < kTopK) atomicAdd(&histogram[chosen], 1);
    if (lane == 0) {
      shared_sigmoid[token] = round_bf16(det_sigmoid(round_bf16(gate_s[slot])));
      atomicAdd(&tally[0], n);
      atomicAdd(&tally[1], 1);
      if (violated) atomicAdd(&tally[2], 1);
      if (audited) atomicAdd(&tally[3], 1);
      if (mismatch) atomicAdd(&tally[4], 1);
    }
  }
  __syncthreads();
  // rows of this block per expert, for the plan; the statistics once per block (8192 tokens adding to the same words in L2
  // one by one)
  if (chunk_counts != nullptr)
    chunk_counts[static_cast<size_t>(blockIdx.x) * kExperts + threadIdx.x] = static_cast<uint8_t>(histogram[threadIdx.x]);
  if (stats != nullptr && threadIdx.x < 5 && tally[threadIdx.x] != 0)
    atomicAdd(stats + threadIdx.x, static_cast<unsigned long long>(tally[threadIdx.x]));
}

// ---------------------------------------------------------------------------
// Router of a short call: all 256 canonical logits straight away, spread over the chip by EXPERT -- a block holds two
// router rows in registers and walks the tokens -- then one warp per token selects.  The tensor-core filter needs the
// whole router matrix in each 32-token tile and then a chain of dependent loads per token: 20 + 13 us at 16 tokens,
// whatever their number, against 17 us for both here, growing with the tokens.  us per layer, filter / all logits: balanced
// routing 126 / 118 at 16 tokens, 236 / 229 at 64, 264 / 261 at 128, 269 / 270 at 160, 272 / 278 at 256; Zipf 79 / 69, 98 / 92,
// 118 / 115, 128 / 127, 145 / 152; eight hot experts 43 / 35, 47 / 41, 53 / 50, 51 / 51, 57 / 63.  They cross at 160 tokens.
// ---------------------------------------------------------------------------
constexpr int kSmallRouterTokens = 128;

__global__ void __launch_bounds__(256, 1)
prefill_logits_small_kernel(const __nv_bfloat16* __restrict__ h2, const __nv_bfloat16* __restrict__ router,
                            const __nv_bfloat16* __restrict__ shared_gate, int tokens, float* __restrict__ logits,
                            float* __restrict__ shared_sigmoid) {
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const bool gate = blockIdx.x == kExperts / 2;              // the last block: the shared expert's gate row
  pdl_enter();
  const uint4* row0 = reinterpret_cast<const uint4*>(gate ? shared_gate : router + static_cast<size_t>(2 * blockIdx.x) * kHidden) + lane;
  const uint4* row1 = gate ? row0 : row0 + kHidden / 8;
  auto token_row = [&](int t) { return reinterpret_cast<const uint4*>(h2 + static_cast<size_t>(t) * kHidden) + lane; };
  uint4 next[8];
  if (warp < tokens) {
#pragma unroll
    for (int i = 0; i < 8; ++i) next[i] = __ldg(token_row(warp) + i * 32);
  }
  float w0[64], w1[64];
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    unpack8(__ldg(row0 + i * 32), w0 + 8 * i);
    unpack8(__ldg(row1 + i * 32), w1 + 8 * i);
  }
  for (int t = warp; t < tokens; t += 8) {
    uint4 x[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) x[i] = next[i];
    if (t + 8 < tokens) {
#pragma unroll
      for (int i = 0; i < 8; ++i) next[i] = __ldg(token_row(t + 8) + i * 32);
    }
    float a = 0.0f, b = 0.0f;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      a = fma8(w0 + 8 * i, x[i], a);
      b = fma8(w1 + 8 * i, x[i], b);
    }
    a = butterfly_sum(a);
    b = butterfly_sum(b);
    if (lane == 0) {
      if (gate) shared_sigmoid[t] = round_bf16(det_sigmoid(round_bf16(a)));
      else *reinterpret_cast<float2*>(logits + static_cast<size_t>(t) * kExperts + 2 * blockIdx.x) = make_float2(a, b);
    }
  }
}

__global__ void __launch_bounds__(kCertWarps * 32)
prefill_select_kernel(const float* __restrict__ logits, const float* __restrict__ bias, int quant_eighths, int tokens,
                      int32_t* __restrict__ ids, float* __restrict__ scores, float* __restrict__ weights,
                      __nv_bfloat16* __restrict__ dbg_weights, uint8_t* __restrict__ chunk_counts) {
  __shared__ float sel_v_s[kCertWarps * 8];
  __shared__ int sel_i_s[kCertWarps * 8];
  __shared__ int histogram[kExperts];
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int token = blockIdx.x * kCertWarps + warp;
  histogram[threadIdx.x] = 0;
  __syncthreads();
  pdl_enter();
  if (token < tokens) {
    float v[8];
#pragma unroll
    for (int q = 0; q < 8; ++q)
      v[q] = selectable(finish_logit(logits[static_cast<size_t>(token) * kExperts + 32 * q + lane],
                                     bias != nullptr ? bias[32 * q + lane] : 0.0f, quant_eighths));
    const int chosen = route_token(v, warp_eighth_largest(v, lane), lane, sel_v_s + warp * 8, sel_i_s + warp * 8,
                                   static_cast<size_t>(token), ids, scores, weights, dbg_weights);
    if (lane < kTopK) atomicAdd(&histogram[chosen], 1);
  }
  __syncthreads();
  chunk_counts[static_cast<size_t>(blockIdx.x) * kExperts + threadIdx.x] = static_cast<uint8_t>(histogram[threadIdx.x]);
}

// Euclidean norms of the 256 router rows, rounded up a little; one warp per row.
__global__ void __launch_bounds__(256)
router_row_norms_kernel(const __nv_bfloat16* __restrict__ router, float* __restrict__ norms) {
  const int lane = threadIdx.x & 31;
  const int row = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (row >= kExperts) return;
  const uint4* src = reinterpret_cast<const uint4*>(router + static_cast<size_t>(row) * kHidden) + lane;
  float sum = 0.0f;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    float w[8];
    unpack8(__ldg(src + i * 32), w);
#pragma unroll
    for (int j = 0; j < 8; ++j) sum = fmaf(w[j], w[j], sum);
  }
  sum = butterfly_sum(sum);
  if (lane == 0) norms[row] = sqrtf(sum) * 1.0001f;
}

// ---------------------------------------------------------------------------
// Dispatch plan: stable counting sort of the 8T routed rows by expert, in one launch.
// ---------------------------------------------------------------------------
// Rows per tile of an expert with `count` rows.  128-row tiles (one-SM products) are filled one after the other.  Tiles
// of up to 256 rows (two-SM products, whose cost goes with the rows in steps of 32) are made equally large: 272 rows
// are 160 + 112, not 256 + 16, so that the last tile does not stream the expert's weights for a handful of rows.  All
// tiles but the last are full multiples of 32, and the last one is never empty (the tiles before it hold at most
// 256 (n - 1) < count rows).
__device__ __forceinline__ int rows_per_tile(int count, int n_tiles, int tile_cap) {
  if (tile_cap <= kTileRows || n_tiles <= 1) return tile_cap;
  return ((count + n_tiles - 1) / n_tiles + 31) & ~31;
}

// Chunks: runs of `chunk_rows` flat rows, and how many rows of each expert a chunk has (one byte each).  The routers leave
// the counts of their own blocks' tokens; count_rows_kernel makes them from the ids where those come from elsewhere (forced
// routing, the all-256 router, other GPUs).  Ids outside [expert_lo, expert_hi) are not in the plan.
constexpr int kCountRows = 64;

__global__ void __launch_bounds__(kExperts)
count_rows_kernel(const int32_t* __restrict__ ids, int routed_rows, int expert_lo, int expert_hi,
                  uint8_t* __restrict__ chunk_counts) {
  __shared__ int histogram[kExperts];
  histogram[threadIdx.x] = 0;
  __syncthreads();
  pdl_enter();
  const int row = blockIdx.x * kCountRows + threadIdx.x;
  if (threadIdx.x < kCountRows && row < routed_rows) {
    const int e = ids[row];
    if (e >= expert_lo && e < expert_hi) atomicAdd(&histogram[e], 1);
  }
  __syncthreads();
  chunk_counts[static_cast<size_t>(blockIdx.x) * kExperts + threadIdx.x] = static_cast<uint8_t>(histogram[threadIdx.x]);
}

// A block owns a run of chunks.  It adds up the counts of the chunks before its own and of all chunks (every block reads the
// whole table, 256 KB at T = 8192, from L2), takes the prefix over the experts, and places its rows: a row's position is its
// expert's offset, the rows of that expert in the chunks before, and its rank in the block, from a bit per row and expert in
// shared memory.  No block waits for another.  Block 0 also publishes the counts, the offsets, the tile list and the
// reference's block-32 padded row count.  Bound by latency: alone 11 us at T = 8192 and 8 at 2048, 8 at 8192 in the running
// layer; one cluster of eight blocks that counted the ids itself took 24 alone at 8192.
constexpr int kPlanThreads = 512;
constexpr int kPlanMaxBlocks = 128;

__global__ void __launch_bounds__(kPlanThreads, 1)
plan_kernel(const int32_t* __restrict__ ids, int routed_rows, int expert_lo, int expert_hi, int tile_cap,
            const uint8_t* __restrict__ chunk_counts, int chunks, int chunk_rows,
            int32_t* __restrict__ expert_counts, int32_t* __restrict__ expert_offsets,
            int32_t* __restrict__ tile_expert, int32_t* __restrict__ tile_row0, int32_t* __restrict__ tile_rows,
            int32_t* __restrict__ tile_count, int32_t* __restrict__ padded_rows,
            int32_t* __restrict__ sorted_rows, int32_t* __restrict__ row_position) {
  constexpr int kWarps = kPlanThreads / 32;
  constexpr int kBits = kWarps + 1;              // words per expert, padded against bank conflicts
  __shared__ __align__(16) int sums[2][kWarps][kExperts];      // of the chunks before this block's, of the others
  unsigned* const bits = reinterpret_cast<unsigned*>(sums);     // once the sums have been read
  static_assert(sizeof(unsigned) * kExperts * kBits <= sizeof(sums), "the bits take the place of the sums");
  __shared__ int base[kExperts];
  __shared__ int warp_sums[3][kExperts / 32];
  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int block = blockIdx.x;
  pdl_enter();
  const int per_block = (chunks + gridDim.x - 1) / gridDim.x;
  const int first = min(chunks, block * per_block);
  const int row_lo = first * chunk_rows;
  const int row_hi = min(routed_rows, min(chunks, first + per_block) * chunk_rows);

  // sixteen experts per thread and load, 32 chunks at a time; the bytes of a batch add up in halves of a word
  const int column = threadIdx.x & 15;
  auto add_chunks = [&](int from, int to, int* out) {
    int total[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) total[k] = 0;
    constexpr int kStep = kPlanThreads / 16, kBatch = 8;       // loads of a batch are under way together
    for (int c = from + (threadIdx.x >> 4); c < to; c += kStep * kBatch) {
      uint4 w[kBatch];
#pragma unroll
      for (int i = 0; i < kBatch; ++i) {
        w[i] = make_uint4(0, 0, 0, 0);
        if (c + kStep * i < to)
          w[i] = __ldg(reinterpret_cast<const uint4*>(chunk_counts + static_cast<size_t>(c + kStep * i) * kExperts) + column);
      }
      unsigned even[4] = {0, 0, 0, 0}, odd[4] = {0, 0, 0, 0};
#pragma unroll
      for (int i = 0; i < kBatch; ++i) {
        const unsigned word[4] = {w[i].x, w[i].y, w[i].z, w[i].w};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          even[k] += word[k] & 0x00ff00ffu;
          odd[k] += (word[k] >> 8) & 0x00ff00ffu;
        }
      }
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        total[4 * k] += even[k] & 0xffffu;
        total[4 * k + 1] += odd[k] & 0xffffu;
        total[4 * k + 2] += even[k] >> 16;
        total[4 * k + 3] += odd[k] >> 16;
      }
    }
#pragma unroll
    for (int k = 0; k < 16; ++k) total[k] += __shfl_xor_sync(0xffffffffu, total[k], 16);
    if (lane < 16) {
#pragma unroll
      for (int k = 0; k < 16; k += 4)
        *reinterpret_cast<int4*>(out + 16 * column + k) = make_int4(total[k], total[k + 1], total[k + 2], total[k + 3]);
    }
  };
  add_chunks(0, first, sums[0][warp]);
  add_chunks(first, chunks, sums[1][warp]);
  __syncthreads();
  int count = 0, before = 0, v0 = 0, v1 = 0, v2 = 0;
  if (threadIdx.x < kExperts) {
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      before += sums[0][w][threadIdx.x];
      count += sums[1][w][threadIdx.x];
    }
    count += before;
    v0 = count;
    v1 = (count + tile_cap - 1) / tile_cap;
    v2 = (count + 31) / 32 * 32;
#pragma unroll
    for (int d = 1; d < 32; d *= 2) {
      const int a0 = __shfl_up_sync(0xffffffffu, v0, d);
      const int a1 = __shfl_up_sync(0xffffffffu, v1, d);
      const int a2 = __shfl_up_sync(0xffffffffu, v2, d);
      if (lane >= d) { v0 += a0; v1 += a1; v2 += a2; }
    }
    if (lane == 31) { warp_sums[0][warp] = v0; warp_sums[1][warp] = v1; warp_sums[2][warp] = v2; }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < kExperts * kBits; i += kPlanThreads) bits[i] = 0u;
  if (threadIdx.x < kExperts) {
    const int e = threadIdx.x;
    const int n_tiles = (count + tile_cap - 1) / tile_cap;
    int offset = v0 - count, first_tile = v1 - n_tiles, total = 0, total_tiles = 0, padded = 0;
#pragma unroll
    for (int w = 0; w < kExperts / 32; ++w) {
      if (w < warp) { offset += warp_sums[0][w]; first_tile += warp_sums[1][w]; }
      total += warp_sums[0][w];
      total_tiles += warp_sums[1][w];
      padded += warp_sums[2][w];
    }
    base[e] = offset + before;
    if (block == 0) {
      expert_counts[e] = count;
      expert_offsets[e] = offset;
      if (e == 0) {
        expert_offsets[kExperts] = total;
        *tile_count = total_tiles;
        *padded_rows = padded;
      }
      const int height = rows_per_tile(count, n_tiles, tile_cap);
      for (int t = 0; t < n_tiles; ++t) {
        tile_expert[first_tile + t] = e;
        tile_row0[first_tile + t] = offset + t * height;
        tile_rows[first_tile + t] = min(height, count - t * height);
      }
    }
  }
  __syncthreads();
  for (int row0 = row_lo; row0 < row_hi; row0 += kPlanThreads) {
    const int row = row0 + static_cast<int>(threadIdx.x);
    int e = row < row_hi ? ids[row] : -1;
    if (e < expert_lo || e >= expert_hi) e = -1;
    if (e >= 0) atomicOr(&bits[e * kBits + warp], 1u << lane);
    __syncthreads();
    if (e >= 0) {
      int pos = base[e] + __popc(bits[e * kBits + warp] & ((1u << lane) - 1u));
      for (int w = 0; w < warp; ++w) pos += __popc(bits[e * kBits + w]);
      sorted_rows[pos] = row;
      row_position[row] = pos;
    }
    if (row0 + kPlanThreads < row_hi) {          // the next rows of this block come behind these
      __syncthreads();
      if (threadIdx.x < kExperts) {
        int held = 0;
#pragma unroll
        for (int w = 0; w < kWarps; ++w) {
          held += __popc(bits[threadIdx.x * kBits + w]);
          bits[threadIdx.x * kBits + w] = 0u;
        }
        base[threadIdx.x] += held;
      }
      __syncthreads();
    }
  }
}

// Enqueues the dispatch plan for `rows` routed rows whose expert ids are `ids`.
// chunk_rows: flat rows per chunk of the counts that the router has left in ws->chunk_counts; 0: they are counted here
// tile_cap: rows per tile of the plan -- 128 for the one-SM product kernels, 256 for the two-SM form
cudaError_t launch_plan(PrefillWorkspace* ws, const int32_t* ids, int rows, int expert_lo, int expert_hi, int chunk_rows,
                        cudaStream_t stream, int* launches, int tile_cap = kTileRows) {
  if (chunk_rows == 0) {
    chunk_rows = kCountRows;
    const cudaError_t code = launch_pdl(count_rows_kernel, dim3((rows + kCountRows - 1) / kCountRows), dim3(kExperts), 0, stream,
                                        ids, rows, expert_lo, expert_hi, ws->chunk_counts);
    if (code != cudaSuccess) return code;
    *launches += 1;
  }
  const int chunks = (rows + chunk_rows - 1) / chunk_rows;
  *launches += 1;
  return launch_pdl(plan_kernel, dim3(min(chunks, kPlanMaxBlocks)), dim3(kPlanThreads), 0, stream, ids, rows, expert_lo,
                    expert_hi, tile_cap, static_cast<const uint8_t*>(ws->chunk_counts), chunks, chunk_rows, ws->expert_counts,
                    ws->expert_offsets, ws->tile_expert, ws->tile_row0, ws->tile_rows, ws->tile_count, ws->padded_rows,
                    ws->sorted_rows, ws->row_position);
}

// ---------------------------------------------------------------------------
// Copy of h2 rows into expert order, for the products that do not fetch their rows by token index (qualification: the
// CUDA-core cross-check, and the flag that asks for the copy).  One block per token, 16 bytes per thread: the row is read
// once and written to the up to eight places the plan gave it.
// ---------------------------------------------------------------------------
constexpr int kCopyThreads = kHidden / 8;

__global__ void __launch_bounds__(kCopyThreads)
gather_rows_kernel(const __nv_bfloat16* __restrict__ h2, const int32_t* __restrict__ ids,
                   const int32_t* __restrict__ row_position, __nv_bfloat16* __restrict__ gathered) {
  pdl_enter();
  const int token = blockIdx.x;
  const uint4 piece = __ldg(reinterpret_cast<const uint4*>(h2 + static_cast<size_t>(token) * kHidden) + threadIdx.x);
#pragma unroll
  for (int slot = 0; slot < kTopK; ++slot) {
    const int e = ids[token * kTopK + slot];
    if (e >= 0 && e < kExperts)            // rows of other ids are not in the plan
      reinterpret_cast<uint4*>(gathered + static_cast<size_t>(row_position[token * kTopK + slot]) * kHidden)[threadIdx.x] = piece;
  }
}

// ---------------------------------------------------------------------------
// Combine: routed = bf16((((r0+r4)+(r1+r5))+(r2+r6))+(r3+r7)) over the eight
// weighted expert outputs of a token, combined = bf16(routed + shared),
// out = bf16(residual + combined).  One block of 256 threads per token.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256)
combine_kernel(const __nv_bfloat16* __restrict__ expert_down,
               const int32_t* __restrict__ row_position,
               const __nv_bfloat16* __restrict__ shared_scaled,
               const __nv_bfloat16* __restrict__ residual, __nv_bfloat16* __restrict__ out,
               __nv_bfloat16* __restrict__ dbg_routed,
               const __nv_bfloat16* __restrict__ next_norm_weight,
               __nv_bfloat16* __restrict__ next_norm_out, float eps) {
  __shared__ float group_sums[8];
  pdl_enter();
  const int token = blockIdx.x;
  const int t = threadIdx.x;
  float slot[kTopK][8];
#pragma unroll
  for (int s = 0; s < kTopK; ++s) {
    const int pos = row_position != nullptr ? row_position[token * kTopK + s] : token * kTopK + s;
    unpack8(__ldg(reinterpret_cast<const uint4*>(expert_down + static_cast<size_t>(pos) * kHidden) + t),
            slot[s]);
  }
  float sh[8], rs[8];
  const size_t base = static_cast<size_t>(token) * kHidden;
  unpack8(__ldg(reinterpret_cast<const uint4*>(shared_scaled + base) + t), sh);
  unpack8(__ldg(reinterpret_cast<const uint4*>(residual + base) + t), rs);
  uint32_t packed[4], packed_routed[4];
  float o8[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const float s04 = __fadd_rn(slot[0][j], slot[4][j]);
    const float s15 = __fadd_rn(slot[1][j], slot[5][j]);
    const float s26 = __fadd_rn(slot[2][j], slot[6][j]);
    const float s37 = __fadd_rn(slot[3][j], slot[7][j]);
    float sum = __fadd_rn(s04, s15);
    sum = __fadd_rn(sum, s26);
    sum = __fadd_rn(sum, s37);
    const uint16_t routed_bits = float_to_bf16_bits(sum);
    const float combined = round_bf16(__fadd_rn(bf16_bits_to_float(routed_bits), sh[j]));
    const uint16_t o = float_to_bf16_bits(__fadd_rn(rs[j], combined));
    o8[j] = bf16_bits_to_float(o);
    if (j & 1) {
      packed[j / 2] |= static_cast<uint32_t>(o) << 16;
      packed_routed[j / 2] |= static_cast<uint32_t>(routed_bits) << 16;
    } else {
      packed[j / 2] = o;
      packed_routed[j / 2] = routed_bits;
    }
  }
  reinterpret_cast<uint4*>(out + base)[t] = make_uint4(packed[0], packed[1], packed[2], packed[3]);
  if (dbg_routed != nullptr) {
    reinterpret_cast<uint4*>(dbg_routed + base)[t] =
        make_uint4(packed_routed[0], packed_routed[1], packed_routed[2], packed_routed[3]);
  }
  // Optional exit: RMSNorm of the row just produced (the next layer's input norm).  Sum of squares in
  // the order of the reference kernel (native/src/native_pointwise.hip.cpp:109-142): partial p of 256
  // adds elements p, p + 256, ... in that order, the partials fold by halving.  Thread t holds elements
  // 8 t .. 8 t + 7, so the squares go through shared memory once and thread p picks up its eight.
  if (next_norm_out != nullptr) {
    __shared__ float squares[kHidden];
    __shared__ float partial[256];
#pragma unroll
    for (int j = 0; j < 8; ++j) squares[8 * t + j] = __fmul_rn(o8[j], o8[j]);   // exact: BF16 squared fits FP32
    __syncthreads();
    float acc = 0.0f;
#pragma unroll
    for (int i = 0; i < 8; ++i) acc = __fadd_rn(acc, squares[t + 256 * i]);
    partial[t] = acc;
    __syncthreads();
    if (t < 32) {
      // widths 128, 64, 32 fold four groups of 64 partials onto lane t, widths 16 .. 1 are lane shuffles
      float q = __fadd_rn(__fadd_rn(__fadd_rn(partial[t], partial[t + 128]), __fadd_rn(partial[t + 64], partial[t + 192])),
                          __fadd_rn(__fadd_rn(partial[t + 32], partial[t + 160]), __fadd_rn(partial[t + 96], partial[t + 224])));
#pragma unroll
      for (int width = 16; width >= 1; width >>= 1) q = __fadd_rn(q, __shfl_down_sync(0xffffffffu, q, width));
      if (t == 0) group_sums[0] = q;
    }
    __syncthreads();
    const float total = group_sums[0];
    const float inv = det_rsqrtf(__fadd_rn(__fdiv_rn(total, static_cast<float>(kHidden)), eps));
    float w[8];
    unpack8(__ldg(reinterpret_cast<const uint4*>(next_norm_weight) + t), w);
    uint32_t normed[4];
#pragma unroll
    for (int j = 0; j < 8; j += 2) {
      const float a = __fmul_rn(__fmul_rn(o8[j], inv), __fadd_rn(w[j], 1.0f));
      const float b = __fmul_rn(__fmul_rn(o8[j + 1], inv), __fadd_rn(w[j + 1], 1.0f));
      normed[j / 2] = static_cast<uint32_t>(float_to_bf16_bits(a)) |
                      (static_cast<uint32_t>(float_to_bf16_bits(b)) << 16);
    }
    reinterpret_cast<uint4*>(next_norm_out + base)[t] = make_uint4(normed[0], normed[1], normed[2], normed[3]);
  }
}


// ---------------------------------------------------------------------------
// Expert-parallel prefill over peer memory (NVLink).  Tokens are sharded T / W
// per GPU, experts 256 / W per GPU.  Everything that crosses NVLink is a plain
// store into a peer's exchange region: every rank's activation rows and routing
// go to every GPU (all-gathers by peer stores), and the weighted expert rows go
// to the GPU that owns their token -- from the down kernel's epilogue, or, in
// the pipelined variant, from the copy kernel below.  The tensor-core kernels
// only ever READ this GPU's own memory.
// ---------------------------------------------------------------------------
struct EpPointers {
  uint8_t* region[8];
};

// every rank's routing (ids, weights) into every rank's table, slot `rank`
__global__ void __launch_bounds__(256)
ep_publish_routing_kernel(const int32_t* __restrict__ ids, const float* __restrict__ weights, int n,
                          EpPointers peers, int world, int rank, size_t off_ids, size_t off_weights) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int id = ids[i];
  const float w = weights[i];
  for (int q = 0; q < world; ++q) {
    reinterpret_cast<int32_t*>(peers.region[q] + off_ids)[static_cast<size_t>(rank) * n + i] = id;
    reinterpret_cast<float*>(peers.region[q] + off_weights)[static_cast<size_t>(rank) * n + i] = w;
  }
}

// every rank's h2 rows into every rank's [T, 2048] table, block `rank`: the all-gather that replaces a
// dispatch of single rows (with eight experts out of 256 per token nearly every rank needs nearly every
// token).  It does not depend on the routing, so it runs beside the router on its own stream; a small grid,
// since NVLink, not the SMs, sets its pace.
__global__ void __launch_bounds__(256)
ep_publish_rows_kernel(const uint4* __restrict__ rows, size_t n_vec, EpPointers peers, int world, int rank,
                       size_t off_h2) {
  const size_t stride = static_cast<size_t>(gridDim.x) * blockDim.x;
  for (size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n_vec; i += stride) {
    const uint4 v = rows[i];
    for (int q = 0; q < world; ++q)
      reinterpret_cast<uint4*>(peers.region[q] + off_h2)[static_cast<size_t>(rank) * n_vec + i] = v;
  }
}

// after the stores of the previous kernel: raise this rank's flag on every GPU
__global__ void ep_signal_kernel(EpPointers peers, int world, int rank, size_t off_flag, unsigned epoch) {
  const int q = threadIdx.x;
  if (q >= world) return;
  __threadfence_system();
  unsigned* flag = reinterpret_cast<unsigned*>(peers.region[q] + off_flag) + rank;
  asm volatile("st.release.sys.global.u32 [%0], %1;" :: "l"(flag), "r"(epoch) : "memory");
}

// bounded wait until every rank's flag in this GPU's region carries `epoch`
__global__ void ep_wait_kernel(const uint8_t* region, int world, size_t off_flag, unsigned epoch, int* status) {
  const int q = threadIdx.x;
  if (q >= world) return;
  const unsigned* flag = reinterpret_cast<const unsigned*>(region + off_flag) + q;
  const unsigned long long start = global_timer_ns();
  unsigned spins = 0;
  while (true) {
    unsigned v;
    asm volatile("ld.acquire.sys.global.u32 %0, [%1];" : "=r"(v) : "l"(flag) : "memory");
    if (static_cast<int>(v - epoch) >= 0) break;      // a later epoch also means this one has passed
    if ((++spins & 63u) == 0u && global_timer_ns() - start > kWaitBudgetNs) {
      atomicCAS(status, 0, kStatusTimeoutPeer);
      break;
    }
  }
}

// Sorted-row range of part `part` of `parts` of the plan's tiles (the same split the product kernel
// makes): tiles follow the sorted order, so a range of tiles is a range of rows.
__device__ __forceinline__ void part_rows(const int32_t* __restrict__ expert_offsets,
                                          const int32_t* __restrict__ tile_row0,
                                          const int32_t* __restrict__ tile_count, int part, int parts,
                                          int& row_lo, int& row_hi) {
  const int total = expert_offsets[kExperts];
  const int n_tiles = *tile_count;
  const int tile_lo = static_cast<int>(static_cast<long long>(n_tiles) * part / parts);
  const int tile_hi = static_cast<int>(static_cast<long long>(n_tiles) * (part + 1) / parts);
  row_lo = tile_lo < n_tiles ? tile_row0[tile_lo] : total;
  row_hi = tile_hi < n_tiles ? tile_row0[tile_hi] : total;
}

// dispatch: row `pos` of this GPU's plan <- h2 row of its token, wherever that token lives
__global__ void __launch_bounds__(256)
ep_gather_rows_kernel(EpPointers peers, size_t off_h2, int tokens_per_rank,
                      const int32_t* __restrict__ sorted_rows, const int32_t* __restrict__ expert_offsets,
                      const int32_t* __restrict__ tile_row0, const int32_t* __restrict__ tile_count,
                      int part, int parts, __nv_bfloat16* __restrict__ gathered) {
  const int lane = threadIdx.x & 31;
  int row_lo, row_hi;
  part_rows(expert_offsets, tile_row0, tile_count, part, parts, row_lo, row_hi);
  // a small grid that loops: the copy kernels share the SMs with the product kernels of another
  // part, whose one-block-per-SM grid must find room at once
  for (int pos = row_lo + blockIdx.x * 8 + (threadIdx.x >> 5); pos < row_hi; pos += gridDim.x * 8) {
    const int token = sorted_rows[pos] >> 3;
    const int owner = token / tokens_per_rank;
    const int local = token - owner * tokens_per_rank;
    const uint4* src = reinterpret_cast<const uint4*>(peers.region[owner] + off_h2) +
                       static_cast<size_t>(local) * (kHidden / 8);
    uint4* dst = reinterpret_cast<uint4*>(gathered + static_cast<size_t>(pos) * kHidden);
    uint4 v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = src[i * 32 + lane];
#pragma unroll
    for (int i = 0; i < 8; ++i) dst[i * 32 + lane] = v[i];
  }
}

// combine, first half: the weighted expert output of plan row `pos` goes to the GPU that owns
// its token, at that token's (token, slot) position
__global__ void __launch_bounds__(256)
ep_return_rows_kernel(const __nv_bfloat16* __restrict__ expert_down, const int32_t* __restrict__ sorted_rows,
                      const int32_t* __restrict__ expert_offsets,
                      const int32_t* __restrict__ tile_row0, const int32_t* __restrict__ tile_count,
                      int part, int parts, EpPointers peers, size_t off_return, int tokens_per_rank) {
  const int lane = threadIdx.x & 31;
  int row_lo, row_hi;
  part_rows(expert_offsets, tile_row0, tile_count, part, parts, row_lo, row_hi);
  for (int pos = row_lo + blockIdx.x * 8 + (threadIdx.x >> 5); pos < row_hi; pos += gridDim.x * 8) {
    const int flat = sorted_rows[pos];
    const int owner = (flat >> 3) / tokens_per_rank;
    const int local_flat = flat - owner * tokens_per_rank * kTopK;
    const uint4* src = reinterpret_cast<const uint4*>(expert_down + static_cast<size_t>(pos) * kHidden);
    uint4* dst = reinterpret_cast<uint4*>(peers.region[owner] + off_return) +
                 static_cast<size_t>(local_flat) * (kHidden / 8);
    uint4 v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = src[i * 32 + lane];
#pragma unroll
    for (int i = 0; i < 8; ++i) dst[i * 32 + lane] = v[i];
  }
}

// qualification view: weighted expert output rows in flat (token, slot) order
__global__ void __launch_bounds__(256)
export_slot_rows_kernel(const __nv_bfloat16* __restrict__ expert_down, const int32_t* __restrict__ row_position,
                        int routed_rows, __nv_bfloat16* __restrict__ out) {
  const int lane = threadIdx.x & 31;
  const int flat = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (flat >= routed_rows) return;
  const uint4* src = reinterpret_cast<const uint4*>(expert_down + static_cast<size_t>(row_position[flat]) * kHidden);
  uint4* dst = reinterpret_cast<uint4*>(out + static_cast<size_t>(flat) * kHidden);
#pragma unroll
  for (int i = 0; i < 8; ++i) dst[i * 32 + lane] = src[i * 32 + lane];
}

int set_error(char* error, size_t error_bytes, cudaError_t code, const char* what) {
  std::snprintf(error, error_bytes, "%s: %s (%s)", what, cudaGetErrorName(code),
                cudaGetErrorString(code));
  (void)cudaGetLastError();
  return static_cast<int>(code);
}

// Warps per token of the certified router: as many as keep every block of the launch resident at once.  us per layer with
// 1 / 2 / 4 warps per token, balanced routing: 268 / 265 / 264 at 129 tokens, 280 / 276 / 276 at 333, 289 / 287 / 284 at
// 592, 311 / 305 / 313 at 1024, 317 / 312 / 320 at 1184 (the last with two), 343 / 349 / 362 at 2047.
int certified_ways(int tokens, int sm_count) {
  const int warps = kCertBlocksPerSm * kCertWarps * sm_count;
  return 4 * tokens <= warps ? 4 : 2 * tokens <= warps ? 2 : 1;
}

// Runs of K of the router logits: few rows are few units, each bound by how fast one pair of SMs can fetch 256 router rows.
// us per layer with 1 / 2 / 4 / 8 runs, balanced routing, weights of three layers in rotation: 265 / 262 / 262 / 262 at 129
// tokens, 278 / 276 / 276 / 277 at 333, 309 / 306 / 306 / 307 at 1024, 348 / 346 / 346 / 349 at 2047, 437 / 438 / 439 / 447 at
// 4096 (the median moves by 1 to 2 % from loop to loop).  Two builds in turn, two runs / four: 287.0 / 286.2 at 333 tokens,
// 309.3 / 308.4 at 1024, two runs of one build within 0.2 %.
constexpr int kSplitMaxTokens = 1024;      // four runs up to here, two beyond
int router_splits(int tokens) { return tokens <= kSplitMaxTokens ? 4 : 2; }
size_t approx_logit_count(size_t tokens) {
  const size_t small = tokens < kSplitMaxTokens ? tokens : kSplitMaxTokens;
  return (2 * tokens > 4 * small ? 2 * tokens : 4 * small) * kExperts;
}

size_t align256(size_t v) { return (v + 255) / 256 * 256; }

struct Layout {
  size_t ids, scores, weights, sigmoid, approx, stats, chunk_counts, counts, offsets, sorted, position,
      tile_expert, tile_row0, tile_rows, tile_count, padded, gathered, act, down, shared_act,
      shared_scaled, x0, x1, h2, total;
};

Layout layout_for(size_t T) {
  Layout l{};
  size_t cursor = 0;
  auto take = [&](size_t bytes) { const size_t at = cursor; cursor += align256(bytes); return at; };
  const size_t rows = T * kTopK;
  const size_t tiles = static_cast<size_t>(max_tiles_for(static_cast<int>(T)));
  l.ids = take(rows * 4);
  l.scores = take(rows * 4);
  l.weights = take(rows * 4);
  l.sigmoid = take(T * 4);
  l.approx = take(approx_logit_count(T) * 4);
  l.stats = take(5 * sizeof(unsigned long long));
  l.chunk_counts = take((T + 1) / 2 * kExperts);      // two tokens per chunk at least
  l.counts = take(kExperts * 4);
  l.offsets = take((kExperts + 1) * 4);
  l.sorted = take(rows * 4);
  l.position = take(rows * 4);
  l.tile_expert = take(tiles * 4);
  l.tile_row0 = take(tiles * 4);
  l.tile_rows = take(tiles * 4);
  l.tile_count = take(4);
  l.padded = take(4);
  l.gathered = take(rows * kHidden * 2);
  l.act = take(rows * kInter * 2);
  l.down = take(rows * kHidden * 2);
  l.shared_act = take(T * kSharedInter * 2);
  l.shared_scaled = take(T * kHidden * 2);
  l.x0 = take(T * kHidden * 2);
  l.x1 = take(T * kHidden * 2);
  l.h2 = take(T * kHidden * 2);
  l.total = cursor;
  return l;
}

}  // namespace

cudaError_t launch_router_row_norms(const __nv_bfloat16* router, float* norms, cudaStream_t stream) {
  router_row_norms_kernel<<<kExperts / 8, 256, 0, stream>>>(router, norms);
  return cudaGetLastError();
}

size_t prefill_workspace_bytes(uint32_t capacity_tokens) {
  return capacity_tokens == 0 ? 0 : layout_for(capacity_tokens).total;
}

int prefill_workspace_allocate(PrefillWorkspace* ws, uint32_t capacity_tokens, int sm_count,
                               char* error, size_t error_bytes) {
  const Layout l = layout_for(capacity_tokens);
  cudaError_t code = cudaMalloc(&ws->base, l.total);
  if (code != cudaSuccess) return set_error(error, error_bytes, code, "cudaMalloc prefill workspace");
  code = cudaMemset(ws->base, 0, l.total);
  if (code != cudaSuccess) return set_error(error, error_bytes, code, "cudaMemset prefill workspace");
  code = cudaStreamCreateWithFlags(&ws->side_stream, cudaStreamNonBlocking);
  if (code == cudaSuccess) code = cudaEventCreateWithFlags(&ws->fork_event, cudaEventDisableTiming);
  if (code == cudaSuccess) code = cudaEventCreateWithFlags(&ws->router_event, cudaEventDisableTiming);
  if (code == cudaSuccess) code = cudaEventCreateWithFlags(&ws->join_event, cudaEventDisableTiming);
  if (code == cudaSuccess) code = cudaStreamCreateWithFlags(&ws->inbound_stream, cudaStreamNonBlocking);
  if (code == cudaSuccess) code = cudaStreamCreateWithFlags(&ws->outbound_stream, cudaStreamNonBlocking);
  if (code == cudaSuccess) code = cudaEventCreateWithFlags(&ws->plan_event, cudaEventDisableTiming);
  if (code == cudaSuccess) code = cudaEventCreateWithFlags(&ws->returned_event, cudaEventDisableTiming);
  if (code == cudaSuccess) code = cudaEventCreateWithFlags(&ws->published_event, cudaEventDisableTiming);
  for (int k = 0; k < PrefillWorkspace::kMaxParts && code == cudaSuccess; ++k) {
    code = cudaEventCreateWithFlags(&ws->gathered_event[k], cudaEventDisableTiming);
    if (code == cudaSuccess) code = cudaEventCreateWithFlags(&ws->computed_event[k], cudaEventDisableTiming);
  }
  if (code != cudaSuccess) return set_error(error, error_bytes, code, "side stream / events of the prefill workspace");
  ws->total_bytes = l.total;
  ws->capacity = static_cast<int>(capacity_tokens);
  ws->sm_count = sm_count;
  uint8_t* b = ws->base;
  ws->topk_ids = reinterpret_cast<int32_t*>(b + l.ids);
  ws->topk_scores = reinterpret_cast<float*>(b + l.scores);
  ws->topk_weights = reinterpret_cast<float*>(b + l.weights);
  ws->shared_sigmoid = reinterpret_cast<float*>(b + l.sigmoid);
  ws->approx_logits = reinterpret_cast<float*>(b + l.approx);
  ws->router_stats = reinterpret_cast<unsigned long long*>(b + l.stats);
  ws->chunk_counts = b + l.chunk_counts;
  ws->expert_counts = reinterpret_cast<int32_t*>(b + l.counts);
  ws->expert_offsets = reinterpret_cast<int32_t*>(b + l.offsets);
  ws->sorted_rows = reinterpret_cast<int32_t*>(b + l.sorted);
  ws->row_position = reinterpret_cast<int32_t*>(b + l.position);
  ws->tile_expert = reinterpret_cast<int32_t*>(b + l.tile_expert);
  ws->tile_row0 = reinterpret_cast<int32_t*>(b + l.tile_row0);
  ws->tile_rows = reinterpret_cast<int32_t*>(b + l.tile_rows);
  ws->tile_count = reinterpret_cast<int32_t*>(b + l.tile_count);
  ws->padded_rows = reinterpret_cast<int32_t*>(b + l.padded);
  ws->gathered = reinterpret_cast<__nv_bfloat16*>(b + l.gathered);
  ws->expert_act = reinterpret_cast<__nv_bfloat16*>(b + l.act);
  ws->expert_down = reinterpret_cast<__nv_bfloat16*>(b + l.down);
  ws->shared_act = reinterpret_cast<__nv_bfloat16*>(b + l.shared_act);
  ws->shared_scaled = reinterpret_cast<__nv_bfloat16*>(b + l.shared_scaled);
  ws->stack_x0 = reinterpret_cast<__nv_bfloat16*>(b + l.x0);
  ws->stack_x1 = reinterpret_cast<__nv_bfloat16*>(b + l.x1);
  ws->stack_h2 = reinterpret_cast<__nv_bfloat16*>(b + l.h2);
  return AIMA_MOE_OK;
}

void prefill_workspace_free(PrefillWorkspace* ws) {
  if (ws->base != nullptr) cudaFree(ws->base);
  if (ws->fork_event != nullptr) cudaEventDestroy(ws->fork_event);
  if (ws->router_event != nullptr) cudaEventDestroy(ws->router_event);
  if (ws->join_event != nullptr) cudaEventDestroy(ws->join_event);
  if (ws->side_stream != nullptr) cudaStreamDestroy(ws->side_stream);
  if (ws->plan_event != nullptr) cudaEventDestroy(ws->plan_event);
  if (ws->returned_event != nullptr) cudaEventDestroy(ws->returned_event);
  if (ws->published_event != nullptr) cudaEventDestroy(ws->published_event);
  for (int k = 0; k < PrefillWorkspace::kMaxParts; ++k) {
    if (ws->gathered_event[k] != nullptr) cudaEventDestroy(ws->gathered_event[k]);
    if (ws->computed_event[k] != nullptr) cudaEventDestroy(ws->computed_event[k]);
  }
  if (ws->inbound_stream != nullptr) cudaStreamDestroy(ws->inbound_stream);
  if (ws->outbound_stream != nullptr) cudaStreamDestroy(ws->outbound_stream);
  *ws = PrefillWorkspace{};
}

// Qualification: routing supplied by the harness replaces the router's ids and weights (the router still
// runs: the shared expert's sigmoid gate comes from it).  Mirrors the reference's "oracle-seeded
// routing" rerun (native/src/native_moe_prefill.hip.cpp:1059-1123), which isolates the expert
// arithmetic from tie-order effects.
__global__ void forced_routing_kernel(const int32_t* __restrict__ ids, const __nv_bfloat16* __restrict__ weights,
                                      int n, int32_t* __restrict__ topk_ids, float* __restrict__ topk_weights,
                                      float* __restrict__ topk_scores) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int id = ids[i];
  topk_ids[i] = (id >= 0 && id < kExperts) ? id : 0;
  topk_weights[i] = __bfloat162float(weights[i]);
  topk_scores[i] = 0.0f;
}

constexpr int kGatherMaxTokens = 128;

int prefill_layer_launch(PrefillWorkspace* ws, const PrefillCall& call, cudaStream_t stream,
                         int* launches, char* error, size_t error_bytes) {
  const int T = call.tokens;
  const PdlScope pdl_scope(T <= pdl_max_tokens());
  const int rows = T * kTopK;
  const aima_moe_debug_views* dbg = call.debug;
  int count = 0;
  cudaError_t code;

  // Products: the two-SM tensor-core form, which takes the shared expert's rows along as tiles of their own, with tiles of
  // up to 256 rows; or the CUDA-core cross-check, with 128-row tiles and the shared expert in launches of its own.
  const bool simt = ws->use_simt_gemm;
  const __nv_bfloat16* h2 = static_cast<const __nv_bfloat16*>(call.h2);

  int chunk_rows = 0;      // of the counts the router leaves for the plan; 0: none
  const bool exact_router = ws->exact_router || (dbg != nullptr && dbg->router_logits != nullptr) ||
                            call.router_row_norms == nullptr;
  if (exact_router) {
    code = opt_in_dynamic_smem<prefill_router_kernel>(kRouterSmemBytes);
    if (code != cudaSuccess) return set_error(error, error_bytes, code, "cudaFuncSetAttribute router");
    prefill_router_kernel<<<(T + kRouterWarps - 1) / kRouterWarps, kRouterWarps * 32, kRouterSmemBytes, stream>>>(
        static_cast<const __nv_bfloat16*>(call.h2), call.layer.router, call.layer.shared_gate,
        call.router_bias, call.quant_eighths, T, ws->topk_ids, ws->topk_scores, ws->topk_weights,
        ws->shared_sigmoid, dbg ? static_cast<float*>(dbg->router_logits) : nullptr,
        dbg ? static_cast<__nv_bfloat16*>(dbg->topk_weights) : nullptr);
    if ((code = cudaGetLastError()) != cudaSuccess) return set_error(error, error_bytes, code, "prefill_router_kernel");
    ++count;
  } else if (T <= kSmallRouterTokens && ws->router_audit_stride == 0) {
    code = launch_pdl(prefill_logits_small_kernel, dim3(kExperts / 2 + 1), dim3(256), 0, stream, h2, call.layer.router,
                      call.layer.shared_gate, T, ws->approx_logits, ws->shared_sigmoid);
    if (code == cudaSuccess)
      code = launch_pdl(prefill_select_kernel, dim3((T + kCertWarps - 1) / kCertWarps), dim3(kCertWarps * 32), 0, stream,
                        static_cast<const float*>(ws->approx_logits), call.router_bias, call.quant_eighths, T,
                        ws->topk_ids, ws->topk_scores, ws->topk_weights,
                        dbg ? static_cast<__nv_bfloat16*>(dbg->topk_weights) : nullptr, ws->chunk_counts);
    if (code != cudaSuccess) return set_error(error, error_bytes, code, "router of a short call");
    chunk_rows = kCertWarps * kTopK;
    count += 2;
  } else {
    // tensor-core logits for the candidate filter, then exact recomputation of the candidates
    GroupedGemm r{};
    r.max_tiles = (T + kTileRows - 1) / kTileRows; r.dense_rows = T;
    r.a = static_cast<const __nv_bfloat16*>(call.h2); r.lda = kHidden; r.k = kHidden;
    r.b0 = call.layer.router; r.n = kExperts; r.c_f32 = ws->approx_logits; r.ldc = kExperts;
    TcExtra rx{};
    rx.status = ws->status; rx.sm_count = ws->sm_count; rx.a_rows = static_cast<uint64_t>(T); rx.experts_in_b = 1;
    rx.pair = true;
    rx.k_splits = router_splits(T);
    if ((code = launch_grouped_gemm_tc(kGemmPlainF32, r, rx, stream)) != cudaSuccess)
      return set_error(error, error_bytes, code, "router logits product");
    const int ways = certified_ways(T, ws->sm_count);
    const auto kernel = ways == 4 ? prefill_router_certified_kernel<4>
                                  : ways == 2 ? prefill_router_certified_kernel<2> : prefill_router_certified_kernel<1>;
    const int block_tokens = kCertWarps / ways;
    chunk_rows = block_tokens * kTopK;
    const ApproxLogits approx{ws->approx_logits, static_cast<size_t>(T) * kExperts, rx.k_splits};
    code = launch_pdl(kernel, dim3((T + block_tokens - 1) / block_tokens), dim3(kCertWarps * 32), 0, stream, h2,
                      call.layer.router, call.layer.shared_gate, approx, call.router_row_norms, call.router_bias,
                      call.quant_eighths, T, ws->topk_ids, ws->topk_scores, ws->topk_weights, ws->shared_sigmoid,
                      dbg ? static_cast<__nv_bfloat16*>(dbg->topk_weights) : nullptr, ws->router_stats,
                      ws->router_audit_stride, ws->chunk_counts);
    if (code != cudaSuccess)
      return set_error(error, error_bytes, code, "prefill_router_certified_kernel");
    count += 2;
  }

  if (call.forced_ids != nullptr) {
    forced_routing_kernel<<<(rows + 255) / 256, 256, 0, stream>>>(
        call.forced_ids, static_cast<const __nv_bfloat16*>(call.forced_weights), rows, ws->topk_ids,
        ws->topk_weights, ws->topk_scores);
    if ((code = cudaGetLastError()) != cudaSuccess) return set_error(error, error_bytes, code, "forced_routing_kernel");
    ++count;
    chunk_rows = 0;
  }

  const int tile_cap = simt ? kTileRows : 2 * kTileRows;
  if ((code = launch_plan(ws, ws->topk_ids, rows, 0, kExperts, chunk_rows, stream, &count, tile_cap)) != cudaSuccess)
    return set_error(error, error_bytes, code, "dispatch plan");

  // Dispatch: the gate_up product takes its rows by token index, through TMA gathers in a short call and through cp.async
  // beyond kGatherMaxTokens.  A gather moves four rows per 45 cycles and is issued by one thread: the shortest way for a few
  // rows, 1440 cycles a stage against 512 of tensor time for a tall tile.  us per layer, TMA gathers / cp.async: balanced
  // routing 118 / 119 at 16 tokens, 232 / 234 at 64, 252 / 256 at 96, 262 / 263 at 128, 275 / 276 at 333, 304 / 305 at 1024;
  // Zipf 69 / 70 at 16, 93 / 93 at 64, 109 / 106 at 96, 117 / 114 at 128, 168 / 156 at 333, 254 / 235 at 1024; eight hot
  // experts 39 / 40 at 16, 41 / 40 at 64, 46 / 43 at 96, 50 / 46 at 128, 63 / 57 at 333, 102 / 82 at 1024.  Balanced rows, which
  // keep the tiles short, never gain from cp.async below 2047 tokens; skewed ones do from 64 on.  The line favours the balanced
  // ones (1 %) up to 128 tokens, at 2 % with Zipf and 9 % with eight hot experts there, and the skewed ones beyond.
  // Above 1024 tokens TMA gathers were once helped by a copy of the rows in expert order, read by tile loads (268 MB written
  // and read back at 8192 tokens); copy / cp.async: balanced 337 / 334 at 2047, 442 / 424 at 4096, 730 / 699 at 8192, Zipf
  // 330 / 313, 489 / 450, 769 / 716, hot 146 / 134, 290 / 261, 585 / 517.
  const bool fused_dispatch = ws->fused_dispatch && !simt;
  if (!fused_dispatch) {
    code = launch_pdl(gather_rows_kernel, dim3(T), dim3(kCopyThreads), 0, stream, h2, ws->topk_ids, ws->row_position, ws->gathered);
    if (code != cudaSuccess) return set_error(error, error_bytes, code, "gather_rows_kernel");
    ++count;
  }

  // routed experts: gate_up + SwiGLU, then down x routing weight
  GroupedGemm g{};
  g.tile_expert = ws->tile_expert; g.tile_row0 = ws->tile_row0; g.tile_rows = ws->tile_rows;
  g.tile_count = ws->tile_count; g.max_tiles = max_tiles_for(T); g.dense_rows = 0;
  g.a = ws->gathered; g.lda = kHidden; g.k = kHidden;
  g.b0 = call.layer.expert_gate_up; g.b1 = nullptr;
  g.b_expert_stride = static_cast<size_t>(2 * kInter) * kHidden;
  g.n = kInter; g.c = ws->expert_act; g.ldc = kInter;
  g.row_scale = nullptr; g.sorted_rows = ws->sorted_rows;
  TcExtra extra{};
  extra.status = ws->status; extra.sm_count = ws->sm_count;
  extra.experts_in_b = call.experts_local;
  extra.pair = !simt;
  if (fused_dispatch) {
    g.gather_src = h2;
    extra.a_rows = static_cast<uint64_t>(T);
    extra.fetch = T > kGatherMaxTokens;
  } else {
    extra.a_rows = static_cast<uint64_t>(ws->capacity) * kTopK;
  }
  extra.shared = SharedProblem{T, h2, call.layer.shared_gate_proj, call.layer.shared_up_proj, ws->shared_act, nullptr};
  if (simt) {
    GroupedGemm s{};
    s.max_tiles = (T + kTileRows - 1) / kTileRows; s.dense_rows = T;
    s.a = h2; s.lda = kHidden; s.k = kHidden;
    s.b0 = call.layer.shared_gate_proj; s.b1 = call.layer.shared_up_proj;
    s.n = kSharedInter; s.c = ws->shared_act; s.ldc = kSharedInter;
    code = launch_grouped_gemm_simt(kGemmSharedGateUp, s, stream);
    if (code == cudaSuccess) {
      s.a = ws->shared_act; s.lda = kSharedInter; s.k = kSharedInter;
      s.b0 = call.layer.shared_down_proj; s.b1 = nullptr;
      s.n = kHidden; s.c = ws->shared_scaled; s.ldc = kHidden;
      s.row_scale = ws->shared_sigmoid;
      code = launch_grouped_gemm_simt(kGemmSharedDown, s, stream);
    }
    if (code == cudaSuccess) code = launch_grouped_gemm_simt(kGemmExpertGateUp, g, stream);
    count += 2;
  } else {
    code = launch_grouped_gemm_tc(kGemmExpertGateUp, g, extra, stream);
  }
  if (code != cudaSuccess) return set_error(error, error_bytes, code, "grouped gemm expert gate_up");
  g.gather_src = nullptr;
  extra.a_rows = static_cast<uint64_t>(ws->capacity) * kTopK;
  g.a = ws->expert_act; g.lda = kInter; g.k = kInter;
  g.b0 = call.layer.expert_down; g.b_expert_stride = static_cast<size_t>(kHidden) * kInter;
  g.n = kHidden; g.c = ws->expert_down; g.ldc = kHidden;
  g.row_scale = ws->topk_weights; g.sorted_rows = ws->sorted_rows;
  extra.shared = SharedProblem{T, ws->shared_act, call.layer.shared_down_proj, nullptr, ws->shared_scaled, ws->shared_sigmoid};
  code = simt ? launch_grouped_gemm_simt(kGemmExpertDown, g, stream)
              : launch_grouped_gemm_tc(kGemmExpertDown, g, extra, stream);
  if (code != cudaSuccess) return set_error(error, error_bytes, code, "grouped gemm expert down");
  count += 2;

  code = launch_pdl(combine_kernel, dim3(T), dim3(256), 0, stream, ws->expert_down, ws->row_position, ws->shared_scaled,
                    static_cast<const __nv_bfloat16*>(call.residual), static_cast<__nv_bfloat16*>(call.out),
                    dbg ? static_cast<__nv_bfloat16*>(dbg->routed) : nullptr,
                    static_cast<const __nv_bfloat16*>(call.next_norm_weight),
                    static_cast<__nv_bfloat16*>(call.next_norm_out), call.eps);
  if (code != cudaSuccess) return set_error(error, error_bytes, code, "combine_kernel");
  ++count;

  if (dbg != nullptr) {
    auto copy = [&](void* dst, const void* src, size_t bytes) {
      if (dst != nullptr) return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToDevice, stream);
      return cudaSuccess;
    };
    code = copy(dbg->h2, call.h2, static_cast<size_t>(T) * kHidden * 2);
    if (code == cudaSuccess) code = copy(dbg->topk_ids, ws->topk_ids, static_cast<size_t>(rows) * 4);
    if (code == cudaSuccess) code = copy(dbg->topk_scores, ws->topk_scores, static_cast<size_t>(rows) * 4);
    if (code == cudaSuccess) code = copy(dbg->shared_scaled, ws->shared_scaled, static_cast<size_t>(T) * kHidden * 2);
    if (code == cudaSuccess) code = copy(dbg->expert_counts, ws->expert_counts, kExperts * 4);
    if (code == cudaSuccess) code = copy(dbg->expert_offsets, ws->expert_offsets, (kExperts + 1) * 4);
    if (code == cudaSuccess) code = copy(dbg->sorted_rows, ws->sorted_rows, static_cast<size_t>(rows) * 4);
    if (code != cudaSuccess) return set_error(error, error_bytes, code, "cudaMemcpyAsync debug views");
    if (dbg->slot_rows != nullptr) {
      export_slot_rows_kernel<<<(rows + 7) / 8, 256, 0, stream>>>(ws->expert_down, ws->row_position, rows,
                                                                  static_cast<__nv_bfloat16*>(dbg->slot_rows));
      if ((code = cudaGetLastError()) != cudaSuccess) return set_error(error, error_bytes, code, "export_slot_rows_kernel");
    }
  }
  *launches = count;
  return AIMA_MOE_OK;
}

size_t ep_prefill_region_bytes(int capacity_tokens, int world, EpPrefillLayout* layout) {
  // capacity_tokens = global tokens per call; every rank holds capacity / world of them at most,
  // but the tables are sized for the global count so that any split fits
  const size_t rows = static_cast<size_t>(capacity_tokens) * kTopK;
  size_t cursor = 0;
  auto take = [&](size_t bytes) { const size_t at = cursor; cursor += (bytes + 255) / 256 * 256; return at; };
  EpPrefillLayout l{};
  l.off_flags_routing = take(64);
  l.off_flags_returned = take(64);
  l.off_ids = take(rows * 4);
  l.off_weights = take(rows * 4);
  l.off_h2 = take(static_cast<size_t>(capacity_tokens) * kHidden * 2);
  l.off_return = take(rows * kHidden * 2);
  l.bytes = cursor;
  (void)world;
  if (layout != nullptr) *layout = l;
  return cursor;
}

int prefill_layer_launch_ep(PrefillWorkspace* ws, const PrefillCall& call, EpPrefill* ep,
                            cudaStream_t stream, int* launches, char* error, size_t error_bytes) {
  const int T_loc = call.tokens;
  const PdlScope pdl_scope(false);   // plain stream order: kernels of this path wait for peers, nothing may sit resident ahead of them
  const int W = ep->world;
  const int T = T_loc * W;
  const int rows_loc = T_loc * kTopK;
  const int rows = T * kTopK;
  const aima_moe_debug_views* dbg = call.debug;
  const EpPrefillLayout& L = ep->layout;
  EpPointers peers{};
  for (int q = 0; q < W; ++q) peers.region[q] = ep->peers[q];
  uint8_t* mine = ep->peers[ep->rank];
  const unsigned epoch = ++ep->epoch;
  int count = 0;
  cudaError_t code;
  int mark_index = 0;
  auto mark = [&]() {
    if (ep->trace && ep->stage_events[mark_index] != nullptr) cudaEventRecord(ep->stage_events[mark_index], stream);
    ++mark_index;
  };
  mark();

  // The shared expert (weights replicated, this rank's tokens) runs on the side stream: its gate/up
  // product starts at once, its down product once the router kernel has written the sigmoid; it
  // fills the SMs while the main stream waits for peers and for rows crossing NVLink.
  cudaStream_t side = ws->side_stream;
  if ((code = cudaEventRecord(ws->fork_event, stream)) != cudaSuccess ||
      (code = cudaStreamWaitEvent(side, ws->fork_event, 0)) != cudaSuccess)
    return set_error(error, error_bytes, code, "fork of the shared-expert stream");
  GroupedGemm s{};
  TcExtra shared_extra{};
  shared_extra.status = ws->status; shared_extra.sm_count = ws->sm_count;
  s.max_tiles = (T_loc + kTileRows - 1) / kTileRows; s.dense_rows = T_loc;
  s.a = static_cast<const __nv_bfloat16*>(call.h2); s.lda = kHidden; s.k = kHidden;
  s.b0 = call.layer.shared_gate_proj; s.b1 = call.layer.shared_up_proj;
  s.n = kSharedInter; s.c = ws->shared_act; s.ldc = kSharedInter;
  shared_extra.a_rows = static_cast<uint64_t>(T_loc); shared_extra.experts_in_b = 1;
  if ((code = launch_grouped_gemm_tc(kGemmSharedGateUp, s, shared_extra, side)) != cudaSuccess)
    return set_error(error, error_bytes, code, "grouped gemm shared gate_up");
  ++count;

  // 0. this rank's h2 rows to every GPU, on the inbound stream beside the router (the flags of step 2 cover it)
  if ((code = cudaStreamWaitEvent(ws->inbound_stream, ws->fork_event, 0)) != cudaSuccess)
    return set_error(error, error_bytes, code, "fork of the row all-gather");
  ep_publish_rows_kernel<<<96, 256, 0, ws->inbound_stream>>>(
      static_cast<const uint4*>(call.h2), static_cast<size_t>(T_loc) * (kHidden / 8), peers, W, ep->rank, L.off_h2);
  if ((code = cudaGetLastError()) != cudaSuccess) return set_error(error, error_bytes, code, "ep_publish_rows_kernel");
  ++count;
  if ((code = cudaEventRecord(ws->published_event, ws->inbound_stream)) != cudaSuccess)
    return set_error(error, error_bytes, code, "published event");

  // 1. route this rank's tokens (certified router)
  GroupedGemm r{};
  r.max_tiles = (T_loc + kTileRows - 1) / kTileRows; r.dense_rows = T_loc;
  r.a = static_cast<const __nv_bfloat16*>(call.h2); r.lda = kHidden; r.k = kHidden;
  r.b0 = call.layer.router; r.n = kExperts; r.c_f32 = ws->approx_logits; r.ldc = kExperts;
  TcExtra rx{};
  rx.status = ws->status; rx.sm_count = ws->sm_count; rx.a_rows = static_cast<uint64_t>(T_loc); rx.experts_in_b = 1;
  if ((code = launch_grouped_gemm_tc(kGemmPlainF32, r, rx, stream)) != cudaSuccess)
    return set_error(error, error_bytes, code, "router logits product");
  prefill_router_certified_kernel<1><<<(T_loc + kCertWarps - 1) / kCertWarps, kCertWarps * 32, 0, stream>>>(
      static_cast<const __nv_bfloat16*>(call.h2), call.layer.router, call.layer.shared_gate,
      ApproxLogits{ws->approx_logits, 0, 1}, call.router_row_norms, call.router_bias, call.quant_eighths, T_loc, ws->topk_ids,
      ws->topk_scores, ws->topk_weights, ws->shared_sigmoid,
      dbg ? static_cast<__nv_bfloat16*>(dbg->topk_weights) : nullptr, ws->router_stats, ws->router_audit_stride, nullptr);
  if ((code = cudaGetLastError()) != cudaSuccess) return set_error(error, error_bytes, code, "prefill_router_certified_kernel");
  count += 2;
  if ((code = cudaEventRecord(ws->router_event, stream)) != cudaSuccess ||
      (code = cudaStreamWaitEvent(side, ws->router_event, 0)) != cudaSuccess)
    return set_error(error, error_bytes, code, "router event of the shared-expert stream");
  s.a = ws->shared_act; s.lda = kSharedInter; s.k = kSharedInter;
  s.b0 = call.layer.shared_down_proj; s.b1 = nullptr;
  s.n = kHidden; s.c = ws->shared_scaled; s.ldc = kHidden; s.row_scale = ws->shared_sigmoid;
  shared_extra.a_rows = static_cast<uint64_t>(ws->capacity);
  if ((code = launch_grouped_gemm_tc(kGemmSharedDown, s, shared_extra, side)) != cudaSuccess)
    return set_error(error, error_bytes, code, "grouped gemm shared down");
  ++count;
  if ((code = cudaEventRecord(ws->join_event, side)) != cudaSuccess)
    return set_error(error, error_bytes, code, "join event of the shared-expert stream");

  mark();
  // 2. all-gather of the routing tables by peer stores, then flags
  ep_publish_routing_kernel<<<(rows_loc + 255) / 256, 256, 0, stream>>>(
      ws->topk_ids, ws->topk_weights, rows_loc, peers, W, ep->rank, L.off_ids, L.off_weights);
  if ((code = cudaStreamWaitEvent(stream, ws->published_event, 0)) != cudaSuccess)
    return set_error(error, error_bytes, code, "join of the row all-gather");
  ep_signal_kernel<<<1, 32, 0, stream>>>(peers, W, ep->rank, L.off_flags_routing, epoch);
  ep_wait_kernel<<<1, 32, 0, stream>>>(mine, W, L.off_flags_routing, epoch, ws->status);
  if ((code = cudaGetLastError()) != cudaSuccess) return set_error(error, error_bytes, code, "routing exchange");
  count += 3;
  const int32_t* ids_all = reinterpret_cast<const int32_t*>(mine + L.off_ids);
  const float* weights_all = reinterpret_cast<const float*>(mine + L.off_weights);

  mark();
  // 3. plan over the global rows that land on this GPU's experts
  const int expert_lo = ep->rank * call.experts_local;
  const int expert_hi = expert_lo + call.experts_local;
  if ((code = launch_plan(ws, ids_all, rows, expert_lo, expert_hi, 0, stream, &count)) != cudaSuccess)
    return set_error(error, error_bytes, code, "dispatch plan");

  mark();
  // 4.-6. dispatch, products and row return, pipelined over `parts` ranges of the plan's tiles:
  //   inbound stream   rows of part k copied from this GPU's table of all activations into expert order
  //   caller's stream  gate_up and down products of part k once its rows are here
  //   outbound stream  weighted rows of part k stored to the GPUs that own their tokens
  const int parts = ws->ep_parts >= 1 && ws->ep_parts <= PrefillWorkspace::kMaxParts ? ws->ep_parts : 1;
  // Row return: with one part the down kernel stores its rows to their owners itself (fused_return); with the
  // pipeline a copy kernel on the outbound stream sends the rows of part k while part k + 1 is computed.
  const bool fused_return = parts == 1 && ws->ep_fused_return;
  // Dispatch: all rows are in this GPU's table since the flags of step 2, in global token order, so with one
  // part the gate_up kernel gathers them itself as on one GPU; otherwise a copy kernel puts them in expert order.
  const bool fused_dispatch = parts == 1 && ws->ep_fused_dispatch;
  EpPointers local_blocks{};      // block q of this GPU's table: the tokens of rank q
  for (int q = 0; q < W; ++q) local_blocks.region[q] = mine + static_cast<size_t>(q) * T_loc * kHidden * 2;
  const int part_blocks = min(((max_tiles_for(T) / parts + 1) * kTileRows + 7) / 8, 2 * ws->sm_count);
  cudaStream_t inbound = ws->inbound_stream, outbound = ws->outbound_stream;
  if ((code = cudaEventRecord(ws->plan_event, stream)) != cudaSuccess ||
      (code = cudaStreamWaitEvent(inbound, ws->plan_event, 0)) != cudaSuccess ||
      (code = cudaStreamWaitEvent(outbound, ws->plan_event, 0)) != cudaSuccess)
    return set_error(error, error_bytes, code, "fork of the dispatch / return streams");
  for (int k = 0; k < parts && !fused_dispatch; ++k) {
    ep_gather_rows_kernel<<<part_blocks, 256, 0, inbound>>>(local_blocks, L.off_h2, T_loc, ws->sorted_rows,
                                                            ws->expert_offsets, ws->tile_row0, ws->tile_count,
                                                            k, parts, ws->gathered);
    if ((code = cudaGetLastError()) != cudaSuccess) return set_error(error, error_bytes, code, "ep_gather_rows_kernel");
    if ((code = cudaEventRecord(ws->gathered_event[k], inbound)) != cudaSuccess)
      return set_error(error, error_bytes, code, "gathered event");
    ++count;
  }
  GroupedGemm g{};
  g.tile_expert = ws->tile_expert; g.tile_row0 = ws->tile_row0; g.tile_rows = ws->tile_rows;
  g.tile_count = ws->tile_count; g.max_tiles = max_tiles_for(T); g.dense_rows = 0;
  g.expert_base = expert_lo;
  g.parts = parts;
  TcExtra extra{};
  extra.status = ws->status; extra.sm_count = ws->sm_count;
  extra.a_rows = static_cast<uint64_t>(ws->capacity) * kTopK; extra.experts_in_b = call.experts_local;
  for (int k = 0; k < parts; ++k) {
    if (!fused_dispatch && (code = cudaStreamWaitEvent(stream, ws->gathered_event[k], 0)) != cudaSuccess)
      return set_error(error, error_bytes, code, "wait for gathered rows");
    if (k == 0) mark();
    g.part = k;
    g.a = ws->gathered; g.lda = kHidden; g.k = kHidden;
    g.gather_src = fused_dispatch ? reinterpret_cast<const __nv_bfloat16*>(mine + L.off_h2) : nullptr;
    extra.a_rows = fused_dispatch ? static_cast<uint64_t>(T) : static_cast<uint64_t>(ws->capacity) * kTopK;
    g.b0 = call.layer.expert_gate_up; g.b_expert_stride = static_cast<size_t>(2 * kInter) * kHidden;
    g.n = kInter; g.c = ws->expert_act; g.ldc = kInter;
    g.row_scale = nullptr; g.sorted_rows = ws->sorted_rows;
    if ((code = launch_grouped_gemm_tc(kGemmExpertGateUp, g, extra, stream)) != cudaSuccess)
      return set_error(error, error_bytes, code, "grouped gemm expert gate_up");
    g.gather_src = nullptr;
    extra.a_rows = static_cast<uint64_t>(ws->capacity) * kTopK;
    g.a = ws->expert_act; g.lda = kInter; g.k = kInter;
    g.b0 = call.layer.expert_down; g.b_expert_stride = static_cast<size_t>(kHidden) * kInter;
    g.n = kHidden; g.c = ws->expert_down; g.ldc = kHidden;
    g.row_scale = weights_all;
    if (fused_return) {
      // the down kernel's epilogue stores every weighted row where its token lives
      for (int q = 0; q < W; ++q) g.scatter_region[q] = ep->peers[q];
      g.scatter_offset = L.off_return;
      g.scatter_tokens_per_rank = T_loc;
    }
    if ((code = launch_grouped_gemm_tc(kGemmExpertDown, g, extra, stream)) != cudaSuccess)
      return set_error(error, error_bytes, code, "grouped gemm expert down");
    count += 2;
    if (fused_return) break;
    if ((code = cudaEventRecord(ws->computed_event[k], stream)) != cudaSuccess ||
        (code = cudaStreamWaitEvent(outbound, ws->computed_event[k], 0)) != cudaSuccess)
      return set_error(error, error_bytes, code, "computed event");
    ep_return_rows_kernel<<<part_blocks, 256, 0, outbound>>>(ws->expert_down, ws->sorted_rows, ws->expert_offsets,
                                                             ws->tile_row0, ws->tile_count, k, parts, peers,
                                                             L.off_return, T_loc);
    if ((code = cudaGetLastError()) != cudaSuccess) return set_error(error, error_bytes, code, "ep_return_rows_kernel");
    ++count;
  }
  mark();
  // all rows stored: raise this rank's flag on every GPU, then rejoin the caller's stream
  ep_signal_kernel<<<1, 32, 0, fused_return ? stream : outbound>>>(peers, W, ep->rank, L.off_flags_returned, epoch);
  if ((code = cudaGetLastError()) != cudaSuccess) return set_error(error, error_bytes, code, "row return");
  ++count;
  if (!fused_return &&
      ((code = cudaEventRecord(ws->returned_event, outbound)) != cudaSuccess ||
       (code = cudaStreamWaitEvent(stream, ws->returned_event, 0)) != cudaSuccess))
    return set_error(error, error_bytes, code, "join of the return stream");

  mark();
  // 7. the shared expert's output is needed from here on
  if ((code = cudaStreamWaitEvent(stream, ws->join_event, 0)) != cudaSuccess)
    return set_error(error, error_bytes, code, "join of the shared-expert stream");

  // 8. combine, second half: wait for all eight rows of every local token, sum, add
  ep_wait_kernel<<<1, 32, 0, stream>>>(mine, W, L.off_flags_returned, epoch, ws->status);
  combine_kernel<<<T_loc, 256, 0, stream>>>(reinterpret_cast<const __nv_bfloat16*>(mine + L.off_return), nullptr,
                                            ws->shared_scaled, static_cast<const __nv_bfloat16*>(call.residual),
                                            static_cast<__nv_bfloat16*>(call.out),
                                            dbg ? static_cast<__nv_bfloat16*>(dbg->routed) : nullptr,
                                            static_cast<const __nv_bfloat16*>(call.next_norm_weight),
                                            static_cast<__nv_bfloat16*>(call.next_norm_out), call.eps);
  if ((code = cudaGetLastError()) != cudaSuccess) return set_error(error, error_bytes, code, "combine_kernel");
  count += 2;
  mark();
  if (dbg != nullptr) {
    auto copy = [&](void* dst, const void* src, size_t bytes) {
      if (dst != nullptr) return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToDevice, stream);
      return cudaSuccess;
    };
    code = copy(dbg->topk_ids, ws->topk_ids, static_cast<size_t>(rows_loc) * 4);
    if (code == cudaSuccess) code = copy(dbg->topk_scores, ws->topk_scores, static_cast<size_t>(rows_loc) * 4);
    if (code == cudaSuccess) code = copy(dbg->shared_scaled, ws->shared_scaled, static_cast<size_t>(T_loc) * kHidden * 2);
    if (code == cudaSuccess) code = copy(dbg->expert_counts, ws->expert_counts, kExperts * 4);
    if (code != cudaSuccess) return set_error(error, error_bytes, code, "cudaMemcpyAsync debug views");
  }
  *launches = count;
  return AIMA_MOE_OK;
}

}  // namespace aima
