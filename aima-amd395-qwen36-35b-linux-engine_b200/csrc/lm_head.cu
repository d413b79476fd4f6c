// LM head with a certified top-1: a row-wise int8 copy of the vocabulary matrix is scanned for
// every token (one byte per weight instead of two), Cauchy-Schwarz bounds around the approximate
// logits decide which rows can still win, and only those are evaluated exactly in BF16.
//
// Follows NativeLmHeadStore::build / quantize_lm_head_rowwise_kernel
// (native/src/native_lm_head.hip.cpp:53-115, 126-176), the row-wise int8 GEMV of
// benchmarks/shape-lab/four_layer_mini_engine.py:1223-1258 and launch_native_lm_head_certificate
// (native/src/native_lm_head_certificate.hip.cpp:44-275): same bounds, same outward rounding,
// same capacity of 1024 candidates, same tie rule (equal logits -> lowest token id).
// The scan is the bandwidth-bound kernel: rows x 2048 bytes per token.
#include "lm_head.cuh"

#include <math_constants.h>

namespace aima {
namespace {

constexpr int kLmThreads = 256;
constexpr int kResidualSafetyUlps = 8;
constexpr int kHiddenSafetyUlps = 4;

// ---------------------------------------------------------------------------
// Build: q = clamp(rint(w / scale)), scale = max|w| * fl(1/127), residual_l2 = ||w - q * scale||_2
// rounded up by 8 ULPs (the arithmetic of native/src/native_lm_head.hip.cpp:53-115).
// One warp per row, 16-byte loads: lane l holds elements 256 g + 8 l + j (g, j in 0..7), writes its
// eight int8 results of a group with one 8-byte store.  The reference sums the squared residuals in
// FP64 as 256 partials (partial t = columns t, t + 256, ... in that order) folded by halving; a lane
// holds all eight columns of partials 8 l .. 8 l + 7, so the halvings of width 128 .. 8 are the lane
// butterfly of each partial and the last three are ((q0+q4)+(q2+q6))+((q1+q5)+(q3+q7)).
// ---------------------------------------------------------------------------
constexpr int kQuantizeWarps = 8;
__global__ void __launch_bounds__(kQuantizeWarps * 32)
lm_head_quantize_kernel(const __nv_bfloat16* __restrict__ source, int8_t* __restrict__ q_weight,
                        float* __restrict__ scales, float* __restrict__ residual_l2, int rows) {
  const int lane = threadIdx.x & 31;
  const int row = blockIdx.x * kQuantizeWarps + (threadIdx.x >> 5);
  if (row >= rows) return;
  const size_t base = static_cast<size_t>(row) * kHidden;
  float v[64];
  float largest = 0.0f;
#pragma unroll
  for (int g = 0; g < 8; ++g) {
    unpack8(__ldg(reinterpret_cast<const uint4*>(source + base + 256 * g) + lane), v + 8 * g);
#pragma unroll
    for (int j = 0; j < 8; ++j) largest = fmaxf(largest, fabsf(v[8 * g + j]));
  }
#pragma unroll
  for (int s = 16; s >= 1; s >>= 1) largest = fmaxf(largest, __shfl_xor_sync(0xffffffffu, largest, s));
  const float scale = __fmul_rn(fmaxf(largest, 1.0e-12f), 1.0f / 127.0f);   // multiplication by the rounded reciprocal
  double partial[8] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
#pragma unroll
  for (int g = 0; g < 8; ++g) {
    uint32_t packed[2] = {0u, 0u};
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float value = v[8 * g + j];
      const int quantized = static_cast<int>(fminf(127.0f, fmaxf(-127.0f, rintf(__fdiv_rn(value, scale)))));
      packed[j >> 2] |= (static_cast<uint32_t>(quantized) & 0xffu) << (8 * (j & 3));
      const double residual = static_cast<double>(__fsub_rn(value, __fmul_rn(static_cast<float>(quantized), scale)));
      partial[j] = __dadd_rn(partial[j], __dmul_rn(residual, residual));
    }
    *reinterpret_cast<uint2*>(q_weight + base + 256 * g + 8 * lane) = make_uint2(packed[0], packed[1]);
  }
#pragma unroll
  for (int j = 0; j < 8; ++j) {
#pragma unroll
    for (int s = 16; s >= 1; s >>= 1) partial[j] = __dadd_rn(partial[j], __shfl_xor_sync(0xffffffffu, partial[j], s));
  }
  if (lane == 0) {
    const double total = __dadd_rn(__dadd_rn(__dadd_rn(partial[0], partial[4]), __dadd_rn(partial[2], partial[6])),
                                   __dadd_rn(__dadd_rn(partial[1], partial[5]), __dadd_rn(partial[3], partial[7])));
    float norm = static_cast<float>(sqrt(total));
    for (int step = 0; step < kResidualSafetyUlps; ++step) norm = nextafterf(norm, CUDART_INF_F);
    scales[row] = scale;
    residual_l2[row] = norm;
  }
}

// ---------------------------------------------------------------------------
// Scan: approximate[row] = scale[row] * sum_c q[row, c] * hidden[c], FP32.
// Lane l owns the 16-byte pieces l, l + 32, l + 64, l + 96 of the
// row (64 weights), multiplies them in ascending order into one accumulator, then the warp
// butterfly (16, 8, 4, 2, 1).  The lane's 64 hidden values stay in registers for all its rows.
// int8 -> FP32 without the conversion pipe: the byte, biased by 128, is placed in the mantissa
// of 2^23 and 2^23 + 128 is subtracted -- exact.
// ---------------------------------------------------------------------------
__device__ __forceinline__ float byte_to_float(uint32_t biased_word, uint32_t selector) {
  return __fsub_rn(__uint_as_float(__byte_perm(biased_word, 0x4B000000u, selector)), 8388736.0f);
}

__device__ __forceinline__ float fma_word(uint32_t word, const float* x, float acc) {
  const uint32_t biased = word ^ 0x80808080u;
  acc = __fmaf_rn(byte_to_float(biased, 0x7540u), x[0], acc);
  acc = __fmaf_rn(byte_to_float(biased, 0x7541u), x[1], acc);
  acc = __fmaf_rn(byte_to_float(biased, 0x7542u), x[2], acc);
  acc = __fmaf_rn(byte_to_float(biased, 0x7543u), x[3], acc);
  return acc;
}

// ||hidden||_2 in FP64, rounded to FP32 and up 4 ULPs.  The order is that of 256 partials (partial t = elements t, t + 256,
// ... in that order) folded by halving; lane l holds partials l + 32 j, so the halvings of width 128, 64 and 32 are its own
// and the rest are lane exchanges.  Every warp of the scan evaluates it for itself while its first rows are on their way.
__device__ __forceinline__ float hidden_norm_in_warp(const __nv_bfloat16* __restrict__ hidden, int lane) {
  double q[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    q[j] = 0.0;
#pragma unroll
    for (int i = 0; i < kHidden / 256; ++i) {
      const double value = static_cast<double>(__bfloat162float(hidden[256 * i + 32 * j + lane]));
      q[j] = __dadd_rn(q[j], __dmul_rn(value, value));
    }
  }
#pragma unroll
  for (int width = 4; width >= 1; width >>= 1) {
#pragma unroll
    for (int j = 0; j < width; ++j) q[j] = __dadd_rn(q[j], q[j + width]);
  }
#pragma unroll
  for (int s = 16; s >= 1; s >>= 1) q[0] = __dadd_rn(q[0], __shfl_xor_sync(0xffffffffu, q[0], s));
  float norm = static_cast<float>(sqrt(q[0]));
  for (int step = 0; step < kHiddenSafetyUlps; ++step) norm = nextafterf(norm, CUDART_INF_F);
  return norm;
}

__device__ __forceinline__ float row_error(float residual, float hidden_l2) {
  return nextafterf(__fmul_rn(residual, hidden_l2), CUDART_INF_F);
}

constexpr int kScanWarps = 12;
constexpr int kScanBuffers = 2;                     // per warp
constexpr int kScanRows = 4;                        // per buffer: one 8 KB copy
constexpr int kScanBufferBytes = kScanRows * kHidden;
constexpr int kScanSmemBytes = kScanWarps * kScanBuffers * (kScanBufferBytes + 8) + 16;
static_assert(32 % kScanRows == 0 && kScanRows % 2 == 0, "logits are finished 32 rows at a time");

// The vocabulary is cut into one contiguous run of rows per warp of the chip.  A warp streams its run four rows (8 KB) at
// a time through two buffers of its own with 1-D bulk copies -- no register holds a load in flight, so twelve warps keep
// up to 192 KB per SM on the way -- and reads them back with conflict-free 16-byte loads.  Logits and bounds are finished
// 32 rows at a time, one per lane.  Bound by HBM; the arithmetic (three instructions per weight, 42 us over the chip at
// 248 320 rows) runs beside it.
__global__ void __launch_bounds__(kScanWarps * 32, 1)
lm_head_scan_kernel(const int8_t* __restrict__ q_weight, const float* __restrict__ scales,
                    const float* __restrict__ residual_l2, const __nv_bfloat16* __restrict__ hidden,
                    float* __restrict__ logits, LmHeadWire* wire, LmHeadTop* top,
                    float* __restrict__ partial, int rows) {
  extern __shared__ __align__(16) uint8_t scan_smem[];
  __shared__ float warp_max[kScanWarps];
  // the kernel after this one is placed while its last blocks drain (see pdl_enter)
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int lane = threadIdx.x & 31;
  const int warp = __shfl_sync(0xffffffffu, static_cast<int>(threadIdx.x >> 5), 0);
  uint8_t* buffers = scan_smem + warp * kScanBuffers * kScanBufferBytes;
  const uint32_t bars = smem_u32(scan_smem + kScanWarps * kScanBuffers * kScanBufferBytes) + warp * kScanBuffers * 8;
  volatile int* abort_flag = reinterpret_cast<volatile int*>(scan_smem + kScanWarps * kScanBuffers * (kScanBufferBytes + 8));
  if (lane == 0) {
    for (int b = 0; b < kScanBuffers; ++b) mbar_init(bars + 8 * b, 1);
    mbar_fence_init();
  }
  if (threadIdx.x == 0) *abort_flag = 0;
  __syncthreads();

  const int warps_total = gridDim.x * kScanWarps;
  const int run = ((rows + warps_total - 1) / warps_total + 1) & ~1;
  const long long first = static_cast<long long>(blockIdx.x * kScanWarps + warp) * run;
  const int lo = static_cast<int>(first < rows ? first : rows);
  const int hi = min(rows, lo + run);
  const int steps = (hi - lo + kScanRows - 1) / kScanRows;
  auto request = [&](int p) {
    const int row = lo + kScanRows * p;
    const uint32_t bytes = min(kScanRows, hi - row) * kHidden;
    const int b = p % kScanBuffers;
    if (elect_one()) {
      mbar_arrive_expect_tx(bars + 8 * b, bytes);
      bulk_g2s(smem_u32(buffers + b * kScanBufferBytes), q_weight + static_cast<size_t>(row) * kHidden, bytes, bars + 8 * b);
    }
    __syncwarp();
  };
  for (int p = 0; p < min(steps, kScanBuffers); ++p) request(p);

  float x[64];
#pragma unroll
  for (int piece = 0; piece < 4; ++piece) {
    // 16 weights of piece (32 piece + lane): hidden elements 16 (32 piece + lane) .. + 15
    const uint4* src = reinterpret_cast<const uint4*>(hidden) + 2 * (32 * piece + lane);
    unpack8(__ldg(src), x + 16 * piece);
    unpack8(__ldg(src + 1), x + 16 * piece + 8);
  }
  const float hidden_l2 = hidden_norm_in_warp(hidden, lane);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    wire->result.hidden_l2 = hidden_l2;
    wire->result.candidate_count = 0;
    wire->result.overflow = 0;
    top->best = 0;
    top->blocks_done = 0;
  }

  float best_lower = -CUDART_INF_F;
  float mine = 0.0f, scale = 0.0f, residual = 0.0f;
  for (int p = 0; p < steps; ++p) {
    const int row = lo + kScanRows * p;
    if (((kScanRows * p) & 31) == 0) {          // 32 rows from here on: this lane finishes row + lane
      const int own = row + lane;
      if (own < hi) { scale = __ldg(scales + own); residual = __ldg(residual_l2 + own); }
    }
    const int b = p % kScanBuffers;
    if (!mbar_wait_bounded_warp(bars + 8 * b, (p / kScanBuffers) & 1, abort_flag)) {
      // read_result then reports the timeout; the copies under way have to land before the block leaves
      if (lane == 0) top->failed = 1;
      volatile int ignore = 0;
      for (int q = p; q < min(steps, p + kScanBuffers); ++q)
        mbar_wait_bounded_warp(bars + 8 * (q % kScanBuffers), (q / kScanBuffers) & 1, &ignore);
      break;
    }
    // (fewer rows left than the buffer holds: the rest of it are older rows, whose sums nobody takes)
#pragma unroll
    for (int r = 0; r < kScanRows; r += 2) {
      const uint4* qa = reinterpret_cast<const uint4*>(buffers + b * kScanBufferBytes + r * kHidden) + lane;
      const uint4* qb = qa + kHidden / 16;
      float acc_a = 0.0f, acc_b = 0.0f;
#pragma unroll
      for (int piece = 0; piece < 4; ++piece) {
        const uint4 wa = qa[32 * piece], wb = qb[32 * piece];
        acc_a = fma_word(wa.x, x + 16 * piece, acc_a);
        acc_b = fma_word(wb.x, x + 16 * piece, acc_b);
        acc_a = fma_word(wa.y, x + 16 * piece + 4, acc_a);
        acc_b = fma_word(wb.y, x + 16 * piece + 4, acc_b);
        acc_a = fma_word(wa.z, x + 16 * piece + 8, acc_a);
        acc_b = fma_word(wb.z, x + 16 * piece + 8, acc_b);
        acc_a = fma_word(wa.w, x + 16 * piece + 12, acc_a);
        acc_b = fma_word(wb.w, x + 16 * piece + 12, acc_b);
      }
      if (r + 2 == kScanRows) {
        __syncwarp();                        // every lane has read the buffer
        if (p + kScanBuffers < steps) request(p + kScanBuffers);
      }
      acc_a = butterfly_sum(acc_a);
      acc_b = butterfly_sum(acc_b);
      if (lane == ((kScanRows * p + r) & 31)) mine = acc_a;
      if (lane == ((kScanRows * p + r + 1) & 31)) mine = acc_b;
    }
    if (((kScanRows * (p + 1)) & 31) == 0 || p + 1 == steps) {
      const int own = lo + ((kScanRows * p) & ~31) + lane;
      if (own < min(hi, row + kScanRows)) {
        const float logit = __fmul_rn(mine, scale);
        logits[own] = logit;
        best_lower = fmaxf(best_lower, nextafterf(__fsub_rn(logit, row_error(residual, hidden_l2)), -CUDART_INF_F));
      }
    }
  }
#pragma unroll
  for (int s = 16; s >= 1; s >>= 1) best_lower = fmaxf(best_lower, __shfl_xor_sync(0xffffffffu, best_lower, s));
  if (lane == 0) warp_max[warp] = best_lower;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < kScanWarps; ++w) best_lower = fmaxf(best_lower, warp_max[w]);
    partial[blockIdx.x] = best_lower;
  }
}

// Every row whose upper bound reaches the largest lower bound is a candidate.  The warp that finds one evaluates its
// exact BF16 logit at once, straight from the raw matrix (no gathered copy, no list): the canonical warp dot, rounded to
// BF16 like the reference's N = 1 GEMV provider.  The exact logit replaces the approximate one in `logits`; the largest --
// equal ones: the lowest token id -- is kept in one 64-bit word, and the last block to finish publishes it.
__global__ void __launch_bounds__(kLmThreads)
lm_head_candidates_kernel(const __nv_bfloat16* __restrict__ weight, const __nv_bfloat16* __restrict__ hidden,
                          const float* __restrict__ residual_l2, const float* __restrict__ partial, int partials,
                          LmHeadWire* wire, LmHeadTop* top, float* logits, int rows) {
  __shared__ float reduction[kLmThreads / 32];
  const int lane = threadIdx.x & 31;
  pdl_enter();
  const int row = blockIdx.x * kLmThreads + threadIdx.x;
  const float logit = row < rows ? logits[row] : 0.0f;
  const float residual = row < rows ? residual_l2[row] : 0.0f;
  const float hidden_l2 = wire->result.hidden_l2;
  float largest = -CUDART_INF_F;
  for (int i = threadIdx.x; i < partials; i += kLmThreads) largest = fmaxf(largest, partial[i]);
#pragma unroll
  for (int s = 16; s >= 1; s >>= 1) largest = fmaxf(largest, __shfl_xor_sync(0xffffffffu, largest, s));
  if (lane == 0) reduction[threadIdx.x >> 5] = largest;
  __syncthreads();
#pragma unroll
  for (int w = 0; w < kLmThreads / 32; ++w) largest = fmaxf(largest, reduction[w]);
  if (blockIdx.x == 0 && threadIdx.x == 0) wire->result.maximum_lower_bound = largest;

  bool candidate = false;
  if (row < rows) {
    const float upper = nextafterf(__fadd_rn(logit, row_error(residual, hidden_l2)), CUDART_INF_F);
    candidate = !(upper < largest);
  }
  unsigned pending = __ballot_sync(0xffffffffu, candidate);
  while (pending != 0u) {
    const int owner = __ffs(pending) - 1;
    pending &= pending - 1u;
    const int token = __shfl_sync(0xffffffffu, row, owner);
    uint32_t slot = 0;
    if (lane == 0) slot = atomicAdd(&wire->result.candidate_count, 1u);
    slot = __shfl_sync(0xffffffffu, slot, 0);
    if (slot >= AIMA_MOE_LM_HEAD_CANDIDATES) {
      if (lane == 0) wire->result.overflow = 1;
      continue;
    }
    const uint4* wrow = reinterpret_cast<const uint4*>(weight + static_cast<size_t>(token) * kHidden) + lane;
    const uint4* xrow = reinterpret_cast<const uint4*>(hidden) + lane;
    uint4 w[kHidden / 256];
#pragma unroll
    for (int i = 0; i < kHidden / 256; ++i) w[i] = __ldg(wrow + i * 32);
    float acc = 0.0f;
#pragma unroll
    for (int i = 0; i < kHidden / 256; ++i) {
      float xf[8];
      unpack8(__ldg(xrow + i * 32), xf);
      acc = fma8(xf, w[i], acc);
    }
    const float value = round_bf16(butterfly_sum(acc));
    if (lane == 0) {
      logits[token] = value;
      if (value > -CUDART_INF_F) {       // neither -inf nor NaN ever wins
        const uint32_t bits = __float_as_uint(value == 0.0f ? 0.0f : value);      // -0 ties with +0
        const uint32_t key = (bits & 0x80000000u) ? ~bits : (bits | 0x80000000u);
        atomicMax(&top->best, (static_cast<unsigned long long>(key) << 32) | (0xffffffffu - static_cast<uint32_t>(token)));
      }
    }
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0 && atomicAdd(&top->blocks_done, 1u) + 1 == gridDim.x) {
    __threadfence();
    const unsigned long long best = atomicAdd(&top->best, 0ull);
    const uint32_t token = best != 0 ? 0xffffffffu - static_cast<uint32_t>(best) : 0u;
    wire->result.exact_top1_token_id = token;
    wire->result.exact_top1_logit = best != 0 ? __ldcg(logits + token) : -CUDART_INF_F;
    wire->failed = top->failed;
    top->failed = 0;
  }
}

}  // namespace

cudaError_t lm_head_quantize(const void* weight, int rows, int8_t* q_weight, float* scales, float* residual_l2,
                             cudaStream_t stream) {
  if (rows <= 0) return cudaSuccess;
  lm_head_quantize_kernel<<<(rows + kQuantizeWarps - 1) / kQuantizeWarps, kQuantizeWarps * 32, 0, stream>>>(
      static_cast<const __nv_bfloat16*>(weight), q_weight, scales, residual_l2, rows);
  return cudaGetLastError();
}

cudaError_t lm_head_certify(const LmHeadBuffers& b, const void* weight, const void* hidden, float* logits,
                            int rows, int sm_count, cudaStream_t stream, int* launches) {
  const __nv_bfloat16* h = static_cast<const __nv_bfloat16*>(hidden);
  cudaError_t code = opt_in_dynamic_smem<lm_head_scan_kernel>(kScanSmemBytes);
  if (code != cudaSuccess) return code;
  const int blocks = sm_count < kLmMaxScanBlocks ? sm_count : kLmMaxScanBlocks;
  lm_head_scan_kernel<<<blocks, kScanWarps * 32, kScanSmemBytes, stream>>>(b.q_weight, b.scales, b.residual_l2, h, logits,
                                                                           b.wire, b.top, b.partial, rows);
  code = cudaGetLastError();
  const PdlScope pdl_scope(true);
  if (code == cudaSuccess)
    code = launch_pdl(lm_head_candidates_kernel, dim3((rows + kLmThreads - 1) / kLmThreads), dim3(kLmThreads), 0, stream,
                      static_cast<const __nv_bfloat16*>(weight), h, static_cast<const float*>(b.residual_l2),
                      static_cast<const float*>(b.partial), blocks, b.wire, b.top, logits, rows);
  *launches = 2;
  return code;
}

}  // namespace aima
