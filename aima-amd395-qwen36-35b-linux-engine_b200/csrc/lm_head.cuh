// LM head with a certified top-1 (see lm_head.cu).
#pragma once

#include "../../include/aima_moe.h"
#include "common.cuh"

namespace aima {

constexpr int kLmMaxScanBlocks = 256;

// State of one launch beside the published result.
struct LmHeadTop {
  unsigned long long best;          // largest exact logit: order-preserving bits, then the complement of the token id
  uint32_t blocks_done;             // blocks of the candidate kernel that have finished
  // a bounded wait of the scan ran out.  Any block of the scan may set it, so none of them clears it: that is done when the
  // head is built and by the last block of the candidate kernel, after it has published it.
  uint32_t failed;
};

// What read_result copies to the host.
struct LmHeadWire {
  aima_moe_lm_head_result result;
  uint32_t failed;
};

struct LmHeadBuffers {
  int8_t* q_weight;                 // [rows, 2048]
  float* scales;                    // [rows]
  float* residual_l2;               // [rows]
  LmHeadWire* wire;                 // device copy of the result
  LmHeadTop* top;
  float* partial;                   // [kLmMaxScanBlocks] per-block maxima of the lower bounds
};

cudaError_t lm_head_quantize(const void* weight, int rows, int8_t* q_weight, float* scales, float* residual_l2,
                             cudaStream_t stream);

// Enqueues the scan with the bounds, and the candidates with their exact logits and arg-max.
cudaError_t lm_head_certify(const LmHeadBuffers& buffers, const void* weight, const void* hidden, float* logits,
                            int rows, int sm_count, cudaStream_t stream, int* launches);

}  // namespace aima
