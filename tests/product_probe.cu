// Test entries for the tensor-core product kernels, launched as the library launches them but with every operand and the
// limit of their waits given by the host: a dense product, and the expert products in the one-SM and in the two-SM form.
#include "grouped_gemm_tc.cu"

namespace {

aima::TcExtra extra_for(int sm_count, int* status, unsigned long long limit_ns, bool pair) {
  aima::TcExtra extra{};
  extra.status = status;
  extra.sm_count = sm_count;
  extra.experts_in_b = 1;
  extra.pair = pair;
  extra.wait_limit_ns = limit_ns;
  return extra;
}

}  // namespace

// Pointers of one MoE half: x [tokens, 2048], weights of `experts` experts, the plan of `rows` routed rows, their weights by
// flat index, the shared expert's matrices and its gate per token; outputs in the plan's order and by token.
struct Operands {
  const __nv_bfloat16 *x, *gate_up, *down, *shared_gate, *shared_up, *shared_down;
  const int *tile_expert, *tile_row0, *tile_rows, *tile_count, *sorted_rows;
  const float *row_scale, *shared_scale;
  __nv_bfloat16 *act, *out, *shared_act, *shared_out;
  long long tokens, rows, experts, max_tiles;
};

extern "C" __attribute__((visibility("default"))) int run_dense(const void* a, const void* b, void* d, int m, int n, int k,
                                                                int sm_count, int* status, unsigned long long limit_ns) {
  aima::GroupedGemm g{};
  g.max_tiles = (m + 127) / 128;
  g.dense_rows = m;
  g.a = static_cast<const __nv_bfloat16*>(a);
  g.lda = g.k = k;
  g.b0 = static_cast<const __nv_bfloat16*>(b);
  g.n = g.ldc = n;
  g.c = static_cast<__nv_bfloat16*>(d);
  aima::TcExtra extra = extra_for(sm_count, status, limit_ns, true);
  extra.a_rows = m;
  return static_cast<int>(aima::launch_grouped_gemm_tc(aima::kGemmPlain, g, extra, nullptr));
}

// gate_up of the routed rows, gathered by token; with_shared: of the shared expert's rows too, in the same launch (two-SM)
// or in one of its own (one-SM)
extern "C" __attribute__((visibility("default"))) int run_gate_up(const Operands* o, int pair, int with_shared, int sm_count,
                                                                  int* status, unsigned long long limit_ns) {
  aima::GroupedGemm g{};
  g.tile_expert = o->tile_expert;
  g.tile_row0 = o->tile_row0;
  g.tile_rows = o->tile_rows;
  g.tile_count = o->tile_count;
  g.max_tiles = static_cast<int>(o->max_tiles);
  g.gather_src = o->x;
  g.lda = g.k = 2048;
  g.b0 = o->gate_up;
  g.b_expert_stride = static_cast<size_t>(2) * 512 * 2048;
  g.n = g.ldc = 512;
  g.c = o->act;
  g.sorted_rows = o->sorted_rows;
  aima::TcExtra extra = extra_for(sm_count, status, limit_ns, pair != 0);
  extra.a_rows = o->tokens;
  extra.experts_in_b = static_cast<int>(o->experts);
  if (pair != 0 && with_shared != 0)
    extra.shared = aima::SharedProblem{static_cast<int>(o->tokens), o->x, o->shared_gate, o->shared_up, o->shared_act, nullptr};
  cudaError_t code = aima::launch_grouped_gemm_tc(aima::kGemmExpertGateUp, g, extra, nullptr);
  if (code != cudaSuccess || pair != 0 || with_shared == 0) return static_cast<int>(code);
  aima::GroupedGemm s{};
  s.max_tiles = static_cast<int>((o->tokens + 127) / 128);
  s.dense_rows = static_cast<int>(o->tokens);
  s.a = o->x;
  s.lda = s.k = 2048;
  s.b0 = o->shared_gate;
  s.b1 = o->shared_up;
  s.n = s.ldc = 512;
  s.c = o->shared_act;
  extra.experts_in_b = 1;
  return static_cast<int>(aima::launch_grouped_gemm_tc(aima::kGemmSharedGateUp, s, extra, nullptr));
}

// down of what run_gate_up wrote, weighted
extern "C" __attribute__((visibility("default"))) int run_down(const Operands* o, int pair, int sm_count, int* status,
                                                               unsigned long long limit_ns) {
  aima::GroupedGemm g{};
  g.tile_expert = o->tile_expert;
  g.tile_row0 = o->tile_row0;
  g.tile_rows = o->tile_rows;
  g.tile_count = o->tile_count;
  g.max_tiles = static_cast<int>(o->max_tiles);
  g.a = o->act;
  g.lda = g.k = 512;
  g.b0 = o->down;
  g.b_expert_stride = static_cast<size_t>(2048) * 512;
  g.n = g.ldc = 2048;
  g.c = o->out;
  g.row_scale = o->row_scale;
  g.sorted_rows = o->sorted_rows;
  aima::TcExtra extra = extra_for(sm_count, status, limit_ns, pair != 0);
  extra.a_rows = o->rows;
  extra.experts_in_b = static_cast<int>(o->experts);
  if (pair != 0)
    extra.shared = aima::SharedProblem{static_cast<int>(o->tokens), o->shared_act, o->shared_down, nullptr, o->shared_out, o->shared_scale};
  cudaError_t code = aima::launch_grouped_gemm_tc(aima::kGemmExpertDown, g, extra, nullptr);
  if (code != cudaSuccess || pair != 0) return static_cast<int>(code);
  aima::GroupedGemm s{};
  s.max_tiles = static_cast<int>((o->tokens + 127) / 128);
  s.dense_rows = static_cast<int>(o->tokens);
  s.a = o->shared_act;
  s.lda = s.k = 512;
  s.b0 = o->shared_down;
  s.n = s.ldc = 2048;
  s.c = o->shared_out;
  s.row_scale = o->shared_scale;
  extra.a_rows = o->tokens;
  extra.experts_in_b = 1;
  return static_cast<int>(aima::launch_grouped_gemm_tc(aima::kGemmSharedDown, s, extra, nullptr));
}
