// Test entries for the two-SM product kernel with a limit on its waits that the host chooses: a dense product, and a gate_up
// product over tiles whose rows it gathers by token.
#include "grouped_gemm_tc.cu"

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
  aima::TcExtra extra{};
  extra.status = status;
  extra.sm_count = sm_count;
  extra.a_rows = m;
  extra.experts_in_b = 1;
  extra.pair = true;
  extra.wait_limit_ns = limit_ns;
  return static_cast<int>(aima::launch_grouped_gemm_tc(aima::kGemmPlain, g, extra, nullptr));
}

// weights [experts, 2 * 512, 2048], rows of x [tokens, 2048] picked by sorted_rows >> 3, output [rows, 512]
extern "C" __attribute__((visibility("default"))) int run_gate_up(const void* x, int tokens, const void* weights, int experts,
                                                                  const int* tile_expert, const int* tile_row0,
                                                                  const int* tile_rows, const int* tile_count, int max_tiles,
                                                                  const int* sorted_rows, void* out, int sm_count, int* status,
                                                                  unsigned long long limit_ns) {
  aima::GroupedGemm g{};
  g.tile_expert = tile_expert;
  g.tile_row0 = tile_row0;
  g.tile_rows = tile_rows;
  g.tile_count = tile_count;
  g.max_tiles = max_tiles;
  g.gather_src = static_cast<const __nv_bfloat16*>(x);
  g.lda = g.k = 2048;
  g.b0 = static_cast<const __nv_bfloat16*>(weights);
  g.b_expert_stride = static_cast<size_t>(2) * 512 * 2048;
  g.n = g.ldc = 512;
  g.c = static_cast<__nv_bfloat16*>(out);
  g.sorted_rows = sorted_rows;
  aima::TcExtra extra{};
  extra.status = status;
  extra.sm_count = sm_count;
  extra.a_rows = tokens;
  extra.experts_in_b = experts;
  extra.pair = true;
  extra.wait_limit_ns = limit_ns;
  return static_cast<int>(aima::launch_grouped_gemm_tc(aima::kGemmExpertGateUp, g, extra, nullptr));
}
