// gate_up in the two-SM form with the way its rows come in chosen by the test: TMA gathers or cp.async.
#include "product_probe.cu"

extern "C" __attribute__((visibility("default"))) int run_gate_up_fed(const Operands* o, int fetch, int with_shared, int sm_count,
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
  aima::TcExtra extra = extra_for(sm_count, status, limit_ns, true);
  extra.fetch = fetch != 0;
  extra.a_rows = o->tokens;
  extra.experts_in_b = static_cast<int>(o->experts);
  if (with_shared != 0)
    extra.shared = aima::SharedProblem{static_cast<int>(o->tokens), o->x, o->shared_gate, o->shared_up, o->shared_act, nullptr};
  return static_cast<int>(aima::launch_grouped_gemm_tc(aima::kGemmExpertGateUp, g, extra, nullptr));
}
