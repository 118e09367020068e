// The launch plans behind C functions, for tests that have no GPU.
#include "../../cute_mma_b200/csrc/prism_plan.h"

extern "C" int plan_fwd_bn(int M, int N, int K, int gs, int bias, int sms) { return prism::fwd_default_bn(M, N, K, gs, bias != 0, sms); }
extern "C" double plan_fwd_us(int M, int N, int K, int bn, int bias, int sms) { return prism::fwd_tile_us(M, N, K, bn, bias != 0, sms / 2); }
extern "C" void plan_db(int M, int N, int K, int gs, int sms, const int* cfg, int* out) {
  prism::DbPlan p;
  prism::db_plan(M, N, K, gs, sms, cfg, &p);
  out[0] = p.bn; out[1] = p.splits; out[2] = p.tail_rows; out[3] = p.tail_splits;
}
extern "C" int plan_db_tma(int bn, int blocks, int bf16_silu) { return prism::db_tma_out(bn, blocks, bf16_silu != 0); }
extern "C" int plan_dadr_per_part(int M, int K, int G, int gs, int pairs, int slots) {
  return prism::dadr_groups_per_part(M, K, G, gs, pairs, slots);
}
