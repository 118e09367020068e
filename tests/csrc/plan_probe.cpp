// The launch plans behind C functions, for tests that have no GPU.
#include "../../cute_mma_b200/csrc/prism_plan.h"

extern "C" int plan_fwd_bn(int M, int N, int K, int gs, int bias, int sms) { return prism::fwd_default_bn(M, N, K, gs, bias != 0, sms); }
extern "C" double plan_fwd_us(int M, int N, int K, int bn, int bias, int sms) { return prism::fwd_tile_us(M, N, K, bn, bias != 0, sms / 2); }
