// 8-bit GEMM with a post-op chain, s32 dst
#include "gemm_chain.cuh"

namespace qmm {
QMM_GEMM_CHAIN(s32, DT_S32)
} // namespace qmm
