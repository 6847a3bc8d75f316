// 8-bit GEMM with a post-op chain, s8 dst
#include "gemm_chain.cuh"

namespace qmm {
QMM_GEMM_CHAIN(s8, DT_S8)
} // namespace qmm
