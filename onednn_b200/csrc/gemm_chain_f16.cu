// 8-bit GEMM with a post-op chain, f16 dst
#include "gemm_chain.cuh"

namespace qmm {
QMM_GEMM_CHAIN(f16, DT_F16)
} // namespace qmm
