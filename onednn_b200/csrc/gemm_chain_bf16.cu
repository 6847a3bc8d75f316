// 8-bit GEMM with a post-op chain, bf16 dst
#include "gemm_chain.cuh"

namespace qmm {
QMM_GEMM_CHAIN(bf16, DT_BF16)
} // namespace qmm
