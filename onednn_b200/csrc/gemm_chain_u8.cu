// 8-bit GEMM with a post-op chain, u8 dst
#include "gemm_chain.cuh"

namespace qmm {
QMM_GEMM_CHAIN(u8, DT_U8)
} // namespace qmm
