// 8-bit GEMM with a post-op chain, f32 dst
#include "gemm_chain.cuh"

namespace qmm {
QMM_GEMM_CHAIN(f32, DT_F32)
} // namespace qmm
