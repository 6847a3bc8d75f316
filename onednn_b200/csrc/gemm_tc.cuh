// "cuda:tcgen05" GEMM for 8-bit operands: int8 (u8/s8 x u8/s8 -> s32
// accumulate) and fp8 (e4m3/e5m2 -> f32 accumulate).
//
// The kernel computes dst^T tiles: the WEIGHTS are the A operand of
// tcgen05.mma (128 dst columns = the 128 TMEM lanes) and the SRC rows are the
// B operand (BT_M dst rows = TMEM columns).  An epilogue thread therefore owns
// one dst column n and reads consecutive rows m from TMEM: the 32 lanes of a
// warp hold 32 adjacent columns, so every global access of the epilogue (dst
// stores, binary post-op operands) is coalesced without a shared-memory
// transpose, and per-column terms (weight scales, bias, zero-point
// compensation) live in registers for the whole tile.
//
// One persistent CTA per SM walks the tiles.  Roles:
//   warp 0     TMA producer: weights tile ([128 k x 128 n] for N-contiguous
//              `ab` weights, [128 n x 128 B of k] for `ba`) and src tile
//              [BT_M rows x 128 B of k] into a ring of 128B-swizzled stages
//   warp 1     issues tcgen05.mma (M=128, N=BT_M, K=32 per instruction) into
//              one of two TMEM accumulator buffers, commits to mbarriers
//   warps 2-9  epilogue (two warps per TMEM lane quarter, each half of the
//              rows): zero-point compensation, scales, bias, post-op chain,
//              dst scale / zero-point, saturating store; overlaps the next
//              tile's multiplication
// Epilogue arithmetic follows the reference (ref_matmul_int8.cpp:241-304,
// ref_matmul.cpp:218-332): integer sums are exact, so int8 results equal the
// reference's bit for bit; fp8 differs only by the f32 summation order.
#pragma once
#include "gemm_split.cuh"

namespace qmm {

namespace {

// Epilogue warps: 8 keep up with the MMAs when the epilogue is scale + bias + store; a post-op chain
// is latency-bound per element: 16 warps (at 96 registers) hide a third more of it than 8, and 24
// (at 72 registers) another 6 % (int8 post-op workload: 12 warps 150 us, 16: 133, 20: 132, 24: 124-127).
#ifndef QMM_CHAIN_EPI_WARPS
#define QMM_CHAIN_EPI_WARPS 24
#endif
#ifndef QMM_CHAIN_CR
#define QMM_CHAIN_CR 8
#endif
constexpr int epi_warps(bool chain) { return chain ? QMM_CHAIN_EPI_WARPS : 8; }
constexpr int num_threads(bool chain) { return 64 + 32 * epi_warps(chain); }

template <int BT_M, int STAGES>
struct SmemLayout {
    static constexpr int W_BYTES = BT_N * BKB;
    static constexpr int S_BYTES = BT_M * BKB;
    static constexpr int STAGE_BYTES = W_BYTES + S_BYTES;
    static constexpr int BAR_OFFSET = STAGES * STAGE_BYTES;
    static constexpr int TOTAL = BAR_OFFSET + 256 + 1024; // barriers + alignment slack
};

template <int KIND, int BT_M, int STAGES, bool CHAIN, int DSTT = -1>
__global__ void __launch_bounds__(num_threads(CHAIN), 1)
gemm_tc_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmS,
        const __grid_constant__ MatmulArgs a, const __grid_constant__ TcParams tp) {
    using L = SmemLayout<BT_M, STAGES>;
    constexpr bool INT = KIND == 1;
    constexpr int ACC_STAGES = 2;
    constexpr uint32_t TMEM_COLS = ACC_STAGES * BT_M; // 128, 256 or 512, a power of two
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint64_t *full_bar = (uint64_t *)(smem + L::BAR_OFFSET);
    uint64_t *empty_bar = full_bar + STAGES;
    uint64_t *tmem_full = empty_bar + STAGES;
    uint64_t *tmem_empty = tmem_full + ACC_STAGES;
    uint32_t *tmem_base_slot = (uint32_t *)(tmem_empty + ACC_STAGES);
    volatile int *abort_flag = (volatile int *)(tmem_base_slot + 1);

    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    const int num_tiles = tp.num_m_tiles * tp.num_n_tiles;

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            ptx::mbar_init(&full_bar[s], 1);
            ptx::mbar_init(&empty_bar[s], 1);
        }
        for (int s = 0; s < ACC_STAGES; ++s) {
            ptx::mbar_init(&tmem_full[s], 1);
            ptx::mbar_init(&tmem_empty[s], epi_warps(CHAIN)); // one arrival per epilogue warp
        }
        *abort_flag = 0;
        ptx::fence_barrier_init();
        ptx::prefetch_tensormap(&tmW);
        ptx::prefetch_tensormap(&tmS);
    }
    if (warp == 1) ptx::tmem_alloc(tmem_base_slot, TMEM_COLS);
    ptx::tc_fence_before_sync();
    __syncthreads();
    ptx::tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_base_slot;

    // A programmatic dependent of whatever precedes it on the stream: the set-up above runs under the predecessor's end.
    // (After a pre-kernel, which was launched when everything before it had ended, only the epilogue warps wait.)
    if (!tp.after_prekernel) ptx::grid_dependency_wait();

    // Tile order: the m index runs fastest, so the CTAs working at any moment
    // share a few weight column blocks and sweep the whole src once per block.
    if (warp == 0) {
        // ------------------------------------------------ TMA producer
        if (ptx::elect_one()) {
            uint32_t it = 0;
            for (int tile = blockIdx.x; tile < num_tiles && !*abort_flag; tile += gridDim.x) {
                const int m0 = (tile % tp.num_m_tiles) * BT_M;
                const int n0 = (tile / tp.num_m_tiles) * BT_N;
                for (int kb = 0; kb < tp.num_k_blocks; ++kb, ++it) {
                    const int s = it % STAGES;
                    const uint32_t ph = (it / STAGES) & 1;
                    if (!ptx::mbar_wait(&empty_bar[s], ph ^ 1)) { *abort_flag = 1; atomicExch(a.status, 5); break; }
                    uint8_t *sw = smem + s * L::STAGE_BYTES, *ss = sw + L::W_BYTES;
                    ptx::mbar_arrive_expect_tx(&full_bar[s], L::STAGE_BYTES);
                    if (tp.w_kmajor) ptx::tma_load_2d(sw, &tmW, &full_bar[s], kb * BKB, n0);
                    else ptx::tma_load_2d(sw, &tmW, &full_bar[s], n0, kb * BKB);
                    ptx::tma_load_2d(ss, &tmS, &full_bar[s], kb * BKB, m0);
                }
            }
        }
        __syncwarp();
        // the successor may start (its set-up allocates tensor memory: every CTA of this grid has its own by now)
        asm volatile("griddepcontrol.launch_dependents;");
    } else if (warp == 1) {
        // ------------------------------------------------ MMA issuer
        // (an elected thread: an MMA then takes about 12 cycles to issue; under a predicate computed from the lane
        // index, which the hardware cannot know to be one lane, about 115 - nearly twice what a 128-row MMA runs)
        if (ptx::elect_one()) {
            uint32_t it = 0, acc_it = 0;
            for (int tile = blockIdx.x; tile < num_tiles && !*abort_flag; tile += gridDim.x, ++acc_it) {
                const int as = acc_it % ACC_STAGES;
                const uint32_t aph = (acc_it / ACC_STAGES) & 1;
                if (!ptx::mbar_wait(&tmem_empty[as], aph ^ 1)) { *abort_flag = 1; atomicExch(a.status, 5); break; }
                ptx::tc_fence_after_sync();
                const uint32_t tmem_d = tmem_base + as * BT_M;
                bool failed = false;
                for (int kb = 0; kb < tp.num_k_blocks; ++kb, ++it) {
                    const int s = it % STAGES;
                    const uint32_t ph = (it / STAGES) & 1;
                    if (!ptx::mbar_wait(&full_bar[s], ph)) { failed = true; break; }
                    ptx::tc_fence_after_sync();
                    const uint32_t sw = ptx::smem_u32(smem + s * L::STAGE_BYTES), ss = sw + L::W_BYTES;
                    // weights: MN-major when N-contiguous (one 128-byte row per k), K-major for `ba`; src
                    // rows: K-major.  One thread issues: descriptors are built once per stage and advanced
                    // by a constant in their start-address field (16-byte units).
                    const uint64_t wd0 = tp.w_kmajor ? ptx::smem_desc_sw128(sw, 0, 1024) : ptx::smem_desc_sw128(sw, 128 * BKB, 1024);
                    const uint64_t wstep = tp.w_kmajor ? (uint64_t)(UMMA_K >> 4) : (uint64_t)((UMMA_K * 128) >> 4);
                    const uint64_t sd0 = ptx::smem_desc_sw128(ss, 0, 1024);
#pragma unroll
                    for (int kk = 0; kk < BKB / UMMA_K; ++kk)
                        ptx::mma_ss<KIND>(tmem_d, wd0 + kk * wstep, sd0 + (uint64_t)(kk * (UMMA_K >> 4)), tp.idesc, (kb | kk) != 0);
                    ptx::tc_commit(&empty_bar[s]); // stage reusable once these MMAs have read it
                }
                if (failed) { *abort_flag = 1; atomicExch(a.status, 5); break; }
                ptx::tc_commit(&tmem_full[as]); // accumulator complete
            }
        }
    } else {
        // ------------------------------------------------ epilogue warps
        const int lane_base = (warp % 4) * 32; // TMEM lanes (dst columns) of this warp
        constexpr int GROUPS = epi_warps(CHAIN) / 4; // warps that share a quarter of the lanes
        constexpr int ROWS_PER_WARP = BT_M / (CHAIN ? 1 : GROUPS);
        const int group = (warp - 2) / 4;
        // without a chain each warp takes a contiguous share of the tile's rows; with one, the warps
        // of a lane quarter take the tile's 8-row pieces in turn (any number of warps divides them)
        const int row_base = CHAIN ? 0 : group * ROWS_PER_WARP;
        const TensorTerms tt = load_tensor_terms<INT>(a, tp);
        // the zero-point sums come from the kernel launched before this one, which runs beside this
        // kernel's set-up and first mainloop: only the epilogue warps wait for it
        if (tp.after_prekernel) ptx::grid_dependency_wait();
        uint32_t acc_it = 0;
        for (int tile = blockIdx.x; tile < num_tiles && !*abort_flag; tile += gridDim.x, ++acc_it) {
            const int as = acc_it % ACC_STAGES;
            const uint32_t aph = (acc_it / ACC_STAGES) & 1;
            const int64_t m_tile = (int64_t)(tile % tp.num_m_tiles) * BT_M + row_base;
            const int64_t n = (int64_t)(tile / tp.num_m_tiles) * BT_N + lane_base + lane;
            const ColTerms ct = load_col_terms<INT>(a, tp, n); // in flight while waiting for the MMAs
            if constexpr (CHAIN) {
                // Operands of binary post-ops that have a value per dst element (a residual) are read once,
                // row by row, in the middle of the chain: a miss there stalls the whole piece.  While the
                // tile is being multiplied, ask L2 for this warp's part of them (its rows x its 32 columns).
                for (int i = 0; i < a.n_po; ++i) {
                    const PostOpArg &e = a.po[i];
                    if (e.kind != PO_BINARY || e.sm == 0 || e.sn != 1) continue;
                    const int esz = (e.src1_dt == DT_F32 || e.src1_dt == DT_S32) ? 4 : (e.src1_dt == DT_BF16 || e.src1_dt == DT_F16) ? 2 : 1;
                    const int64_t nq = (int64_t)(tile / tp.num_m_tiles) * BT_N + lane_base;
                    if (nq >= a.N) continue;
                    constexpr int CRP = QMM_CHAIN_CR, PIECES_P = BT_M / CRP;
                    for (int idx = lane; idx < (PIECES_P + GROUPS - 1) / GROUPS * CRP; idx += 32) {
                        const int piece = group + GROUPS * (idx / CRP);
                        const int64_t m = m_tile + piece * CRP + idx % CRP;
                        if (piece < PIECES_P && m < a.M)
                            asm volatile("prefetch.global.L2 [%0];" ::"l"((const char *)e.src1 + (m * e.sm + nq) * esz));
                    }
                }
            }
            if (!ptx::mbar_wait(&tmem_full[as], aph)) { *abort_flag = 1; atomicExch(a.status, 5); break; }
            ptx::tc_fence_after_sync();
#ifdef QMM_PROFILE
            if (tp.mainloop_only == 1) { // results are not stored
                ptx::tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) ptx::mbar_arrive(&tmem_empty[as]);
                continue;
            }
#endif
            if constexpr (CHAIN) {
                // With a post-op chain the code of 32 unrolled rows exceeds the instruction cache, so the
                // rows go through a rolled loop of 8-row pieces (8 independent dependency chains each).
                constexpr int CR = QMM_CHAIN_CR; // rows per piece: 4 leave too few independent chains (152 us on the int8 post-op workload), 16 overflow the instruction cache (175 us), 8: 134 us
                constexpr int PIECES = BT_M / CR;
#pragma unroll 1
                for (int c = group; c < PIECES; c += GROUPS) {
                    uint32_t r[CR];
                    ptx::tmem_ld_32xn(tmem_base + ((uint32_t)lane_base << 16) + as * BT_M + c * CR, r);
                    const int64_t m0 = m_tile + c * CR;
                    ptx::tmem_ld_wait();
                    if (c + GROUPS >= PIECES) { // accumulator fully read: hand the buffer back
                        ptx::tc_fence_before_sync();
                        __syncwarp();
                        if (lane == 0) ptx::mbar_arrive(&tmem_empty[as]);
                    }
#ifdef QMM_PROFILE
                    if (tp.mainloop_only == 2) continue; // TMEM reads only
#endif
                    if (m0 < a.M) epilogue_rows_any<INT, CHAIN, CR, DSTT>(a, tp, tt, ct, r, m0, n);
                }
            } else {
#pragma unroll 1
                for (int c = 0; c < ROWS_PER_WARP / 32; ++c) {
                    uint32_t r[32];
                    ptx::tmem_ld_32x32(tmem_base + ((uint32_t)lane_base << 16) + as * BT_M + row_base + c * 32, r);
                    ptx::tmem_ld_wait();
                    if (c == ROWS_PER_WARP / 32 - 1) { // accumulator fully read: hand the buffer back
                        ptx::tc_fence_before_sync();
                        __syncwarp();
                        if (lane == 0) ptx::mbar_arrive(&tmem_empty[as]);
                    }
                    const int64_t m0 = m_tile + c * 32;
#ifdef QMM_PROFILE
                    if (tp.mainloop_only == 2) continue; // TMEM reads only
#endif
                    if (m0 < a.M) epilogue_rows_any<INT, CHAIN, 32>(a, tp, tt, ct, r, m0, n);
                }
            }
        }
    }

    // ---------------------------------------------------- teardown
    if (!CHAIN && a.peers.count) __threadfence_system(); // this thread's peer stores, before the CTA is counted
    ptx::tc_fence_before_sync();
    __syncthreads();
    if (warp == 1) {
        __syncwarp();
        ptx::tc_fence_after_sync();
        ptx::tmem_dealloc(tmem_base, TMEM_COLS);
    }
    if (!CHAIN && a.peers.count && threadIdx.x == 0) {
        // the last CTA to get here tells every rank that this rank's block is complete
        if (atomicAdd(a.peers.done, 1u) == gridDim.x - 1) {
            __threadfence_system();
            for (int r = 0; r < a.peers.world; ++r) {
                volatile unsigned *f = a.peers.flags[r] + a.peers.rank;
                *f = a.peers.epoch;
            }
            *a.peers.done = 0u;
        }
    }
}

template <int KIND, int BT_M, int STAGES, bool CHAIN, int DSTT = -1>
int launch_cfg(const CUtensorMap &mw, const CUtensorMap &ms, const MatmulArgs &a, TcParams tp, int sm_count,
        cudaStream_t st) {
    using L = SmemLayout<BT_M, STAGES>;
    auto kern = gemm_tc_kernel<KIND, BT_M, STAGES, CHAIN, DSTT>;
    static std::atomic<unsigned long long> configured; // one per instantiation of this template
    if (!opt_in_dynamic_smem(kern, L::TOTAL, configured)) return 5;
    const int tiles = tp.num_m_tiles * tp.num_n_tiles;
    const int grid = tiles < sm_count ? tiles : sm_count;
    cudaLaunchConfig_t cfg {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)num_threads(CHAIN));
    cfg.dynamicSmemBytes = (size_t)L::TOTAL;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    // (long problems gain nothing from it and lost 1.5 %: fp8 4096 x 4096 x 14336 211.6 -> 214.9 us)
    cfg.numAttrs = tiles <= 2 * sm_count || tp.after_prekernel ? 1 : 0;
    if (cudaLaunchKernelEx(&cfg, kern, mw, ms, a, tp) != cudaSuccess) return 5;
    count_launch("gemm_tc");
    return 0;
}

} // namespace

// Kernels with a post-op chain, instantiated per dst data type, each type in a translation unit of its own
// (gemm_chain_*.cu).  `sp`: split K; nullptr: the persistent kernel with tiles of `bt` (256 or 128) dst rows.
#define QMM_GEMM_CHAIN_ARGS \
    bool int_path, int bt, const CUtensorMap &mw, const CUtensorMap &ms, const MatmulArgs &a, const TcParams &tp, const SplitParams *sp, \
            int sm_count, cudaStream_t st
int launch_gemm_chain_s8(QMM_GEMM_CHAIN_ARGS);
int launch_gemm_chain_u8(QMM_GEMM_CHAIN_ARGS);
int launch_gemm_chain_bf16(QMM_GEMM_CHAIN_ARGS);
int launch_gemm_chain_f16(QMM_GEMM_CHAIN_ARGS);
int launch_gemm_chain_f32(QMM_GEMM_CHAIN_ARGS);
int launch_gemm_chain_s32(QMM_GEMM_CHAIN_ARGS);

} // namespace qmm
