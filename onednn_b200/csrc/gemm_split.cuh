// The 8-bit GEMM for problems with too few tiles for the GPU: K is split over the CTAs of a cluster.
//
// One cluster of `splits` CTAs computes one tile of 128 dst columns x bt (32 to 128) dst rows, each CTA over a contiguous
// share of K, with the operands and roles of gemm_tc_kernel (dst^T in tensor memory: lane = dst column).  Each CTA then
// owns some of the tile's pieces of 8 rows: the epilogue warps send the other pieces of their partial sums to their owners
// with asynchronous stores that count themselves at the owner's barrier, and every owner adds the shares in rank order
// (integers exactly, floats in the same order every time) and runs the epilogue on its pieces.  No scratch in global
// memory, no second kernel.
//
// A src zero-point needs the weights' column sums.  They come from one more MMA per 32 k against a tile of ones (16
// columns of tensor memory), so the weights are read once and the memset and column-sum kernels before the GEMM are
// gone; each CTA's share of them is sent to every CTA of the cluster.
//
// What bounds these problems is the latency of a launch, of the first loads and of the exchange, and the bytes an SM has
// in flight: more CTAs with shorter shares of K shorten all but the first two.
#pragma once
#include "gemm_epilogue.cuh"

namespace qmm {

struct SplitParams {
    int bt; // dst rows per tile: 32, 64 or 128
    int splits; // CTAs per tile
    int stages, stage_bytes;
    int ones; // column sums are wanted (src zero-point)
    int off_ones, off_recv, off_colsum, off_bars; // shared memory, from its 1024-byte aligned start
    int tmem_cols;
    uint32_t idesc_ones;
};

namespace {

constexpr int SPLIT_EPI_WARPS = 8;
constexpr int SPLIT_THREADS = 64 + 32 * SPLIT_EPI_WARPS;
constexpr int SPLIT_MAX_STAGES = 12, SPLIT_MAX = 8;
constexpr int PIECE_BYTES = 8 * BT_N * 4; // sums of 8 rows x 128 columns
constexpr int ONES_COLS = 16, ONES_BYTES = ONES_COLS * BKB;

__device__ __forceinline__ uint32_t map_to_rank(uint32_t addr, int rank) { // the same place in another CTA of the cluster
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void send_v4(uint32_t addr, uint32_t x, uint32_t y, uint32_t z, uint32_t w, uint32_t bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(addr), "r"(x),
                 "r"(y), "r"(z), "r"(w), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void send_b32(uint32_t addr, uint32_t x, uint32_t bar) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(addr), "r"(x), "r"(bar) : "memory");
}

template <int KIND, bool CHAIN, int DSTT = -1>
__global__ void __launch_bounds__(SPLIT_THREADS, 2)
gemm_split_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmS, const __grid_constant__ MatmulArgs a,
        const __grid_constant__ TcParams tp, const __grid_constant__ SplitParams sp) {
    constexpr bool INT = KIND == 1;
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint64_t *full_bar = (uint64_t *)(smem + sp.off_bars);
    uint64_t *empty_bar = full_bar + SPLIT_MAX_STAGES, *acc_bar = empty_bar + SPLIT_MAX_STAGES, *recv_bar = acc_bar + 1;
    uint32_t *tmem_base_slot = (uint32_t *)(recv_bar + 1);
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    const int splits = sp.splits, tile = (int)blockIdx.x / splits, rank = (int)blockIdx.x - tile * splits;
    const int m_tile = (tile % tp.num_m_tiles) * sp.bt, n_tile = (tile / tp.num_m_tiles) * BT_N;
    const int kb0 = tp.num_k_blocks * rank / splits, kb1 = tp.num_k_blocks * (rank + 1) / splits;
    // pieces of 8 rows that exist, and which of them this CTA owns: piece p belongs to rank p * splits / pieces
    const int pieces = (int)(min((int64_t)sp.bt, a.M - m_tile) + 7) / 8;
    const int own0 = (rank * pieces + splits - 1) / splits, own1 = ((rank + 1) * pieces + splits - 1) / splits;

    if (threadIdx.x == 0) {
        for (int s = 0; s < sp.stages; ++s) {
            ptx::mbar_init(&full_bar[s], 1);
            ptx::mbar_init(&empty_bar[s], 1);
        }
        ptx::mbar_init(acc_bar, 1);
        ptx::mbar_init(recv_bar, 1);
        ptx::fence_barrier_init();
        ptx::mbar_arrive_expect_tx(recv_bar, (uint32_t)splits * ((own1 - own0) * PIECE_BYTES + (sp.ones ? BT_N * 4 : 0)));
        ptx::prefetch_tensormap(&tmW);
        ptx::prefetch_tensormap(&tmS);
    }
    if (warp == 1) ptx::tmem_alloc(tmem_base_slot, sp.tmem_cols);
    if (sp.ones) {
        for (int i = threadIdx.x; i < ONES_BYTES / 4; i += SPLIT_THREADS) ((uint32_t *)(smem + sp.off_ones))[i] = 0x01010101u;
        ptx::fence_proxy_async(); // the MMAs read them through the asynchronous proxy
    }
    ptx::tc_fence_before_sync();
    __syncthreads();
    ptx::tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_base_slot;
    if (splits > 1) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); // recv_bar is ready
    // a programmatic dependent of whatever precedes it on the stream: what is above runs under the predecessor's end
    ptx::grid_dependency_wait();
    bool late = false; // the wait for the other CTAs' sums ran out

    if (warp == 0) {
        // ------------------------------------------------ TMA producer
        if (ptx::elect_one()) {
            int s = 0;
            uint32_t ph = 1;
            for (int kb = kb0; kb < kb1; ++kb) {
                if (!ptx::mbar_wait(&empty_bar[s], ph)) { atomicExch(a.status, 5); break; }
                uint8_t *sw = smem + s * sp.stage_bytes, *ss = sw + BT_N * BKB;
                ptx::mbar_arrive_expect_tx(&full_bar[s], sp.stage_bytes);
                if (tp.w_kmajor) ptx::tma_load_2d(sw, &tmW, &full_bar[s], kb * BKB, n_tile);
                else ptx::tma_load_2d(sw, &tmW, &full_bar[s], n_tile, kb * BKB);
                ptx::tma_load_2d(ss, &tmS, &full_bar[s], kb * BKB, m_tile);
                if (++s == sp.stages) { s = 0; ph ^= 1; }
            }
        }
        __syncwarp();
        // the successor may start (its set-up allocates tensor memory: every CTA of this grid has its own by now)
        asm volatile("griddepcontrol.launch_dependents;");
        if (splits > 1) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    } else if (warp == 1) {
        // ------------------------------------------------ MMA issuer
        if (ptx::elect_one()) {
            int s = 0;
            uint32_t ph = 0;
            const uint64_t od = ptx::smem_desc_sw128(ptx::smem_u32(smem + sp.off_ones), 0, 1024);
            for (int kb = kb0; kb < kb1; ++kb) {
                if (!ptx::mbar_wait(&full_bar[s], ph)) { atomicExch(a.status, 5); break; }
                ptx::tc_fence_after_sync();
                const uint32_t sw = ptx::smem_u32(smem + s * sp.stage_bytes), ss = sw + BT_N * BKB;
                const uint64_t wd0 = tp.w_kmajor ? ptx::smem_desc_sw128(sw, 0, 1024) : ptx::smem_desc_sw128(sw, 128 * BKB, 1024);
                const uint64_t wstep = tp.w_kmajor ? (uint64_t)(UMMA_K >> 4) : (uint64_t)((UMMA_K * 128) >> 4);
                const uint64_t sd0 = ptx::smem_desc_sw128(ss, 0, 1024);
#pragma unroll
                for (int kk = 0; kk < BKB / UMMA_K; ++kk) {
                    ptx::mma_ss<KIND>(tmem_base, wd0 + kk * wstep, sd0 + (uint64_t)(kk * (UMMA_K >> 4)), tp.idesc, kb != kb0 || kk != 0);
                    if (INT && sp.ones) ptx::mma_ss<KIND>(tmem_base + sp.bt, wd0 + kk * wstep, od, sp.idesc_ones, kb != kb0 || kk != 0);
                }
                ptx::tc_commit(&empty_bar[s]);
                if (++s == sp.stages) { s = 0; ph ^= 1; }
            }
            ptx::tc_commit(acc_bar);
        }
        __syncwarp();
        if (splits > 1) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    } else {
        // ------------------------------------------------ epilogue warps: two per lane quarter, pieces in turn
        const int lane_base = (warp % 4) * 32, half = (warp - 2) / 4;
        const int64_t n = n_tile + lane_base + lane;
        const TensorTerms tt = load_tensor_terms<INT>(a, tp);
        ColTerms ct = load_col_terms<INT>(a, tp, n); // in flight while waiting for the MMAs
        if constexpr (CHAIN) {
            // binary operands with a value per element (a residual): ask L2 for this warp's part
            for (int i = 0; i < a.n_po; ++i) {
                const PostOpArg &e = a.po[i];
                if (e.kind != PO_BINARY || e.sm == 0 || e.sn != 1 || n_tile + lane_base >= a.N) continue;
                const int esz = (e.src1_dt == DT_F32 || e.src1_dt == DT_S32) ? 4 : (e.src1_dt == DT_BF16 || e.src1_dt == DT_F16) ? 2 : 1;
                for (int r = own0 * 8 + lane; r < own1 * 8 && m_tile + r < a.M; r += 32)
                    asm volatile("prefetch.global.L2 [%0];" ::"l"((const char *)e.src1 + ((m_tile + r) * e.sm + n_tile + lane_base) * esz));
            }
        }
        const uint32_t recv = ptx::smem_u32(smem + sp.off_recv), colsum_at = ptx::smem_u32(smem + sp.off_colsum), bar = ptx::smem_u32(recv_bar);
        const bool done = ptx::mbar_wait(acc_bar, 0);
        if (!done) atomicExch(a.status, 5);
        ptx::tc_fence_after_sync();
        __syncwarp();
        if (splits > 1) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        const uint32_t lanes = tmem_base + ((uint32_t)lane_base << 16);
        const int col = lane_base + lane, most = (pieces + splits - 1) / splits; // pieces of a rank, at most
        for (int p = half; p < pieces; p += 2) {
            uint32_t r[8];
            ptx::tmem_ld_32x8(lanes + p * 8, r);
            ptx::tmem_ld_wait();
            const int owner = p * splits / pieces, idx = p - (owner * pieces + splits - 1) / splits;
            const uint32_t at = map_to_rank(recv + (rank * most + idx) * PIECE_BYTES + col * 16, owner), ob = map_to_rank(bar, owner);
            send_v4(at, r[0], r[1], r[2], r[3], ob);
            send_v4(at + BT_N * 16, r[4], r[5], r[6], r[7], ob);
        }
        if (INT && sp.ones && half == 0) {
            uint32_t r[4];
            ptx::tmem_ld_32x4(lanes + sp.bt, r); // every column holds the sum
            ptx::tmem_ld_wait();
            for (int q = 0; q < splits; ++q) send_b32(map_to_rank(colsum_at + (rank * BT_N + col) * 4, q), r[0], map_to_rank(bar, q));
        }
        late = !ptx::mbar_wait(recv_bar, 0);
        if (late) atomicExch(a.status, 5);
        if (INT && sp.ones && n < a.N) {
            int sum = 0;
            for (int q = 0; q < splits; ++q) sum += ((const int *)(smem + sp.off_colsum))[q * BT_N + col];
            const int zs = ((const int *)a.src_zp.ptr)[0];
            ct.zs_colsum = zs * sum - (int)a.K * zs * ct.wei_zp;
        }
#pragma unroll 1
        for (int p = own0 + half; p < own1; p += 2) {
            const uint4 *part = reinterpret_cast<const uint4 *>(smem + sp.off_recv + (p - own0) * PIECE_BYTES) + col;
            uint4 x = part[0], y = part[BT_N];
            for (int q = 1; q < splits; ++q) {
                part += most * (PIECE_BYTES / 16);
                const uint4 u = part[0], v = part[BT_N];
                if constexpr (INT) {
                    x.x += u.x; x.y += u.y; x.z += u.z; x.w += u.w;
                    y.x += v.x; y.y += v.y; y.z += v.z; y.w += v.w;
                } else {
                    auto add = [](uint32_t &s, uint32_t t) { s = __float_as_uint(__uint_as_float(s) + __uint_as_float(t)); };
                    add(x.x, u.x); add(x.y, u.y); add(x.z, u.z); add(x.w, u.w);
                    add(y.x, v.x); add(y.y, v.y); add(y.z, v.z); add(y.w, v.w);
                }
            }
            const uint32_t r[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
            epilogue_rows_any<INT, CHAIN, 8, DSTT>(a, tp, tt, ct, r, m_tile + p * 8, n);
        }
    }

    // ---------------------------------------------------- teardown
    ptx::tc_fence_before_sync();
    const bool some_late = __syncthreads_or(late);
    if (warp == 1) {
        __syncwarp();
        ptx::tc_fence_after_sync();
        ptx::tmem_dealloc(tmem_base, sp.tmem_cols);
        __syncwarp();
    }
    if (some_late && splits > 1) ptx::outlast_cluster(recv_bar);
}

template <int KIND, bool CHAIN, int DSTT = -1>
int launch_split_cfg(const CUtensorMap &mw, const CUtensorMap &ms, const MatmulArgs &a, const TcParams &tp, const SplitParams &sp, cudaStream_t st) {
    auto kern = gemm_split_kernel<KIND, CHAIN, DSTT>;
    static std::atomic<unsigned long long> configured; // one per instantiation of this template
    if (!opt_in_dynamic_smem(kern, 227 * 1024, configured)) return 5;
    cudaLaunchConfig_t cfg {};
    cfg.gridDim = dim3((unsigned)(tp.num_m_tiles * tp.num_n_tiles * sp.splits));
    cfg.blockDim = dim3((unsigned)SPLIT_THREADS);
    cfg.dynamicSmemBytes = (size_t)(sp.off_bars + (2 * SPLIT_MAX_STAGES + 2) * 8 + 16 + 1024);
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)sp.splits;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    if (cudaLaunchKernelEx(&cfg, kern, mw, ms, a, tp, sp) != cudaSuccess) return 5;
    count_launch("gemm_split");
    return 0;
}

} // namespace

} // namespace qmm
