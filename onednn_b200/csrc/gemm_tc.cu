// Host side of the "cuda:tcgen05" GEMM for 8-bit operands (kernels: gemm_tc.cuh, gemm_split.cuh): the choice of tiles,
// the kernels that sum the weights' columns and the src rows, and the allocation-free entry point.
#include <mutex>
#include <string>

#include "gemm_tc.cuh"
#include "objects.hpp"

namespace qmm {

namespace {

// ---- zero-point compensation terms (int8 path) ----------------------------
// colsum[n] += sum over a chunk of k of w[k][n] (colsum zeroed beforehand).
// A block covers 128 columns x `kchunk` rows with 8 warps: a lane owns four
// neighbouring columns, the warps take every 8th row, the block adds its
// warps' sums in shared memory and issues one atomic add per column (integer
// addition: the result does not depend on the order).  VEC: weights are
// N-contiguous bytes with a 4-byte aligned pitch, so a lane's four columns are
// one 32-bit load and dp4a adds each byte into its own sum.
template <bool VEC>
__global__ void __launch_bounds__(256) colsum_kernel(const __grid_constant__ MatmulArgs a, int32_t *colsum, int kchunk) {
    asm volatile("griddepcontrol.launch_dependents;"); // the GEMM may start; its epilogue warps wait for this grid
    __shared__ int part[8][128];
    const int lane = threadIdx.x & 31, kl = threadIdx.x >> 5;
    const int64_t n0 = (int64_t)blockIdx.x * 128 + lane * 4;
    const int64_t k0 = (int64_t)blockIdx.y * kchunk, k1 = min(a.K, k0 + kchunk);
    int s0 = 0, s1 = 0, s2 = 0, s3 = 0;
    if (VEC) {
        if (n0 < a.N) {
            const char *col = (const char *)a.wei + n0;
            if (a.wei_dt == DT_S8) {
#pragma unroll 4
                for (int64_t k = k0 + kl; k < k1; k += 8) {
                    const int v = *(const int *)(col + k * a.wei_sk);
                    s0 = __dp4a(v, 0x00000001, s0);
                    s1 = __dp4a(v, 0x00000100, s1);
                    s2 = __dp4a(v, 0x00010000, s2);
                    s3 = __dp4a(v, 0x01000000, s3);
                }
            } else {
#pragma unroll 4
                for (int64_t k = k0 + kl; k < k1; k += 8) {
                    const unsigned v = *(const unsigned *)(col + k * a.wei_sk);
                    s0 += v & 0xffu;
                    s1 += (v >> 8) & 0xffu;
                    s2 += (v >> 16) & 0xffu;
                    s3 += v >> 24;
                }
            }
        }
    } else {
        for (int64_t k = k0 + kl; k < k1; k += 8) {
            if (n0 + 0 < a.N) s0 += load_int(a.wei_dt, a.wei, k * a.wei_sk + (n0 + 0) * a.wei_sn);
            if (n0 + 1 < a.N) s1 += load_int(a.wei_dt, a.wei, k * a.wei_sk + (n0 + 1) * a.wei_sn);
            if (n0 + 2 < a.N) s2 += load_int(a.wei_dt, a.wei, k * a.wei_sk + (n0 + 2) * a.wei_sn);
            if (n0 + 3 < a.N) s3 += load_int(a.wei_dt, a.wei, k * a.wei_sk + (n0 + 3) * a.wei_sn);
        }
    }
    part[kl][lane * 4 + 0] = s0;
    part[kl][lane * 4 + 1] = s1;
    part[kl][lane * 4 + 2] = s2;
    part[kl][lane * 4 + 3] = s3;
    __syncthreads();
    if (threadIdx.x < 128) {
        const int64_t n = (int64_t)blockIdx.x * 128 + threadIdx.x;
        int s = 0;
#pragma unroll
        for (int w = 0; w < 8; ++w) s += part[w][threadIdx.x];
        if (n < a.N) atomicAdd(colsum + n, s);
    }
}
// rowsum[m] = sum_k s[m][k]; one warp per row
__global__ void rowsum_kernel(const __grid_constant__ MatmulArgs a, int32_t *rowsum) {
    asm volatile("griddepcontrol.launch_dependents;");
    const int64_t m = (int64_t)blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32;
    if (m >= a.M) return;
    int s = 0;
    for (int64_t k = threadIdx.x % 32; k < a.K; k += 32) s += load_int(a.src_dt, a.src, m * a.src_sm + k * a.src_sk);
    for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (threadIdx.x % 32 == 0) rowsum[m] = s;
}

// How a problem is cut.  splits = 0: the persistent kernel, dst rows per tile `bt` (256, 128 or 64); else a cluster of
// `splits` CTAs per tile of 32, 64 or 128 rows, `per_sm` CTAs sharing an SM's shared memory.
struct GemmPlan {
    int bt, splits, per_sm;
};

// CTAs that clusters of 1 to 8 can place on 148 SMs at a time (cudaOccupancyMaxActiveClusters), with one or two to an SM
const int cluster_places[2][SPLIT_MAX] = {{148, 148, 135, 132, 130, 132, 105, 120}, {296, 296, 279, 284, 280, 270, 259, 264}};

void split_smem(const GemmPlan &plan, bool ones, SplitParams &sp) {
    const int most = (plan.bt / 8 + plan.splits - 1) / plan.splits;
    const int fixed = (ones ? ONES_BYTES + plan.splits * BT_N * 4 : 0) + plan.splits * most * PIECE_BYTES;
    const int limit = (plan.per_sm == 2 ? 112 : 226) * 1024 - 1024 - 512; // alignment slack, barriers
    sp.stage_bytes = (BT_N + plan.bt) * BKB;
    sp.stages = (limit - fixed) / sp.stage_bytes;
    if (sp.stages > SPLIT_MAX_STAGES) sp.stages = SPLIT_MAX_STAGES;
    sp.off_ones = sp.stages * sp.stage_bytes;
    sp.off_recv = sp.off_ones + (ones ? ONES_BYTES : 0);
    sp.off_colsum = sp.off_recv + plan.splits * most * PIECE_BYTES;
    sp.off_bars = sp.off_colsum + (ones ? plan.splits * BT_N * 4 : 0);
}

// The choice between them is a model of a call's time in nanoseconds, fitted to 56 problems (M 1 to 3504, K 528 to 7824, N 720
// to 13968, every kind of epilogue) timed with up to 25 cuts each; the cut it picks is 3.6 % slower than the best one
// measured, on average.  With one tile per CTA a stage costs 89 + 2.3 bt (or, where fewer bytes are in flight, 203 per SM),
// the epilogue 33 a row of a CTA's share (67 with a post-op chain), the exchange 8 a row and 135 a CTA of the cluster, a second
// wave 4500; the persistent kernel's stages cost 133 + 1.7 bt (248 at least), its last tile's epilogue 20 a row, and
// separate column-sum kernels 4050.  (A second wave of clusters takes as long as the first: 144 CTAs in clusters of three, of which
// 135 find a place at a time, took 33.5 us for a chain 384 x 8192 x 2048 that two CTAs a tile do in 23.4.)  us a call, before -> now: int8 256 x 1024 x 1024 with a src zero-point 12.0 -> 6.1,
// int8 17 x 4096 x 11008 20.5 -> 13.5, fp8 161 x 576 x 1824 10.2 -> 5.1, chain 3 x 6512 x 2912 27 -> 9.3.
GemmPlan gemm_plan(int64_t M, int ntiles, int kblocks, int sm_count, bool chain, bool want_colsum, bool may_split) {
    if (sm_count < 1) sm_count = 148;
    GemmPlan best {128, 0, 1};
    int64_t cost = INT64_MAX;
    auto consider = [&](int bt, int splits, int per_sm) {
        const int64_t tiles = (int64_t)ntiles * ((M + bt - 1) / bt), rows = M < bt ? M : bt;
        int64_t ns = chain ? 2012 : 0;
        if (!splits) {
            int64_t tile = kblocks * (133 + 17 * bt / 10 < 248 ? 248 : 133 + 17 * bt / 10);
            if (chain && tile < 48 * rows) tile = 48 * rows;
            ns += 3270 + (want_colsum ? 4050 : 0) + (tiles + sm_count - 1) / sm_count * tile + 20 * rows;
        } else {
            const int64_t ctas = tiles * splits, places = (int64_t)cluster_places[per_sm - 1][splits - 1] * sm_count / 148;
            const int64_t waves = (ctas + places - 1) / (places ? places : 1);
            // CTAs that one SM runs: clusters that find no place wait for the end of a whole wave
            const int64_t busiest = (waves - 1) * per_sm + (ctas - (waves - 1) * places + sm_count - 1) / sm_count;
            const int64_t alone = 203 / (busiest < per_sm ? busiest : per_sm), full = 89 + 23 * bt / 10;
            ns += 4090 + (waves - 1) * 4530 + 135 * splits
                    + busiest * ((kblocks + splits - 1) / splits * (full > alone ? full : alone) + rows * (chain ? 67 : 33) / splits + (splits > 1 ? 8 * rows : 0));
        }
        if (ns < cost) { cost = ns; best = GemmPlan {bt, splits, per_sm}; }
    };
    for (int bt = chain ? 128 : 64; bt <= 256; bt *= 2) consider(bt, 0, 1);
    for (int s = 1; may_split && s <= SPLIT_MAX && s <= kblocks; ++s) {
        consider(32, s, 2);
        consider(64, s, 1);
        consider(64, s, 2);
        consider(128, s, 1);
    }
    return best;
}

} // namespace

size_t gemm_tc_scratch_bytes(int64_t M, int64_t N) { return (size_t)(M + N) * sizeof(int32_t) + 256; }

bool gemm_tc_pointers_ok(const MatmulArgs &a) {
    return ((uintptr_t)a.src % 16 == 0) && ((uintptr_t)a.wei % 16 == 0);
}

// `scratch`: gemm_tc_scratch_bytes(M, N) bytes of device memory, needed only
// when zero-points are present.
int launch_gemm_tc(const MatmulArgs &a_in, void *scratch, int sm_count, cudaStream_t st) {
#ifdef QMM_PROFILE
    MatmulArgs a = a_in;
    if (getenv("ONEDNN_CUDA_TC_MAINLOOP_ONLY") && atoi(getenv("ONEDNN_CUDA_TC_MAINLOOP_ONLY")) == 4)
        for (int i = 0; i < a.n_po; ++i) a.po[i].sm = a.po[i].sn = 0;
#else
    const MatmulArgs &a = a_in;
#endif
    if (a.M == 0 || a.N == 0) return 0;
    if (a.K == 0) return 3;
    const bool int_path = a.src_dt == DT_S8 || a.src_dt == DT_U8;
    const bool w_kmajor = a.wei_sk == 1 && a.wei_sn != 1;
    TcParams tp {};
    tp.num_n_tiles = (int)((a.N + BT_N - 1) / BT_N);
    tp.num_k_blocks = (int)((a.K + BKB - 1) / BKB);
    tp.w_kmajor = w_kmajor;
#ifdef QMM_PROFILE // a build with -DQMM_PROFILE reads the switch; the shipped library has no such code
    static const int mainloop_only = getenv("ONEDNN_CUDA_TC_MAINLOOP_ONLY") ? atoi(getenv("ONEDNN_CUDA_TC_MAINLOOP_ONLY")) : 0;
    tp.mainloop_only = mainloop_only;
#endif

    const bool chain = a.n_po > 0 || (a.bias && a.bias_sm != 0); // a bias varying along M rides the generic tail
    if (chain && a.peers.count) return 3; // refused when the replication is registered; not reached
    const bool want_colsum = int_path && a.src_zp.ptr;
    const GemmPlan plan = gemm_plan(a.M, tp.num_n_tiles, tp.num_k_blocks, sm_count, chain, want_colsum, a.peers.count == 0);
    tp.num_m_tiles = (int)((a.M + plan.bt - 1) / plan.bt);

    int32_t *colsum = (int32_t *)scratch;
    int32_t *rowsum = colsum ? colsum + ((a.N + 63) / 64) * 64 : nullptr;
    if (want_colsum && !plan.splits) {
        if (!scratch) return 5;
        // enough blocks to fill the GPU, at least 64 rows each
        const unsigned nb = (unsigned)((a.N + 127) / 128);
        int64_t chunks = (4 * (int64_t)(sm_count > 0 ? sm_count : 148) + nb - 1) / nb;
        chunks = chunks < 1 ? 1 : (chunks > (a.K + 63) / 64 ? (a.K + 63) / 64 : chunks);
        const int kchunk = (int)(((a.K + chunks - 1) / chunks + 7) / 8 * 8);
        const dim3 grid(nb, (unsigned)((a.K + kchunk - 1) / kchunk));
        if (cudaMemsetAsync(colsum, 0, (size_t)a.N * sizeof(int32_t), st) != cudaSuccess) return 5;
        const bool vec = a.wei_sn == 1 && a.wei_sk % 4 == 0 && (uintptr_t)a.wei % 4 == 0 && a.N % 4 == 0
                && (a.wei_dt == DT_S8 || a.wei_dt == DT_U8);
        if (vec) colsum_kernel<true><<<grid, 256, 0, st>>>(a, colsum, kchunk);
        else colsum_kernel<false><<<grid, 256, 0, st>>>(a, colsum, kchunk);
        count_launch();
        tp.colsum = colsum;
    }
    if (int_path && a.wei_zp.ptr) {
        if (!scratch) return 5;
        rowsum_kernel<<<(unsigned)((a.M + 3) / 4), 128, 0, st>>>(a, rowsum);
        count_launch();
        tp.rowsum = rowsum;
    }
    tp.after_prekernel = tp.colsum != nullptr || tp.rowsum != nullptr;

    CUtensorMap mw, ms;
    if (!make_map_2d(&ms, a.src, (uint64_t)a.K, (uint64_t)a.M, (uint64_t)a.src_sm, plan.bt)) return 5;
    if (w_kmajor) {
        if (!make_map_2d(&mw, a.wei, (uint64_t)a.K, (uint64_t)a.N, (uint64_t)a.wei_sn, BT_N)) return 5;
    } else {
        if (!make_map_2d(&mw, a.wei, (uint64_t)a.N, (uint64_t)a.K, (uint64_t)a.wei_sk, BKB)) return 5;
    }
    // operand A = weights, operand B = src
    uint32_t wfmt, sfmt, cfmt;
    if (int_path) {
        wfmt = a.wei_dt == DT_S8 ? ptx::FMT_S8 : ptx::FMT_U8;
        sfmt = a.src_dt == DT_S8 ? ptx::FMT_S8 : ptx::FMT_U8;
        cfmt = ptx::CFMT_S32;
    } else {
        wfmt = a.wei_dt == DT_F8_E4M3 ? ptx::FMT_E4M3 : ptx::FMT_E5M2;
        sfmt = a.src_dt == DT_F8_E4M3 ? ptx::FMT_E4M3 : ptx::FMT_E5M2;
        cfmt = ptx::CFMT_F32;
    }
    tp.idesc = ptx::make_idesc(cfmt, wfmt, sfmt, !w_kmajor, false, BT_N, plan.bt);
    SplitParams sp {};
    if (plan.splits) {
        sp.bt = plan.bt;
        sp.splits = plan.splits;
        sp.ones = want_colsum;
        sp.idesc_ones = ptx::make_idesc(cfmt, wfmt, sfmt, !w_kmajor, false, BT_N, ONES_COLS);
        sp.tmem_cols = plan.bt * (sp.ones ? 2 : 1);
        split_smem(plan, sp.ones, sp);
        if (!chain) return int_path ? launch_split_cfg<1, false>(mw, ms, a, tp, sp, st) : launch_split_cfg<0, false>(mw, ms, a, tp, sp, st);
    }
    if (chain) {
        const auto launch = a.dst_dt == DT_S8   ? launch_gemm_chain_s8
                : a.dst_dt == DT_U8   ? launch_gemm_chain_u8
                : a.dst_dt == DT_BF16 ? launch_gemm_chain_bf16
                : a.dst_dt == DT_F16  ? launch_gemm_chain_f16
                : a.dst_dt == DT_F32  ? launch_gemm_chain_f32
                                      : launch_gemm_chain_s32;
        return launch(int_path, plan.bt, mw, ms, a, tp, plan.splits ? &sp : nullptr, sm_count, st);
    }
#define QMM_TC(KIND) \
    (plan.bt == 256 ? launch_cfg<KIND, 256, 4, false>(mw, ms, a, tp, sm_count, st) \
                    : plan.bt == 64 ? launch_cfg<KIND, 64, 9, false>(mw, ms, a, tp, sm_count, st) \
                                    : launch_cfg<KIND, 128, 6, false>(mw, ms, a, tp, sm_count, st))
    return int_path ? QMM_TC(1) : QMM_TC(0);
#undef QMM_TC
}

// ---- allocation-free variant ----------------------------------------------
// Scratch of dnnl_cuda_interop_matmul_u8s8s32_zp_static: the column sums of
// the weights (zero-point compensation), preceded by a small header (the
// zero-point value and the kernel status word).  It is part of the library
// image: every GPU that loads the library holds these bytes until exit.
constexpr int64_t STATIC_MAX_N = 131072;
constexpr int STATIC_HEADER_WORDS = 64;
static __device__ __align__(256) int32_t g_static_scratch[STATIC_HEADER_WORDS + STATIC_MAX_N];

// hdr[0]: the src zero-point of the call in flight, read by the GEMM epilogue.
// hdr[1]: the kernels' status word.  It starts at zero when the library is
// loaded and is sticky: a call never clears it, so a bounded wait that expired
// in any earlier call stays visible until ..._static_status reads and resets it.
__global__ void static_scratch_header_kernel(int32_t *hdr, int32_t zero_point) { hdr[0] = zero_point; }
__global__ void static_scratch_status_reset_kernel(int32_t *hdr) { hdr[1] = 0; }

// Device address of the static scratch on the current device (looked up once
// per device; the table is filled under a mutex so that two host threads may
// make their first calls together).
constexpr int STATIC_MAX_DEVICES = 64;
struct StaticScratchSlot {
    int32_t *ptr = nullptr;
    int sm_count = 0;
};
bool static_scratch_of_current_device(StaticScratchSlot *out) {
    static StaticScratchSlot slots[STATIC_MAX_DEVICES];
    static std::mutex mu;
    int dev = 0;
    if (!cuda_ok(cudaGetDevice(&dev), "cudaGetDevice")) return false;
    if (dev < 0 || dev >= STATIC_MAX_DEVICES) {
        set_last_error("static scratch: device ordinal beyond 63");
        return false;
    }
    std::lock_guard<std::mutex> lock(mu);
    if (!slots[dev].ptr) { // set-up, once per device; not to be done under stream capture
        void *p = nullptr;
        // the array's NAME is a host-side stand-in here; kernels need its device address
        if (!cuda_ok(cudaGetSymbolAddress(&p, g_static_scratch), "cudaGetSymbolAddress")) return false;
        int sms = 0;
        if (!cuda_ok(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev), "cudaDeviceGetAttribute"))
            return false;
        slots[dev].sm_count = sms;
        slots[dev].ptr = (int32_t *)p;
    }
    *out = slots[dev];
    return true;
}

} // namespace qmm

// Host side of the static scratch: the array's NAME is only a host-side
// stand-in here; kernels need its device address, looked up once per device
// (with that device current) by cudaGetSymbolAddress.  The call allocates
// nothing: it enqueues a header kernel and the GEMM on the caller's stream, and
// before the persistent GEMM (enough tiles to fill the GPU) a memset of the
// column sums and the kernel that makes them.
extern "C" dnnl_status_t dnnl_cuda_interop_matmul_u8s8s32_zp_static(void *cuda_stream, int64_t M, int64_t N,
        int64_t K, const uint8_t *src, const int8_t *weights, int32_t src_zero_point, int32_t *dst) {
    using namespace qmm;
    if (M < 0 || N < 0 || K < 0 || ((M && K) && !src) || ((K && N) && !weights) || ((M && N) && !dst))
        return (dnnl_status_t)2; // invalid_arguments
    if (N > STATIC_MAX_N) {
        set_last_error("dnnl_cuda_interop_matmul_u8s8s32_zp_static: N exceeds the static scratch (131072 columns)");
        return (dnnl_status_t)2;
    }
    if (M == 0 || N == 0 || K == 0) return (dnnl_status_t)0; // nothing to compute, as the primitive does
    if (K % 16 || N % 16 || (uintptr_t)src % 16 || (uintptr_t)weights % 16 || M >= (1LL << 31)
            || K >= (1LL << 31)) {
        set_last_error("dnnl_cuda_interop_matmul_u8s8s32_zp_static: K and N must be multiples of 16 and the "
                       "src / weights pointers 16-byte aligned");
        return (dnnl_status_t)3; // unimplemented
    }
    StaticScratchSlot slot;
    if (!static_scratch_of_current_device(&slot)) return (dnnl_status_t)5;
    int32_t *hdr = slot.ptr;
    cudaStream_t st = (cudaStream_t)cuda_stream;
    static_scratch_header_kernel<<<1, 1, 0, st>>>(hdr, src_zero_point);
    count_launch();

    MatmulArgs a {};
    a.M = M; a.N = N; a.K = K;
    a.src = src; a.src_dt = DT_U8; a.src_sm = K; a.src_sk = 1;
    a.wei = weights; a.wei_dt = DT_S8; a.wei_sk = N; a.wei_sn = 1;
    a.dst = dst; a.dst_dt = DT_S32; a.dst_sm = N; a.dst_sn = 1;
    for (QParam *q : {&a.src_scale, &a.wei_scale, &a.dst_scale, &a.src_zp, &a.wei_zp, &a.dst_zp, &a.src_pr})
        q->g0 = q->g1 = 1;
    a.src_zp.ptr = hdr; // word 0 of the header
    a.src_zp.dt = DT_S32;
    a.non_default_attr = 1;
    a.sum_dt = DT_S32;
    a.status = hdr + 1;
    const int rc = launch_gemm_tc(a, hdr + STATIC_HEADER_WORDS, slot.sm_count, st);
    if (rc == 5) set_last_error(std::string("kernel launch: ") + cudaGetErrorString(cudaGetLastError()));
    return (dnnl_status_t)rc;
}

// Reads the sticky status word of the static entry point on the current
// device: waits for the work already enqueued on `cuda_stream`, copies the word
// to *status (0 = every call since the last query completed; 5 = a bounded
// wait inside a kernel expired and its dst is incomplete) and resets it.
// Allocates nothing; synchronises the stream, so it is not for use while the
// stream is being captured.
extern "C" dnnl_status_t dnnl_cuda_interop_matmul_u8s8s32_zp_static_status(void *cuda_stream, int *status) {
    using namespace qmm;
    if (!status) return (dnnl_status_t)2;
    StaticScratchSlot slot;
    if (!static_scratch_of_current_device(&slot)) return (dnnl_status_t)5;
    cudaStream_t st = (cudaStream_t)cuda_stream;
    int32_t word = 0;
    if (!cuda_ok(cudaMemcpyAsync(&word, slot.ptr + 1, sizeof(word), cudaMemcpyDeviceToHost, st), "cudaMemcpyAsync"))
        return (dnnl_status_t)5;
    if (!cuda_ok(cudaStreamSynchronize(st), "cudaStreamSynchronize")) return (dnnl_status_t)5;
    *status = word;
    if (word != 0) {
        static_scratch_status_reset_kernel<<<1, 1, 0, st>>>(slot.ptr);
        count_launch();
        if (!cuda_ok(cudaGetLastError(), "status reset")) return (dnnl_status_t)5;
    }
    return (dnnl_status_t)0;
}
