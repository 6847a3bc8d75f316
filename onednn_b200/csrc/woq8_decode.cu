// s8 weight-decompression matmul for few rows, dense and grouped (token generation):
//   dst[rows, :] = (src[rows, :] (bf16) x float(W[K, N] (s8))) * scale[n]   (per expert in the grouped form)
// the reference's arithmetic (src/cpu/matmul/ref_matmul.cpp:193-233, ref_grouped_gemm.cpp:312-339) up to f32 summation order.
//
// The structure is that of the int4 decode kernel (woq_decode.cu): four consumer warps of 32 columns that build the 16-row
// operand of mma.sync in registers - PRMT pairs two k-rows, one LOP3 and one packed FMA make x / 64 of two weights, exactly,
// and the sums are multiplied by 64 -, a producer warp, several such CTAs per SM, and the CTAs of a tile's K shares a
// cluster that adds its sums in rank order through distributed shared memory.  A tile is 128 columns x up to 32 rows.
//
// A grouped call has a CTA (cluster) for every column tile and every block of up to 32 rows of one expert that there can be: no
// more blocks than rows, nor than experts and a block more for every 32 rows.  Each finds its rows from the offsets on the
// device, checking those of all experts: one wrong offset leaves all of dst unwritten, as with the planning kernel of
// grouped_tc.cu.  (CTAs for every expert and block left at once where there were no rows, 0.09 us of an SM each: us a call, that
// kernel / CTAs for all / now, 8 x 1024 x 2048, 512 experts 20 / 33 / 14; 40 x 512 x 1024, 1024 experts 27 / 38 / 25;
// 1 x 4096 x 14336, 64 experts 36 / 48 / 14; 33 x 2048 x 4096, 128 experts 70 / 76 / 57; 37 x 4096 x 14336, 8 experts 112 / 104 / 96.)
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <string>

#include "decode_ptx.cuh"
#include "device_math.cuh"
#include "launch.h"
#include "objects.hpp"

namespace qmm {

namespace {

constexpr int WARPS = 4, THREADS = 32 * (WARPS + 1);
constexpr int NB = 32 * WARPS, NB_LOG = 7; // columns per tile
constexpr int KS = 64, W_BYTES = KS * NB; // k-rows and weight bytes per stage
constexpr int MAX_STAGES = 12, MAX_CLUSTER = 8;
constexpr int CTAS = 4; // per SM: 96 registers, 55 KB each
constexpr int BAR_BYTES = 2 * MAX_STAGES * 8 + 64, FOUND_OFFSET = 2 * MAX_STAGES * 8 + 16;
constexpr int SMEM = 55 * 1024;

struct W8Params {
    int kstages; // ceil(K / 64)
    int rows; // src rows per CTA (at most 8 * MT)
    int split_log; // log2 of the CTAs per tile = cluster size
    int fast_store; // the value is scaled, converted and stored, four columns at a time
    int stages, stage_bytes, off_bars;
};

// Grouped: the `y`-th block of up to 32 rows of one expert, {expert, first src row, first dst row, rows}, by a warp; no rows where
// there are not as many blocks, or where the offsets of any expert are wrong.  (Out of line, so that the code of the consumers'
// loop does not change with it, which cost 2 %.)
__device__ __noinline__ int4 find_rows(const MatmulArgs &a, int y, int lane) {
    int4 mine = make_int4(0, 0, 0, 0);
    int before = 0; // blocks of the experts before these 32
    bool wrong = false;
    for (int g0 = 0; g0 < a.group_count; g0 += 32) {
        const int g = g0 + lane;
        int rows = 0, src_row = 0, dst_row = 0;
        if (g < a.group_count) {
            const int64_t b = g == 0 ? 0 : a.offsets[g - 1], e = a.offsets[g];
            const int64_t db = g == 0 ? 0 : a.dst_offsets[g - 1], de = a.dst_offsets[g];
            const bool bad = b < 0 || e > a.M || e < b || db < 0 || de > a.M || de < db || de - db != e - b;
            wrong |= bad;
            rows = bad ? 0 : (int)(e - b);
            src_row = (int)b;
            dst_row = (int)db;
        }
        const int blocks = (rows + 31) >> 5;
        int upto = blocks; // inclusive sum over the lanes
#pragma unroll
        for (int d = 1; d < 32; d *= 2) {
            const int x = __shfl_up_sync(0xffffffffu, upto, d);
            if (lane >= d) upto += x;
        }
        const int at = y - before - (upto - blocks); // of this expert's blocks
        const unsigned found = __ballot_sync(0xffffffffu, at >= 0 && at < blocks);
        if (found) {
            const int from = __ffs(found) - 1, r0 = __shfl_sync(0xffffffffu, at, from) * 32;
            mine = make_int4(g0 + from, __shfl_sync(0xffffffffu, src_row, from) + r0, __shfl_sync(0xffffffffu, dst_row, from) + r0,
                    min(32, __shfl_sync(0xffffffffu, rows, from) - r0));
        }
        before += __shfl_sync(0xffffffffu, upto, 31);
    }
    if (__any_sync(0xffffffffu, wrong)) {
        if (lane == 0) atomicExch(a.status, 2); // invalid_arguments, reported when the stream is waited on
        mine.w = 0;
    }
    return mine;
}
// general store: bias (per expert row, or the dense problem's own broadcast), post-ops, any dst type
__device__ __noinline__ void finish_store_w8(const MatmulArgs &a, float d, int64_t m, int64_t n, int g) {
    if (a.bias)
        d = __fadd_rn(d, load_float(a.bias_dt, a.bias, a.group_count > 0 ? (int64_t)g * a.bias_sg + n : m * a.bias_sm + n * a.bias_sn));
    d = apply_post_ops(a, d, 0.f, m, n, g);
    store_float(a.dst_dt, d, a.dst, m * a.dst_sm + n * a.dst_sn);
}
// two s8 (bytes 0 and 2 of t) -> bf16 x / 64: see grouped_tc.cu
__device__ __forceinline__ uint32_t widen(uint32_t t) { return fma2<false>(and_xor(t, 0x00FF00FFu, 0x00800080u), 0x7F007F00u, 0xC000C000u); }

template <int MT>
__global__ void __launch_bounds__(THREADS, CTAS)
woq8_decode_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmS, const __grid_constant__ MatmulArgs a,
        const __grid_constant__ W8Params p) {
    extern __shared__ __align__(1024) uint8_t smem[];
    float *const sums = reinterpret_cast<float *>(smem + p.stages * p.stage_bytes); // [rank][rows][columns of this CTA's slice]
    uint64_t *full = (uint64_t *)(smem + p.off_bars);
    uint64_t *empty = full + MAX_STAGES, *sums_bar = empty + MAX_STAGES;
    const int warp = threadIdx.x / 32, lane = in_reg(threadIdx.x % 32);
    const int split_log = p.split_log, splits = 1 << split_log, rank = (int)blockIdx.x & (splits - 1), tile = (int)blockIdx.x >> split_log;
    if (threadIdx.x == 0) {
        for (int s = 0; s < p.stages; ++s) {
            ptx::mbar_init(&full[s], 1);
            ptx::mbar_init(&empty[s], WARPS);
        }
        ptx::mbar_init(sums_bar, 1);
        ptx::fence_barrier_init();
        ptx::prefetch_tensormap(&tmW);
        ptx::prefetch_tensormap(&tmS);
    }
    // A programmatic dependent of whatever precedes it on the stream (its set-up runs under the predecessor's end).
    ptx::grid_dependency_wait();
    int g = 0, src_row, dst_row, rows;
    if (a.group_count > 0) {
        int4 *const found = reinterpret_cast<int4 *>(smem + p.off_bars + FOUND_OFFSET);
        if (warp == 0) {
            const int4 mine = find_rows(a, (int)blockIdx.y, lane);
            if (lane == 0) {
                *found = mine;
                ptx::mbar_arrive_expect_tx(sums_bar, (uint32_t)mine.w * NB * 4); // every CTA's share of this CTA's slice
            }
        }
        __syncthreads();
        g = found->x;
        src_row = found->y;
        dst_row = found->z;
        rows = found->w;
        if (rows <= 0) return; // (every CTA of the cluster)
    } else {
        src_row = dst_row = (int)blockIdx.y * p.rows;
        rows = min((int64_t)p.rows, a.M - src_row);
        if (threadIdx.x == 0) ptx::mbar_arrive_expect_tx(sums_bar, (uint32_t)rows * NB * 4);
        __syncthreads();
    }
    if (splits > 1) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); // sums_bar is ready

    const int st0 = (int)((unsigned)p.kstages * rank >> split_log), st1 = (int)((unsigned)p.kstages * (rank + 1) >> split_log);
    const uint32_t ring = ptx::smem_u32(smem), bars = ptx::smem_u32(full);
    const int stages = in_reg(p.stages), stage_bytes = in_reg(p.stage_bytes);
    if (warp == WARPS) {
        // ------------------------------------------------ producer
        if (ptx::elect_one()) {
            const uint64_t map_w = reinterpret_cast<uint64_t>(&tmW), map_s = reinterpret_cast<uint64_t>(&tmS);
            const uint32_t bars_end = bars + stages * 8;
            uint32_t bar = bars, sw = ring, ph = 1;
            for (int st = st0; st < st1; ++st) {
                if (!wait<200>(bar + MAX_STAGES * 8, ph)) { atomicExch(a.status, 5); break; }
                arrive_expect_tx(bar, W_BYTES + MT * 1024);
                tma_load_3d(sw, map_w, bar, tile * NB, st * KS, g);
                tma_load(sw + W_BYTES, map_s, bar, st * KS, src_row);
                bar += 8;
                sw += stage_bytes;
                if (bar == bars_end) { bar = bars; sw = ring; ph ^= 1; }
            }
        }
        __syncwarp();
        asm volatile("griddepcontrol.launch_dependents;"); // the CTA's loads are all on their way
        if (splits > 1) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    } else {
        // ------------------------------------------------ consumers
        const int gq = lane >> 2, t4 = lane & 3;
        // the lane's 4 columns are one word of a k-row, at byte 32 * warp + 4 gq; addresses as in woq_decode.cu
        const uint32_t chunk = (32 * warp + 4 * gq) >> 4, within = (4 * gq) & 15;
        const uint32_t lds0 = (2 * t4) * 128 + ((chunk ^ (uint32_t)(2 * t4)) << 4) + within;
        const uint32_t lds1 = (2 * t4 + 1) * 128 + ((chunk ^ (uint32_t)(2 * t4 + 1)) << 4) + within;
        const uint32_t mrow = lane & 7, moct = (lane >> 3) & 1;
        const uint32_t lds_s = W_BYTES + (MT > 1 ? (lane >> 4) * 1024 : 0) + mrow * 128 + ((moct ^ mrow) << 4);
        const int blocks = (rows + 7) / 8; // of the MT that have rows
        float acc[2][MT][4];
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int t = 0; t < MT; ++t)
#pragma unroll
                for (int e = 0; e < 4; ++e) acc[j][t][e] = 0.f;
        struct Step {
            uint32_t w[4];
            uint32_t b[2 * MT];
        };
        auto load_step = [&](Step &x, uint32_t sw, int q) {
            x.w[0] = lds32(sw + lds0 + q * 2048);
            x.w[1] = lds32(sw + lds1 + q * 2048);
            x.w[2] = lds32(sw + lds0 + q * 2048 + 1024);
            x.w[3] = lds32(sw + lds1 + q * 2048 + 1024);
            const uint32_t bs = (sw + lds_s) ^ (q << 5);
#pragma unroll
            for (int t = 0; t + 1 < MT; t += 2) ldsm_x4(x.b + 2 * t, bs + t * 1024);
            if (MT & 1) ldsm_x2(x.b + 2 * (MT - 1), bs + (MT - 1) * 1024);
        };
        auto multiply = [&](const Step &x) {
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const uint32_t sel0 = j ? 0x7662u : 0x5440u, sel1 = j ? 0x7773u : 0x5551u; // byte 2j (2j + 1) of two rows, in bytes 0 and 2
                uint32_t w[4];
                w[0] = widen(perm(x.w[0], x.w[1], sel0));
                w[1] = widen(perm(x.w[0], x.w[1], sel1));
                w[2] = widen(perm(x.w[2], x.w[3], sel0));
                w[3] = widen(perm(x.w[2], x.w[3], sel1));
#pragma unroll
                for (int t = 0; t < MT; ++t)
                    if (MT == 1 || t < blocks) mma<false>(acc[j][t], w, x.b[2 * t], x.b[2 * t + 1]);
            }
        };
        uint32_t ph = 0, so = 0, bar = bars; // parity, offset and full barrier of the stage
        const uint32_t ring_bytes = stages * stage_bytes;
        Step x0, x1;
        bool ok = __all_sync(0xffffffffu, wait<20>(bar, 0));
        if (ok) load_step(x0, ring, 0);
        for (int st = st0; st < st1 && ok; ++st) {
            const uint32_t sw = ring + so;
            uint32_t pn = ph, son = so + stage_bytes, barn = bar + 8;
            if (son == ring_bytes) { son = 0; barn = bars; pn ^= 1; }
            uint32_t ready = 1;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                Step &cur = q & 1 ? x1 : x0, &next = q & 1 ? x0 : x1;
                if (q < 3) {
                    load_step(next, sw, q + 1);
                    if (q == 2 && st + 1 < st1) ready = try_wait(barn, pn);
                } else {
                    __syncwarp();
                    if (lane == 0) arrive(bar + MAX_STAGES * 8); // everything of the stage is in registers
                    if (!__all_sync(0xffffffffu, ready)) ready = __all_sync(0xffffffffu, wait_long<20>(barn, pn));
                    load_step(next, ring + son, 0); // (after the last stage: what a stage holds by then, not used)
                }
                multiply(cur);
            }
            ok = ready;
            bar = barn;
            so = son;
            ph = pn;
        }
        if (!ok) atomicExch(a.status, 5);
        if (splits > 1) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); // long since complete
        const int slice_log = NB_LOG - split_log, slice = 1 << slice_log;
        const int col = 32 * warp + 4 * gq, owner = col >> slice_log, c = col & (slice - 1);
        const uint32_t sums_at = map_rank(ptx::smem_u32(sums), owner), bar_at = map_rank(ptx::smem_u32(sums_bar), owner);
#pragma unroll
        for (int t = 0; t < MT; ++t)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int m = 8 * t + 2 * t4 + h;
                if (m >= rows) continue;
                st_async_v4(sums_at + (uint32_t)((rank * rows + m) * slice + c) * 4, __float_as_uint(acc[0][t][h]), __float_as_uint(acc[0][t][2 + h]),
                        __float_as_uint(acc[1][t][h]), __float_as_uint(acc[1][t][2 + h]), bar_at);
            }
    }

    // ---------------------------------------------------- this CTA's slice: the sum over the ranks, in order -> dst
    const int slice_log = NB_LOG - split_log, slice = 1 << slice_log;
    const bool late = !ptx::mbar_wait(sums_bar, 0);
    if (late) atomicExch(a.status, 5);
    if (__syncthreads_or(late)) {
        if (splits > 1) ptx::outlast_cluster(sums_bar);
        return;
    }
    const int nvec = rows << (slice_log - 2);
    for (int i = threadIdx.x; i < nvec; i += THREADS) {
        const int m = i >> (slice_log - 2), c = (i << 2) & (slice - 1);
        const int64_t n = (int64_t)tile * NB + rank * slice + c;
        if (n >= a.N) continue;
        const float *at = sums + m * slice + c;
        float4 v = *reinterpret_cast<const float4 *>(at);
        for (int r = 1; r < splits; ++r) {
            const float4 w = *reinterpret_cast<const float4 *>(at + r * rows * slice);
            v.x += w.x; v.y += w.y; v.z += w.z; v.w += w.w;
        }
        float d[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float scale = n + e < a.N ? load_float(a.wei_scale.dt, a.wei_scale.ptr, (int64_t)g * a.wei_scale.gstride + ((a.wei_scale.mask & 2) ? n + e : 0)) : 0.f;
            d[e] = __fmul_rn(d[e] * 64.f, scale);
        }
        const int64_t mg = dst_row + m;
        if (p.fast_store && n + 3 < a.N) {
            const int64_t o = mg * a.dst_sm + n;
            if (a.dst_dt == DT_F32) {
                *reinterpret_cast<float4 *>((float *)a.dst + o) = make_float4(d[0], d[1], d[2], d[3]);
            } else if (a.dst_dt == DT_BF16) {
                *reinterpret_cast<uint2 *>((unsigned short *)a.dst + o) = make_uint2((uint32_t)f32_to_bf16_bits(d[0]) | ((uint32_t)f32_to_bf16_bits(d[1]) << 16),
                        (uint32_t)f32_to_bf16_bits(d[2]) | ((uint32_t)f32_to_bf16_bits(d[3]) << 16));
            } else {
                auto h = [](float x) { return (uint32_t)__half_as_ushort(__float2half_rn(x)); };
                *reinterpret_cast<uint2 *>((unsigned short *)a.dst + o) = make_uint2(h(d[0]) | (h(d[1]) << 16), h(d[2]) | (h(d[3]) << 16));
            }
        } else {
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if (n + e < a.N) finish_store_w8(a, d[e], mg, n + e, g);
        }
    }
}

typedef CUresult (*encode_tiled_fn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
        const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
        CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

encode_tiled_fn w8_get_encode() {
    static encode_tiled_fn fn = nullptr;
    if (!fn) {
        void *ptr = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &q) == cudaSuccess
                && q == cudaDriverEntryPointSuccess)
            fn = (encode_tiled_fn)ptr;
    }
    return fn;
}

template <int MT>
int w8_launch(const CUtensorMap &tw, const CUtensorMap &ts, const MatmulArgs &a, W8Params p, int ntiles, int ny, cudaStream_t st) {
    auto kern = woq8_decode_kernel<MT>;
    const int sums_bytes = p.rows * NB * 4;
    p.stage_bytes = W_BYTES + MT * 1024;
    p.stages = (SMEM - BAR_BYTES - sums_bytes) / p.stage_bytes;
    if (p.stages > MAX_STAGES) p.stages = MAX_STAGES;
    p.off_bars = p.stages * p.stage_bytes + sums_bytes;
    static std::atomic<unsigned long long> configured;
    if (!opt_in_dynamic_smem(kern, SMEM, configured)) return 5;
    cudaLaunchConfig_t cfg {};
    cfg.gridDim = dim3((unsigned)ntiles << p.split_log, (unsigned)ny);
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = (size_t)(p.off_bars + BAR_BYTES);
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1u << p.split_log;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, tw, ts, a, p);
    if (e != cudaSuccess) {
        (void)cudaGetLastError();
        set_last_error(std::string("cuda:tcgen05:woq8 launch: ") + cudaGetErrorString(e));
        return 5;
    }
    count_launch("woq8_decode");
    return 0;
}

// Blocks of rows that a call can need
int64_t w8_blocks(const MatmulArgs &a) {
    if (a.group_count == 0) return (a.M + 31) / 32;
    const int64_t most = a.group_count + a.M / 32;
    return a.M < most ? a.M : most;
}

// log2 of the CTAs per tile, as in woq_decode.cu: the busiest SM's stages, a CTA's start and end counted as 3 + mt, a stage alone on an
// SM as 2.5
int w8_split_log(int64_t tiles, int kstages, int mt, int sms) {
    int best = 0;
    int64_t cost = INT64_MAX;
    for (int l = 0; 1 << l <= MAX_CLUSTER && 1 << l <= kstages; ++l) {
        const int64_t busiest = ((tiles << l) + sms - 1) / sms, share = 2 * busiest > 5 ? 2 * busiest : 5;
        const int64_t c = share * (((kstages + (1 << l) - 1) >> l) + 3 + mt);
        if (c < cost) { cost = c; best = l; }
    }
    return best;
}

} // namespace

// Whether this kernel is the faster one (else grouped_tc.cu), by a model of both in microseconds: the busiest SM's stages with its
// CTAs' starts and ends at 0.18 here (0.205 for more than 24 rows), a 64-k slot of a wave of tiles 0.14 there and more with its rows.
// Fitted to 130 problems (24 to 1000 rows, K 512 to 8192, N 1024 to 16384) timed with both kernels: the choice costs 0.1 % on average, and
// 15 % once, 3 % at most otherwise (a model of stages alone 0.9 % and 27 %: 256 x 4096 x 4096 36.8 for 29.0).  Grouped calls: up to 64 rows.
// us a call, that kernel -> this one: dense 1 x 4096 x 4096 22.6 -> 6.7, 16 x 4096 x 11008 24.7 -> 15.7, 64 x 4096 x 4096
// 26.7 -> 14.1, 128 x 8192 x 1024 45.2 -> 15.0, 256 x 1024 x 1024 20.5 -> 7.7, 32 x 8192 x 16384 42.9 -> 38.0; grouped 37 rows, 8 experts,
// 4096 x 14336 112 -> 96 (72 are the stream), 64 rows, 16 experts, 2048 x 4096 40.5 -> 33.8, 9 rows, 8 experts, 1024 x 2048 13.9 -> 7.
// How the rows are spread is not known here.  All of them with one expert is the worst case: 64 rows, 8 experts, 4096 x 14336
// 28.9 -> 48, of narrow layers 64 x 1024 x 1024 16.6 -> 7.7.
bool woq8_decode_wins(const MatmulArgs &a, int sm_count) {
    if (a.wei_zp.ptr || (uintptr_t)a.wei % 16 || (uintptr_t)a.src % 16) return false;
    const int sms = sm_count > 0 ? sm_count : 148;
    if (a.group_count > 0) return a.M <= 64 && a.group_count <= 1024; // (every CTA looks through them: 3 rows, 2000 experts 33 us, there 29)
    const int64_t kst = (a.K + KS - 1) / KS, ntiles = (a.N + NB - 1) / NB, blocks = w8_blocks(a);
    if (blocks > 1024) return false;
    const int mt = (int)(((a.M + blocks - 1) / blocks + 7) / 8), l = w8_split_log(ntiles * blocks, (int)kst, mt, sms);
    const float busiest = (float)(((ntiles * blocks << l) + sms - 1) / sms), share = (float)((kst + (1 << l) - 1) >> l);
    const float here = 3.8f + (mt > 3 ? 0.205f : 0.18f) * busiest * (share + 3.8f + 1.4f * (float)mt);
    const int64_t mtiles = (a.M + 207) / 208, waves = (ntiles * mtiles + sms - 1) / sms, rows = ((a.M + mtiles - 1) / mtiles + 15) / 16 * 16;
    const float there = 9.f + (float)(waves * kst) * (0.14f + 0.0014f * (float)rows);
    return here < there;
}

// bf16 src [M, K], s8 weights [G, K, N] (dense: [K, N]), N contiguous, scales per tensor or per (expert,) column
int launch_woq8_decode(const MatmulArgs &a, int sm_count, cudaStream_t st) {
    if (a.M == 0 || a.N == 0) return 0;
    encode_tiled_fn enc = w8_get_encode();
    if (!enc) return 5;
    const bool grouped = a.group_count > 0;
    W8Params p {};
    int ny;
    if (grouped) {
        p.rows = a.M < 32 ? (int)a.M : 32;
        ny = (int)w8_blocks(a);
    } else {
        const int blocks = (int)((a.M + 31) / 32);
        p.rows = (int)((a.M + blocks - 1) / blocks);
        ny = blocks;
    }
    const int mt = (p.rows + 7) / 8;
    if (ny > 65535) return 3;
    CUtensorMap tw, ts;
    {
        const int64_t groups = grouped ? a.group_count : 1, group_pitch = grouped ? a.wei_sg : a.K * a.wei_sk;
        cuuint64_t dims[3] = {(cuuint64_t)a.N, (cuuint64_t)a.K, (cuuint64_t)groups};
        cuuint64_t strides[2] = {(cuuint64_t)a.wei_sk, (cuuint64_t)group_pitch};
        cuuint32_t box[3] = {NB, KS, 1};
        cuuint32_t estr[3] = {1, 1, 1};
        if (enc(&tw, CU_TENSOR_MAP_DATA_TYPE_UINT8, 3, const_cast<void *>(a.wei), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                    CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE)
                != CUDA_SUCCESS)
            return 5;
    }
    {
        cuuint64_t dims[2] = {(cuuint64_t)a.K, (cuuint64_t)a.M};
        cuuint64_t strides[1] = {(cuuint64_t)(a.src_sm * 2)};
        cuuint32_t box[2] = {KS, (cuuint32_t)(8 * mt)};
        cuuint32_t estr[2] = {1, 1};
        if (enc(&ts, CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, const_cast<void *>(a.src), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                    CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE)
                != CUDA_SUCCESS)
            return 5;
    }
    p.kstages = (int)((a.K + KS - 1) / KS);
    {
        const int es = a.dst_dt == DT_F32 ? 4 : 2;
        p.fast_store = !a.bias && a.n_po == 0 && (a.dst_dt == DT_F32 || a.dst_dt == DT_BF16 || a.dst_dt == DT_F16) && a.dst_sn == 1
                && a.dst_sm % 4 == 0 && (uintptr_t)a.dst % (4 * es) == 0;
    }
    const int ntiles = (int)((a.N + NB - 1) / NB);
    p.split_log = w8_split_log(ntiles * w8_blocks(a), p.kstages, mt, sm_count > 0 ? sm_count : 148);
    switch (mt) {
        case 1: return w8_launch<1>(tw, ts, a, p, ntiles, ny, st);
        case 2: return w8_launch<2>(tw, ts, a, p, ntiles, ny, st);
        case 3: return w8_launch<3>(tw, ts, a, p, ntiles, ny, st);
        default: return w8_launch<4>(tw, ts, a, p, ntiles, ny, st);
    }
}

} // namespace qmm
