// "cuda:tcgen05:woq4_rows": int4 weight-decompression matmul for more rows than the decode kernels take
// (prompt processing, M > 32):
//   dst[M,N] = src[M,K] (bf16/f16) x dequant(weights[K,N] s4/u4 `ab`),
// scales per column or per (K-group, column), optional 4-bit zero-points (f16 src: 8-bit ones too) with the
// same grouping or per tensor (fpmath apply_to_int; reference arithmetic: src/cpu/matmul/ref_matmul.cpp:193-233).
//
// w - zero_point is an integer that bf16 (f16) holds exactly, so the operand of the MMAs is exact.  bf16: a lower
// byte u under a zero upper byte is the number u * 2^-133 (the step from subnormal to normal numbers included), so
// one LOP3 and one packed FMA make (w - zero_point) / 64 of two nibbles, low ones or high ones where they stand
// (u * 2^-133 * 2^127, or * 2^123, less (8 for s4 + zero_point) / 64); the group sum is multiplied by the 64.  f16: a nibble
// under 0x64 is 1024 + u (or 1024 + 16 u), and a packed subtraction (or FMA) takes the rest off.  The sums of a
// K-group are exact products added in f32, and the group's scale multiplies the finished group sum:
// tot += scale * sum, in f32 registers of the epilogue.  Nothing is rounded to 16 bits before dst, and no
// correction by row sums is needed.
//
// As in the other decompression kernels the weights are the A operand, in TENSOR MEMORY (128 dst columns = TMEM
// lanes), and the src rows the B operand from shared memory, so an epilogue lane owns one dst column.  A tile is
// 128 columns x up to 128 rows (two accumulators of 128 columns and four operand slots of 64 fill the 512).
//
// What bounds the kernel is the chain of dependent instructions of each role, not a pipe: a satisfied barrier
// wait costs 150 to 300 cycles, the conversion of a warp's share of a 128-k stage about 1500, the fold of 32 rows
// by an epilogue warp about 750, while one thread issues the eight MMAs of a stage in 100.  Hence stages of 128 k
// with one barrier for operand and src tile together, 16 epilogue warps with 32 rows each, and loads of scales
// and zero-points issued groups ahead.
//
// Roles (28 warps): 0 weight tiles by TMA, 1 src tiles by TMA, 2 issues all MMAs, 4-11 converters (two per lane
// quarter, taking the stages in turn), 12-27 epilogue (four per lane quarter, each a quarter of the rows).  Every mbarrier wait is bounded.
//
// Measured on a B200, us a call of this kernel at K = N = 4096, bf16, zero-points per group, by the group size (every group costs
// a fold of the whole accumulator and two hand-offs; launch_woq_rows gives most of these problems to woq_decode.cu):
//   group            32    64   128   256
//   M = 64          118    66    40    33
//   M = 128         136    76    43    35
//   M = 300         116    70    43    36
//   M = 512         137    77    44    37
// 32 tiles and 96 at M = 64 and 300 leave SMs idle: K is not split.  300 rows in groups of 128 without zero-points 37;
// the generic kernel takes 54.3 ms for them.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <string>

#include "device_math.cuh"
#include "launch.h"
#include "objects.hpp"
#include "sm100_ptx.cuh"

namespace qmm {

namespace {

constexpr int RT_N = 128; // dst columns per tile = TMEM lanes
constexpr int RT_M = 128; // most src rows per tile
constexpr int RK = 128; // k per stage: eight MMAs share one pair of hand-offs
constexpr int W_STAGES = 10; // nibble tiles (from HBM)
constexpr int STAGES = 4; // operand slots in tensor memory and src tiles, used and released together
constexpr int ACC_BUFS = 2;
constexpr int W_BYTES = RK * RT_N / 2; // nibbles as loaded: 64-byte rows
constexpr int B_BYTES = RT_M * RK * 2; // src rows: two boxes of 64 k
constexpr int CONV_SETS = 2; // sets of four converter warps, which take the stages in turn
// a set that could run ahead of the other by more than the ring would take an older phase of a slot for its own
static_assert(CONV_SETS <= STAGES, "barrier parity");
constexpr int R_CONV_WARPS = 4 * CONV_SETS, R_EPI_WARPS = 16;
constexpr int EPI_PIECES = RT_M / 16 / (R_EPI_WARPS / 4); // 16-row pieces of the accumulator per epilogue warp
constexpr int R_CONV0 = 4, R_EPI0 = R_CONV0 + R_CONV_WARPS;
constexpr int R_THREADS = 32 * (R_EPI0 + R_EPI_WARPS);
constexpr int SPS = RK / 16; // k16 steps per stage
constexpr int A_SLOT_COLS = RK / 2;
constexpr int R_A_COL0 = ACC_BUFS * RT_M;
static_assert(R_A_COL0 + STAGES * A_SLOT_COLS <= 512, "tensor memory");
constexpr int R_B_OFFSET = 0, R_W_OFFSET = STAGES * B_BYTES;
constexpr int R_BAR_OFFSET = R_W_OFFSET + W_STAGES * W_BYTES;
constexpr int R_SMEM_BYTES = R_BAR_OFFSET + 512 + 1024;
static_assert(R_SMEM_BYTES <= 227 * 1024, "shared memory");

struct RowsParams {
    int num_m_tiles, num_tiles;
    int tile_rows; // a multiple of 16, at most RT_M: the MMAs' N and the rows of a src box
    int ksteps; // K / 16
    int kstages; // ceil(K / 128)
    int group_steps; // k16 steps per quantization group (ksteps when not grouped along K)
    int sgn4; // weights are s4 (else u4)
    int zp_mode; // 0 none, 1 per (group, column), 2 per tensor
    int fast_store; // no post-ops / dst scale: the value is converted and stored
    uint32_t idesc;
};

__device__ __forceinline__ uint32_t and_xor(uint32_t x, uint32_t mask, uint32_t magic) { // (x & mask) ^ magic
    uint32_t r;
    asm("lop3.b32 %0, %1, %2, %3, 0x6a;" : "=r"(r) : "r"(x), "r"(mask), "r"(magic));
    return r;
}
__device__ __forceinline__ uint32_t perm(uint32_t a, uint32_t b, uint32_t sel) {
    uint32_t r;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(sel));
    return r;
}
__device__ __forceinline__ uint32_t fma_bf16x2(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t d;
    asm("fma.rn.bf16x2 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}
__device__ __forceinline__ uint32_t sub_f16x2(uint32_t a, uint32_t b) {
    uint32_t d;
    asm("sub.rn.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
}
__device__ __forceinline__ uint32_t fma_f16x2(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t d;
    asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}
// 16 TMEM lanes x 32 columns (four k16 steps): see the s8 kernel (grouped_tc.cu) for the fragment
__device__ __forceinline__ void st_16x128b_x8(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile(
            "tcgen05.st.sync.aligned.16x128b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(taddr),
            "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),
            "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
            : "memory");
}
__device__ __forceinline__ void mma_ts_16bit(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, bool acc) {
    asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(tmem_d),
            "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"((uint32_t)acc)
            : "memory");
}
__device__ __forceinline__ uint64_t pack2(uint32_t lo, uint32_t hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(lo), "r"(hi));
    return r;
}
// two fused multiply-adds: d = sc * {v0, v1} + d
__device__ __forceinline__ void fma_f32x2(uint64_t &d, uint64_t sc, uint64_t v) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(sc), "l"(v));
}
__device__ __forceinline__ uint64_t mul_f32x2(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
// bias, post-ops, dst scale, any dst type: rare and large, out of line
__device__ __noinline__ void finish_store_general(const MatmulArgs &a, float d, int64_t m, int64_t n) {
    if (a.bias) d = __fadd_rn(d, load_float(a.bias_dt, a.bias, m * a.bias_sm + n * a.bias_sn));
    finish_store(a, d, m, n, false);
}
// A kernel parameter held in a register.  Read where they are used, parameters come from a constant cache
// that five roles with their own corners of a 3 KB parameter block keep missing (hundreds of cycles a miss).
__device__ __forceinline__ int in_reg(int v) {
    asm volatile("" : "+r"(v));
    return v;
}
__device__ __forceinline__ bool warp_wait(uint64_t *bar, uint32_t parity) {
    return __all_sync(0xffffffffu, ptx::mbar_wait(bar, parity));
}

// Loads that must be issued where they stand, well before their use: the compiler is free to move an
// ordinary one down to it.  Coherent: the call before may have written the parameters.
__device__ __forceinline__ uint32_t ld_early_u32(const uint32_t *p) {
    uint32_t v;
    asm volatile("ld.global.u32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ uint32_t ld_early_u16(const unsigned short *p) {
    unsigned short v;
    asm volatile("ld.global.u16 %0, [%1];" : "=h"(v) : "l"(p));
    return v;
}
// The zero-points of a lane's four columns (n .. n + 3) in group g, as loaded: four nibbles or four bytes
__device__ __forceinline__ uint32_t load_zp4(const MatmulArgs &a, int g, int64_t n) {
    if (n >= a.N) return 0u;
    const int64_t e = (int64_t)g * a.wei_zp.ld + n;
    if (a.wei_zp.dt == DT_U4 || a.wei_zp.dt == DT_S4) return ld_early_u16((const unsigned short *)a.wei_zp.ptr + (e >> 2));
    return ld_early_u32((const uint32_t *)a.wei_zp.ptr + (e >> 2));
}
__device__ __forceinline__ int zp_of(int dt, uint32_t raw, int i) {
    if (dt == DT_U4 || dt == DT_S4) {
        const int v = (int)((raw >> (4 * i)) & 15u);
        return dt == DT_S4 ? (v ^ 8) - 8 : v;
    }
    const int v = (int)((raw >> (8 * i)) & 255u);
    return dt == DT_S8 ? (int)(signed char)v : v;
}

// MULTI: a 128-k stage may touch several groups (group size not a multiple of 128): the offsets are looked up
// per k16 step instead of per stage.
template <bool F16, bool MULTI>
__global__ void __launch_bounds__(R_THREADS, 1)
woq_rows_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmS,
        const __grid_constant__ MatmulArgs a, const __grid_constant__ RowsParams p) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint64_t *w_full = (uint64_t *)(smem + R_BAR_OFFSET);
    uint64_t *w_empty = w_full + W_STAGES;
    uint64_t *ab_full = w_empty + W_STAGES; // src tile and operand slot of a stage
    uint64_t *ab_empty = ab_full + STAGES;
    uint64_t *acc_full = ab_empty + STAGES;
    uint64_t *acc_empty = acc_full + ACC_BUFS;
    uint32_t *tmem_slot = (uint32_t *)(acc_empty + ACC_BUFS);
    volatile int *abort_flag = (volatile int *)(tmem_slot + 1);

    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    if (threadIdx.x == 0) {
        for (int s = 0; s < W_STAGES; ++s) {
            ptx::mbar_init(&w_full[s], 1);
            ptx::mbar_init(&w_empty[s], 4); // the stage's four converter warps
        }
        for (int s = 0; s < STAGES; ++s) {
            ptx::mbar_init(&ab_full[s], 1 + 4); // the src tile's producer, the stage's converters
            ptx::mbar_init(&ab_empty[s], 1);
        }
        for (int s = 0; s < ACC_BUFS; ++s) {
            ptx::mbar_init(&acc_full[s], 1);
            ptx::mbar_init(&acc_empty[s], R_EPI_WARPS);
        }
        *abort_flag = 0;
        ptx::fence_barrier_init();
        ptx::prefetch_tensormap(&tmW);
        ptx::prefetch_tensormap(&tmS);
    }
    if (warp == 3) ptx::tmem_alloc(tmem_slot, 512);
    ptx::tc_fence_before_sync();
    __syncthreads();
    ptx::tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;
    // a programmatic dependent of whatever precedes it on the stream: what is above runs under the predecessor's end
    ptx::grid_dependency_wait();

    // The three single-thread roles: one elected thread runs the whole loop.  A role's time per stage is its
    // chain of dependent instructions (about five cycles each), so these loops are kept short.
    if (warp == 0) {
        // ------------------------------------------------ TMA producer of the nibble tiles
        if (ptx::elect_one()) {
            const int kstages = in_reg(p.kstages);
            int s = 0;
            uint32_t ph = 1;
            bool ok = true;
            for (int t = blockIdx.x; t < p.num_tiles && ok && !*abort_flag; t += gridDim.x) {
                const int x = (t / p.num_m_tiles) * (RT_N / 2);
                for (int st = 0; st < kstages; ++st) {
                    if (!ptx::mbar_wait(&w_empty[s], ph)) { ok = false; break; }
                    ptx::mbar_arrive_expect_tx(&w_full[s], W_BYTES);
                    ptx::tma_load_2d(smem + R_W_OFFSET + s * W_BYTES, &tmW, &w_full[s], x, st * RK);
                    if (++s == W_STAGES) { s = 0; ph ^= 1; }
                }
            }
            if (!ok) { *abort_flag = 1; atomicExch(a.status, 5); }
        }
        __syncwarp();
        // the successor may start (its set-up allocates tensor memory: every CTA of this grid has its own by now)
        asm volatile("griddepcontrol.launch_dependents;");
    } else if (warp == 1) {
        // ------------------------------------------------ TMA producer of the src tiles
        if (ptx::elect_one()) {
            int s = 0;
            uint32_t ph = 1;
            bool ok = true;
            const int kstages = in_reg(p.kstages);
            const uint32_t bytes = (uint32_t)in_reg(p.tile_rows * RK * 2);
            for (int t = blockIdx.x; t < p.num_tiles && ok && !*abort_flag; t += gridDim.x) {
                const int m0 = (t % p.num_m_tiles) * p.tile_rows;
                for (int st = 0; st < kstages; ++st) {
                    if (!ptx::mbar_wait(&ab_empty[s], ph)) { ok = false; break; }
                    uint8_t *d = smem + R_B_OFFSET + s * B_BYTES;
                    ptx::mbar_arrive_expect_tx(&ab_full[s], bytes); // (k beyond K reads as zeros and counts)
                    ptx::tma_load_2d(d, &tmS, &ab_full[s], st * RK, m0);
                    ptx::tma_load_2d(d + B_BYTES / 2, &tmS, &ab_full[s], st * RK + RK / 2, m0);
                    if (++s == STAGES) { s = 0; ph ^= 1; }
                }
            }
            if (!ok) { *abort_flag = 1; atomicExch(a.status, 5); }
        }
    } else if (warp == 2) {
        // ------------------------------------------------ MMA issuer
        if (ptx::elect_one()) {
            const int kstages = in_reg(p.kstages), ksteps = in_reg(p.ksteps), group_steps = in_reg(p.group_steps);
            const uint32_t idesc = (uint32_t)in_reg((int)p.idesc);
            int s = 0, buf = 0;
            uint32_t ph = 0, pacc = 1;
            bool ok = true;
            for (int t = blockIdx.x; t < p.num_tiles && ok && !*abort_flag; t += gridDim.x) {
                int left = 0; // k16 steps left in the open group (0: none open)
                int todo = ksteps;
                for (int st = 0; st < kstages && ok; ++st) {
                    if (!ptx::mbar_wait(&ab_full[s], ph)) { ok = false; break; }
                    ptx::tc_fence_after_sync();
                    const uint64_t bd = ptx::smem_desc_sw128(ptx::smem_u32(smem + R_B_OFFSET + s * B_BYTES), 0, 1024);
                    const uint32_t ta = tmem_base + R_A_COL0 + s * A_SLOT_COLS;
                    if (todo >= SPS && (left >= SPS || (left == 0 && group_steps >= SPS))) {
                        // the common stage, whole and inside one group: straight-line code
                        const bool fresh = left == 0;
                        if (fresh) {
                            if (!ptx::mbar_wait(&acc_empty[buf], pacc)) { ok = false; break; }
                            ptx::tc_fence_after_sync();
                            left = min(group_steps, todo);
                        }
                        const uint32_t d = tmem_base + buf * RT_M;
#pragma unroll
                        for (int q = 0; q < SPS; ++q)
                            mma_ts_16bit(d, ta + 8 * q, bd + (uint64_t)((q >> 2) * (B_BYTES / 2 >> 4) + (q & 3) * 2), idesc, q > 0 || !fresh);
                        left -= SPS;
                        if (left == 0) {
                            ptx::tc_commit(&acc_full[buf]);
                            if (++buf == ACC_BUFS) { buf = 0; pacc ^= 1; }
                        }
                    } else {
                        const int nst = min(SPS, todo);
                        for (int q = 0; q < nst; ++q) {
                            const bool fresh = left == 0;
                            if (fresh) {
                                if (!ptx::mbar_wait(&acc_empty[buf], pacc)) { ok = false; break; }
                                ptx::tc_fence_after_sync();
                                left = min(group_steps, todo - q);
                            }
                            mma_ts_16bit(tmem_base + buf * RT_M, ta + 8 * q,
                                    bd + (uint64_t)((q >> 2) * (B_BYTES / 2 >> 4) + (q & 3) * 2), idesc, !fresh);
                            if (--left == 0) {
                                ptx::tc_commit(&acc_full[buf]);
                                if (++buf == ACC_BUFS) { buf = 0; pacc ^= 1; }
                            }
                        }
                    }
                    todo -= SPS;
                    ptx::tc_commit(&ab_empty[s]); // src tile and operand slot are free once these MMAs have read them
                    if (++s == STAGES) { s = 0; ph ^= 1; }
                }
            }
            if (!ok) { *abort_flag = 1; atomicExch(a.status, 5); }
        }
    } else if (warp >= R_CONV0 && warp < R_EPI0) {
        // ------------------------------------------------ converters: nibbles -> exact 16-bit w - zero_point
        // Warp (q = warp % 4, r): TMEM lanes 32q .. 32q+31, the stages of parity r.  Lane (g, tq) owns the
        // columns 32q + 4g .. +3 (two bytes of a row) and, per k16 step, the k-rows 2tq, 2tq+1, 2tq+8, 2tq+9.
        // Byte h, low nibble goes to TMEM lane 32q + 16h + g, the high one to 32q + 16h + 8 + g.
        const int q = warp & 3, r = (warp - R_CONV0) >> 2;
        const int g = lane >> 2, tq = lane & 3;
        uint32_t off[4]; // 64-byte rows, 64B swizzle: 16-byte chunk index XOR ((row >> 1) & 3)
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const uint32_t row = 2 * tq + (i & 1) + 8 * (i >> 1);
            off[i] = row * 64 + (((uint32_t)q ^ ((row >> 1) & 3)) << 4) + 2 * g;
        }
        const int kstages = in_reg(p.kstages), ksteps = in_reg(p.ksteps), group_steps = in_reg(p.group_steps);
        const int zp_mode = in_reg(p.zp_mode), zp_dt = in_reg(a.wei_zp.dt);
        const uint32_t magic = (uint32_t)in_reg(F16 ? (p.sgn4 ? 0x64086408 : 0x64006400) : (p.sgn4 ? 0x00080008 : 0));
        const uint32_t magic_hi = (uint32_t)in_reg((F16 ? 0x64006400 : 0) | (p.sgn4 ? 0x00800080 : 0)); // the high nibble in its place
        const int base_off = in_reg(p.sgn4 ? 8 : 0);
        const int zt = zp_mode == 2 ? load_int(zp_dt, a.wei_zp.ptr, 0) : 0;
        // offsets of the four columns, as packed pairs: what the packed subtraction (or the f16 fma) takes
        uint32_t o2[4];
        // v = zero-point + 8 for s4.  bf16: -v / 64.  f16: 1024 + v in units of the last place (half as large below
        // 1024), or -(64 + v); 8-bit zero-points go through a conversion.
        const bool zp4 = zp_mode == 0 || zp_dt == DT_U4 || zp_dt == DT_S4;
        auto set_offsets = [&](uint32_t raw) {
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const int v = base_off + (zp_mode == 1 ? zp_of(zp_dt, raw, c) : zt);
                const int u = v + min(v, 0);
                uint32_t b;
                if (!F16) b = __float_as_uint((float)v * -0.015625f) >> 16; // exact for 4-bit zero-points
                else if (zp4) b = (c & 1) ? 0xD400u + 16 * u : 0x6400u + u;
                else b = __half_as_ushort(__int2half_rn((c & 1) ? -(64 + v) : 1024 + v));
                o2[c] = b * 0x10001u;
            }
        };
        set_offsets(0u);
        int turn = r; // stages until this warp's next one
        int sw = 0, s = 0;
        uint32_t pw = 0, ph = 1;
        bool ok = true;
        for (int t = blockIdx.x; t < p.num_tiles && ok && !*abort_flag; t += gridDim.x) {
            const int64_t n = (int64_t)(t / p.num_m_tiles) * RT_N + 32 * q + 4 * g;
            // Zero-points: the four lanes of a column group load those of four K-groups, one each, and the next
            // four while these are in use (a load under this kernel's own traffic takes longer than a stage)
            const int groups = zp_mode == 1 ? (ksteps + group_steps - 1) / group_steps : 0;
            auto fetch = [&](int batch) { return 4 * batch + tq < groups ? load_zp4(a, 4 * batch + tq, n) : 0u; };
            int batch = 0, gi = 0, left = group_steps; // batch held in zcur; group of the next step, its steps left
            bool fresh = true; // the offsets of group gi are not set yet
            uint32_t zcur = fetch(0), znext = fetch(1);
            auto open_group = [&]() {
                if (!fresh || gi >= groups) return;
                fresh = false;
                if (gi >> 2 != batch) {
                    zcur = gi >> 2 == batch + 1 ? znext : fetch(gi >> 2); // (the other converter's stage held a whole batch)
                    batch = gi >> 2;
                    znext = fetch(batch + 1);
                }
                set_offsets(__shfl_sync(0xffffffffu, zcur, (lane & ~3) | (gi & 3)));
            };
            auto advance = [&](int steps) {
                left -= steps;
                while (left <= 0) { left += group_steps; ++gi; fresh = true; }
            };
            for (int st = 0; st < kstages; ++st) {
                if (turn-- == 0) {
                    turn = CONV_SETS - 1;
                    if (!MULTI && zp_mode == 1) {
                        open_group();
                        advance(SPS);
                    }
                    if (!warp_wait(&w_full[sw], pw)) { ok = false; break; }
                    const uint8_t *raw = smem + R_W_OFFSET + sw * W_BYTES;
                    const uint32_t slot = tmem_base + ((uint32_t)(32 * q) << 16) + R_A_COL0 + s * A_SLOT_COLS;
#pragma unroll
                    for (int half = 0; half < 2; ++half) {
                        uint32_t w[4][4]; // [step][k-row], two bytes each
#pragma unroll
                        for (int k = 0; k < 4; ++k)
#pragma unroll
                            for (int i = 0; i < 4; ++i)
                                w[k][i] = *reinterpret_cast<const unsigned short *>(raw + (4 * half + k) * 1024 + off[i]);
                        if (half == 0) {
                            if (!warp_wait(&ab_empty[s], ph)) { ok = false; break; }
                            ptx::tc_fence_after_sync();
                        } else {
                            __syncwarp();
                            if (lane == 0) ptx::mbar_arrive(&w_empty[sw]);
                        }
                        uint32_t oz[MULTI ? 4 : 1][4]; // the offsets of each step
#pragma unroll
                        for (int k = 0; k < (MULTI ? 4 : 1); ++k) {
                            if (MULTI) {
                                open_group();
                                advance(1);
                            }
#pragma unroll
                            for (int c = 0; c < 4; ++c) oz[k][c] = o2[c];
                        }
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            const uint32_t sel = h ? 0x5511u : 0x4400u; // byte h of both rows
                            uint32_t o[16];
#pragma unroll
                            for (int k = 0; k < 4; ++k) {
                                const uint32_t ol = oz[MULTI ? k : 0][2 * h], oh = oz[MULTI ? k : 0][2 * h + 1];
                                const uint32_t x01 = perm(w[k][0], w[k][1], sel), x23 = perm(w[k][2], w[k][3], sel);
                                if (F16) {
                                    o[4 * k + 0] = sub_f16x2(and_xor(x01, 0x000F000Fu, magic), ol);
                                    o[4 * k + 1] = fma_f16x2(and_xor(x01, 0x00F000F0u, magic_hi), 0x2C002C00u, oh);
                                    o[4 * k + 2] = sub_f16x2(and_xor(x23, 0x000F000Fu, magic), ol);
                                    o[4 * k + 3] = fma_f16x2(and_xor(x23, 0x00F000F0u, magic_hi), 0x2C002C00u, oh);
                                } else {
                                    o[4 * k + 0] = fma_bf16x2(and_xor(x01, 0x000F000Fu, magic), 0x7F007F00u, ol);
                                    o[4 * k + 1] = fma_bf16x2(and_xor(x01, 0x00F000F0u, magic_hi), 0x7D007D00u, oh);
                                    o[4 * k + 2] = fma_bf16x2(and_xor(x23, 0x000F000Fu, magic), 0x7F007F00u, ol);
                                    o[4 * k + 3] = fma_bf16x2(and_xor(x23, 0x00F000F0u, magic_hi), 0x7D007D00u, oh);
                                }
                            }
                            st_16x128b_x8(slot + ((uint32_t)(16 * h) << 16) + 32 * half, o);
                        }
                    }
                    if (!ok) break;
                    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                    ptx::tc_fence_before_sync();
                    __syncwarp(); // every lane's stores to tensor memory are done
                    if (lane == 0) ptx::mbar_arrive(&ab_full[s]);
                } else if (zp_mode == 1) {
                    advance(SPS);
                }
                if (++sw == W_STAGES) { sw = 0; pw ^= 1; }
                if (++s == STAGES) { s = 0; ph ^= 1; }
            }
        }
        if (!ok) { *abort_flag = 1; atomicExch(a.status, 5); }
    } else if (warp >= R_EPI0) {
        // ------------------------------------------------ epilogue: tot += scale * group sum, then the store
        const int q = warp & 3, h = (warp - R_EPI0) >> 2;
        // 16-row pieces of the tile, dealt to the warps of a lane quarter in turn
        const int pieces = p.tile_rows / 16;
        const int each = (pieces + R_EPI_WARPS / 4 - 1) / (R_EPI_WARPS / 4);
        const int c0 = h * each, cn = in_reg(max(0, min(each, pieces - c0)));
        const int col = 32 * q + 4 * (lane & 7) + 2 * (lane >> 4) + ((lane >> 3) & 1);
        const int groups = in_reg((p.ksteps + p.group_steps - 1) / p.group_steps);
        const int sc_dt = in_reg(a.wei_scale.dt), N = in_reg((int)a.N);
        const int sc_size = sc_dt == DT_F32 ? 4 : sc_dt == DT_BF16 || sc_dt == DT_F16 ? 2 : 1;
        const int sc_pitch = in_reg((a.wei_scale.mask & 1) ? (int)a.wei_scale.ld * sc_size : 0); // N < 2^29 elements
        float ssc = 1.f;
        if (a.src_scale.ptr) ssc = load_float(a.src_scale.dt, a.src_scale.ptr, 0);
        else if (a.src_scale.on_host) ssc = a.src_scale.host_value;
        int buf = 0;
        uint32_t pacc = 0;
        bool ok = true;
        for (int t = blockIdx.x; t < p.num_tiles && ok && !*abort_flag; t += gridDim.x) {
            const int64_t n = (int64_t)(t / p.num_m_tiles) * RT_N + col;
            const int m0 = (t % p.num_m_tiles) * p.tile_rows;
            uint64_t tot[EPI_PIECES][8]; // pairs of rows: the packed FMA takes half the issue slots
#pragma unroll
            for (int c = 0; c < EPI_PIECES; ++c)
#pragma unroll
                for (int j = 0; j < 8; ++j) tot[c][j] = 0ull;
            // Scales of two groups at a time, loaded as raw bits while the two before are folded: a conversion
            // beside the load would wait for it
            const char *sc_ptr = (const char *)a.wei_scale.ptr + n * sc_size;
            auto raw_scale = [&](int g) -> uint32_t {
                if (g >= groups || n >= N) return 0u;
                const char *e = sc_ptr + (int64_t)g * sc_pitch;
                if (sc_dt == DT_F32) return ld_early_u32((const uint32_t *)e);
                if (sc_size == 2) return ld_early_u16((const unsigned short *)e);
                return __float_as_uint(load_float(sc_dt, e, 0));
            };
            auto scale_of = [&](uint32_t raw) {
                return sc_dt == DT_BF16 ? __uint_as_float(raw << 16)
                        : sc_dt == DT_F16 ? __half2float(__ushort_as_half((unsigned short)raw)) : __uint_as_float(raw);
            };
            uint32_t cur[2], nxt[2];
#pragma unroll
            for (int i = 0; i < 2; ++i) nxt[i] = raw_scale(i);
            for (int g0 = 0; g0 < groups && ok; g0 += 2) {
#pragma unroll
                for (int i = 0; i < 2; ++i) cur[i] = nxt[i];
#pragma unroll
                for (int i = 0; i < 2; ++i) nxt[i] = raw_scale(g0 + 2 + i);
#pragma unroll 1
                for (int i = 0; i < 2 && g0 + i < groups; ++i) {
                const float sc = scale_of(i == 0 ? cur[0] : cur[1]);
                const uint64_t sc2 = pack2(__float_as_uint(sc), __float_as_uint(sc));
                if (!warp_wait(&acc_full[buf], pacc)) { ok = false; break; }
                ptx::tc_fence_after_sync();
                const uint32_t acc = tmem_base + ((uint32_t)(32 * q) << 16) + buf * RT_M + c0 * 16;
#pragma unroll
                for (int c = 0; c < EPI_PIECES; ++c) {
                    if (c < cn) {
                        uint32_t v[16];
                        ptx::tmem_ld_32x16(acc + 16 * c, v);
                        ptx::tmem_ld_wait();
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            uint64_t sum = pack2(v[2 * j], v[2 * j + 1]);
                            // bf16: the operand was (w - zero_point) / 64; the 64 goes on the sum (a scale above
                            // 2^122 would overflow), exactly
                            if (!F16) sum = mul_f32x2(sum, 0x4280000042800000ull);
                            fma_f32x2(tot[c][j], sc2, sum);
                        }
                    }
                }
                ptx::tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) ptx::mbar_arrive(&acc_empty[buf]);
                if (++buf == ACC_BUFS) { buf = 0; pacc ^= 1; }
                }
            }
            if (!ok) break;
            if (n < a.N) {
#pragma unroll
                for (int c = 0; c < EPI_PIECES; ++c) {
                    if (c >= cn) continue;
                    const int64_t mc = m0 + (c0 + c) * 16;
                    const int rows = (int)min((int64_t)16, min((int64_t)m0 + p.tile_rows, a.M) - mc);
                    float d[16];
#pragma unroll
                    for (int j = 0; j < 16; ++j) d[j] = __uint_as_float((uint32_t)(tot[c][j >> 1] >> (32 * (j & 1)))) * ssc;
                    if (p.fast_store && !a.bias) {
                        const int64_t o = mc * a.dst_sm + n;
                        if (a.dst_dt == DT_BF16) {
                            unsigned short *dp = (unsigned short *)a.dst + o;
#pragma unroll
                            for (int j = 0; j < 16; ++j)
                                if (j < rows) dp[j * a.dst_sm] = f32_to_bf16_bits(d[j]);
                        } else if (a.dst_dt == DT_F16) {
                            __half *dp = (__half *)a.dst + o;
#pragma unroll
                            for (int j = 0; j < 16; ++j)
                                if (j < rows) dp[j * a.dst_sm] = __float2half_rn(d[j]);
                        } else {
                            float *dp = (float *)a.dst + o;
#pragma unroll
                            for (int j = 0; j < 16; ++j)
                                if (j < rows) dp[j * a.dst_sm] = d[j];
                        }
                    } else {
#pragma unroll
                        for (int j = 0; j < 16; ++j)
                            if (j < rows) finish_store_general(a, d[j], mc + j, n);
                    }
                }
            }
        }
        if (!ok) { *abort_flag = 1; atomicExch(a.status, 5); }
    }

    // ---------------------------------------------------- teardown
    ptx::tc_fence_before_sync();
    __syncthreads();
    if (warp == 3) {
        __syncwarp();
        ptx::tc_fence_after_sync();
        ptx::tmem_dealloc(tmem_base, 512);
    }
}

typedef CUresult (*encode_tiled_fn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
        const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
        CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

encode_tiled_fn rows_get_encode() {
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

template <bool F16, bool MULTI>
int rows_launch(const CUtensorMap &tw, const CUtensorMap &ts, const MatmulArgs &a, const RowsParams &p, int sm_count,
        cudaStream_t st) {
    auto kern = woq_rows_kernel<F16, MULTI>;
    static std::atomic<unsigned long long> configured;
    if (!opt_in_dynamic_smem(kern, R_SMEM_BYTES, configured)) return 5;
    cudaLaunchConfig_t cfg {};
    cfg.gridDim = dim3((unsigned)(p.num_tiles < sm_count ? p.num_tiles : sm_count));
    cfg.blockDim = dim3((unsigned)R_THREADS);
    cfg.dynamicSmemBytes = (size_t)R_SMEM_BYTES;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, tw, ts, a, p);
    count_launch("woq_rows");
    if (e != cudaSuccess) {
        (void)cudaGetLastError();
        set_last_error(std::string("cuda:tcgen05:woq4_rows launch: ") + cudaGetErrorString(e));
        return 5;
    }
    return 0;
}

} // namespace

// TMA bases on 16 bytes; a lane reads the zero-points of four columns at once
bool woq_rows_pointers_ok(const MatmulArgs &a) {
    return (uintptr_t)a.wei % 16 == 0 && (uintptr_t)a.src % 16 == 0 && (uintptr_t)a.wei_zp.ptr % 4 == 0;
}

int launch_woq_rows(const MatmulArgs &a, int sm_count, cudaStream_t st) {
    if (a.M == 0 || a.N == 0) return 0;
    encode_tiled_fn enc = rows_get_encode();
    if (!enc) return 5;
    if (sm_count < 1) sm_count = 148;
    const int64_t group = (a.wei_scale.ptr && (a.wei_scale.mask & 1)) ? a.wei_scale.g0
            : (a.wei_zp.ptr && (a.wei_zp.mask & 1))                    ? a.wei_zp.g0
                                                                       : a.K;
    {
        // The decode kernel in blocks of up to 32 rows, where it is the faster one.  This kernel takes 0.4 us a stage of a wave of
        // tiles, and for every group end in it 0.38 and 0.0027 a row of the tile; nothing splits its K.
        // us a call, this kernel -> that one: 64 x 4096 x 4096 in groups of 128 31.6 -> 18.8, of 32 102 -> 29; 128 rows, f16, groups of
        // 64 63.6 -> 27; 40 x 8192 x 1024 66.6 -> 11.8; 48 x 8192 x 28672 139 -> 105; (a model without the CTAs' starts and ends sent
        // there, too:) 300 x 1024 x 4096 in groups of 64 20.6 -> 27.7, 128 x 1024 x 28672 in groups of 32 71 -> 92.
        // 300 x 4096 x 4096 in groups of 128 stays here (39.3).  Both models are for 16-bit scales with no or 4-bit zero-points per
        // group.  All others stay here: used for them too, the models were wrong by up to five times (f32 scales, when that kernel
        // read them one at a time, here / there: 64 x 4096 x 11008 in groups of 128 32.7 / 100, 300 x 4096 x 4096 in groups of 32 111 / 423).
        const int64_t mtiles = (a.M + RT_M - 1) / RT_M, rows = ((a.M + mtiles - 1) / mtiles + 15) / 16 * 16;
        const int64_t waves = (mtiles * ((a.N + RT_N - 1) / RT_N) + sm_count - 1) / sm_count;
        const float ends = (float)RK / (float)(group < 4 * RK ? group : 4 * RK), zp = a.wei_zp.ptr ? 0.07f : 0.f; // of groups in a stage
        const float here = 7.5f + (float)(waves * ((a.K + RK - 1) / RK)) * (0.4f + ends * (0.38f + 0.0027f * (float)rows + zp));
        if (a.M <= 65536 && woq_decode_common_form(a) && woq_decode_pointers_ok(a) && woq_decode_fits(a.M, a.K, group, a.wei_scale.dt, a.wei_zp.ptr && a.wei_zp.mask ? a.wei_zp.dt : -1)
                && woq_decode_us(a.M, a.N, a.K, group, a.wei_zp.ptr != nullptr, sm_count) < here)
            return launch_woq_decode(a, sm_count, st);
    }
    RowsParams p {};
    // as few row tiles as cover M, of equal size
    p.num_m_tiles = (int)((a.M + RT_M - 1) / RT_M);
    p.tile_rows = (int)(((a.M + p.num_m_tiles - 1) / p.num_m_tiles + 15) / 16 * 16);
    const int64_t tiles = (int64_t)p.num_m_tiles * ((a.N + RT_N - 1) / RT_N);
    if (tiles >= (1LL << 31)) return 3;
    p.num_tiles = (int)tiles;
    CUtensorMap tw, ts;
    {
        cuuint64_t dims[2] = {(cuuint64_t)(a.N / 2), (cuuint64_t)a.K};
        cuuint64_t strides[1] = {(cuuint64_t)(a.wei_sk / 2)};
        cuuint32_t box[2] = {RT_N / 2, RK};
        cuuint32_t estr[2] = {1, 1};
        if (enc(&tw, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void *>(a.wei), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE)
                != CUDA_SUCCESS)
            return 5;
    }
    {
        cuuint64_t dims[2] = {(cuuint64_t)a.K, (cuuint64_t)a.M};
        cuuint64_t strides[1] = {(cuuint64_t)(a.src_sm * 2)};
        cuuint32_t box[2] = {64, (cuuint32_t)p.tile_rows};
        cuuint32_t estr[2] = {1, 1};
        if (enc(&ts, CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, const_cast<void *>(a.src), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE)
                != CUDA_SUCCESS)
            return 5;
    }
    p.ksteps = (int)(a.K / 16);
    p.kstages = (int)((a.K + RK - 1) / RK);
    p.group_steps = (int)(group / 16);
    if (p.group_steps < 1 || p.group_steps > p.ksteps) p.group_steps = p.ksteps;
    p.sgn4 = a.wei_dt == DT_S4;
    p.zp_mode = !a.wei_zp.ptr ? 0 : (a.wei_zp.mask ? 1 : 2);
    p.fast_store = a.dst_sn == 1 && a.n_po == 0 && !a.dst_scale.ptr && !a.dst_scale.on_host
            && (a.dst_dt == DT_F32 || a.dst_dt == DT_BF16 || a.dst_dt == DT_F16);
    const bool f16 = a.src_dt == DT_F16;
    const uint32_t fmt = f16 ? ptx::FMT_F16 : ptx::FMT_BF16;
    p.idesc = ptx::make_idesc(ptx::CFMT_F32, fmt, fmt, false, false, RT_N, (uint32_t)p.tile_rows);
    const bool multi = p.group_steps % SPS != 0 && p.zp_mode == 1;
    if (f16) return multi ? rows_launch<true, true>(tw, ts, a, p, sm_count, st) : rows_launch<true, false>(tw, ts, a, p, sm_count, st);
    return multi ? rows_launch<false, true>(tw, ts, a, p, sm_count, st) : rows_launch<false, false>(tw, ts, a, p, sm_count, st);
}

} // namespace qmm
