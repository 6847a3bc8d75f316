// int4 weight-decompression matmul for few rows (token generation; more rows where woq_rows.cu would leave SMs idle or
// pay for small groups):
//   dst[M,N] = src[M,K] (bf16/f16) x dequant(weights[K,N] s4/u4 `ab`),
// scales per column or per (K-group, column), optional zero-points (fpmath
// apply_to_int; reference arithmetic: src/cpu/matmul/ref_matmul.cpp:193-233).
//
// The work is the HBM stream of the packed weights and, at that stream's rate,
// the instructions that make 16-bit floats of nibbles.  So the kernel has as few
// instructions per weight and as few hand-offs as possible: the weights are the
// 16-row operand of mma.sync, whose registers a lane builds itself - an operand in
// tensor memory costs the same conversion plus a store, a fence and two barrier
// hand-offs per stage between roles of one or two warps, and that chain, not a pipe,
// bounded the tensor-memory form of this kernel.
//   * A CTA is four consumer warps and a producer warp; a tile is 256 columns, 64 per
//     consumer warp, over a contiguous share of K.  A consumer warp meets nobody but the
//     producer: one wait and one arrival per stage of 64 k x 256 columns (8 KB).
//   * Two to four such CTAs share an SM (by registers), so one CTA's start and end run
//     under the others' streams, and 12 to 16 warps hide each other's latencies.
//   * The CTAs of a tile's K shares are a cluster and add their sums through distributed
//     shared memory, in rank order (the same sum every time): no scratch in global memory.
//   * w - zero_point is an integer that the src's type holds exactly.  bf16: a nibble u
//     under a zero upper byte is u * 2^-133 where it stands low and u * 2^-129 where it
//     stands high (the step from subnormal to normal numbers included); f16: u * 2^-24 and
//     u * 2^-20.  One LOP3 and one packed FMA make (w - zero_point) / 64 (f16: / 512) of two
//     nibbles, and the group's sum is multiplied by the 64.  What of a wide zero-point is not
//     exact is taken off the sums at the end.
// us a call, before (operand in tensor memory, two launches) -> now: 8192 x 28672, groups of 128, bf16, M = 1 49.3 -> 36.1,
// 8 57.9 -> 36.2, 16 73.8 -> 49.5, 32 83.9 -> 82.4; 4096 x 11008 f16, groups of 64, M = 13 41.1 -> 11.7; 4096 x 1024, groups of
// 32, M = 32 39.4 -> 14.6; 4096 x 4096, groups of 32, M = 4 21.6 -> 10.7.
// Other parameters, 8192 x 28672, groups of 128, bf16, that kernel / this one with scales and zero-points read one at a time and
// the zero-points taken off the sums / now: f32 scales M = 1 47 / 76 / 35, 16 71 / 113 / 48, 32 76 / 253 / 78; f32 scales
// and u4 zero-points in groups of 32, M = 1 90 / 204 / 57, 32 179 / 612 / 145; one s8 zero-point M = 1 47 / 74 / 35, 32 77 / 253 / 78;
// u8 ones per group (the only form still behind at 32 rows) M = 1 49 / 90 / 43, 16 73 / 144 / 60, 32 80 / 290 / 87.
// What bounds it: issue and the pipes behind it.  A stage is 64 LOP3, 32 PRMT, 64 packed FMAs, 16 MMAs and 20 shared-memory
// reads of a warp, about 350 cycles of a scheduler in a loop of nothing else, where the packed instructions of the two
// pipes get in each other's way (192 would be the busiest pipe alone); M = 32 is bound by mma.sync (8 cycles each).
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <string>

#include "device_math.cuh"
#include "launch.h"
#include "objects.hpp"
#include "decode_ptx.cuh"

namespace qmm {

namespace {

constexpr int WARPS = 4; // consumer warps
constexpr int THREADS = 32 * (WARPS + 1);
constexpr int NB = 64 * WARPS, NB_LOG = 8; // columns per tile
static_assert(NB == 1 << NB_LOG, "column slices are found by shifts");
constexpr int KS = 64; // k-rows per stage
constexpr int W_BYTES = KS * NB / 2;
constexpr int MAX_STAGES = 16;
constexpr int MAX_CLUSTER = 8;
constexpr int SMEM_PER_SM = 227 * 1024;
constexpr int BAR_BYTES = 2 * MAX_STAGES * 8 + 64;

// MT: blocks of 8 src rows
template <int MT>
struct WdCfg {
    static constexpr int CTAS = MT == 1 ? 4 : MT == 2 ? 3 : 2; // per SM: what the registers allow
    static constexpr int S_BYTES = 8 * MT * KS * 2; // src tile of a stage
    static constexpr int SMEM = (SMEM_PER_SM / CTAS - 1024) / 1024 * 1024; // 1 KB of each is the system's
};

struct WdParams {
    int ksteps; // K / 16
    int kstages; // ceil(K / 64)
    int rows; // src rows per CTA (at most 32)
    int group_steps; // k16 steps per quantization group (ksteps when not grouped along K)
    int sc_grouped; // scales have a row per group (else one row)
    int split_log; // log2 of the CTAs per tile = cluster size
    int sgn4; // weights are s4 (else u4)
    int fast_store; // no post-ops / dst scale, 16-bit or f32 dst rows that take 4-column vectors
    int zp_common; // one zero-point for the whole tensor
    int sc_bits, zp_bits; // of an element of the parameter rows; zp_bits 0: no rows
    int stages, stage_bytes, off_sc, off_zp; // ring
    int off_bars, off_held;
};

// Scales held as f32, 8 a lane, are kept in shared memory (a place of the lane's own) where the registers do not hold them.
template <int MT, bool SC32>
constexpr bool scales_held = SC32 && MT >= 3;
constexpr int HELD_BYTES = 32 * WARPS * 32;

__device__ __noinline__ void finish_store_cold(const MatmulArgs &a, float d, int64_t m, int64_t n) {
    if (a.bias) d = __fadd_rn(d, load_float(a.bias_dt, a.bias, m * a.bias_sm + n * a.bias_sn));
    finish_store(a, d, m, n, false);
}

// The part of a zero-point for which w - zero_point is exact in the src's type.  That is all of it but for s32 ones beyond these
// bounds and, with a bf16 src and s4 weights, u8 ones above 248.
template <bool F16>
__device__ __forceinline__ int exact_part(int z, int sgn4) {
    return F16 ? min(max(z, -1024), 1024) : min(max(z, -128), sgn4 ? 248 : 255);
}
// What the rest of the zero-points takes off the sums of src row m over k0 .. k1 - 1, in the columns n .. n + 7
template <bool F16>
__device__ __noinline__ void rest_terms(const MatmulArgs &a, const WdParams &p, int64_t m, int64_t n, int k0, int k1, float (&term)[8]) {
    for (int i = 0; i < 8; ++i) term[i] = 0.f;
    const int group = p.group_steps * 16;
    for (int k = k0; k < k1;) {
        const int g = k / group, end = min((g + 1) * group, k1);
        float sum = 0.f;
        for (; k < end; ++k) sum += load_float(a.src_dt, a.src, m * a.src_sm + k);
        for (int i = 0; i < 8 && n + i < a.N; ++i) {
            const int z = load_int(a.wei_zp.dt, a.wei_zp.ptr, p.zp_common ? 0 : g * a.wei_zp.ld + n + i);
            const float scale = load_float(a.wei_scale.dt, a.wei_scale.ptr, (p.sc_grouped ? g * a.wei_scale.ld : 0) + n + i);
            term[i] = fmaf((float)(z - exact_part<F16>(z, p.sgn4)) * scale, sum, term[i]);
        }
    }
}

// ZPM, zero-points: 0 none; 1 s4 / u4 per (group, column); 2 8-bit ones per (group, column); 3 those, or s32 ones, whose type has
// values that are not exact (see exact_part); 4 none, or one for the tensor.  What is exact of a zero-point goes into the
// weights; a warp that met a rest takes it off its sums after the loop, slowly.  SC32: the group's scales are held as f32
// (any type), else as 16-bit pairs.  STEPS: k16 steps that surely belong to one group (4: groups are multiples of 64 k, 2: of
// 32, 1: of 16).
// (0 is a form of its own, for 16-bit scales: the constant from a zero-point in it cost 1 to 10 %, 13 x 4096 x 11008 11.65 ->
// 12.08 us, 100 x 4096 x 4096 in groups of 32 33.8 -> 37.3.)
template <int MT, bool F16, int ZPM, bool SC32, int STEPS>
__global__ void __launch_bounds__(THREADS, WdCfg<MT>::CTAS)
woq_decode_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmS,
        const __grid_constant__ MatmulArgs a, const __grid_constant__ WdParams p) {
    using C = WdCfg<MT>;
    extern __shared__ __align__(1024) uint8_t smem[];
    float *const sums = reinterpret_cast<float *>(smem + p.stages * p.stage_bytes); // [rank][M][columns of this CTA's slice]
    uint64_t *full = (uint64_t *)(smem + p.off_bars);
    uint64_t *empty = full + MAX_STAGES, *sums_bar = empty + MAX_STAGES;
    const int warp = threadIdx.x / 32, lane = in_reg(threadIdx.x % 32);
    const int split_log = p.split_log, splits = 1 << split_log, rank = (int)blockIdx.x & (splits - 1), tile = (int)blockIdx.x >> split_log;
    const int m0 = (int)blockIdx.y * p.rows, M = min(p.rows, (int)a.M - m0); // this CTA's rows
    if (threadIdx.x == 0) {
        for (int s = 0; s < p.stages; ++s) {
            ptx::mbar_init(&full[s], 1);
            ptx::mbar_init(&empty[s], WARPS);
        }
        ptx::mbar_init(sums_bar, 1);
        ptx::fence_barrier_init();
        ptx::mbar_arrive_expect_tx(sums_bar, (uint32_t)M * NB * 4); // every CTA's share of this CTA's slice
        ptx::prefetch_tensormap(&tmW);
        ptx::prefetch_tensormap(&tmS);
    }
    __syncthreads();
    if (splits > 1) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); // sums_bar is ready
    const int st0 = (int)((unsigned)p.kstages * rank >> split_log), st1 = (int)((unsigned)p.kstages * (rank + 1) >> split_log);
    const uint32_t ring = ptx::smem_u32(smem);
    // Launched as a programmatic dependent of whatever precedes it on the stream: the set-up runs under the predecessor's
    // end, and every role waits for that end before it reads or writes memory.
    bool ok = true;
    if (warp == WARPS) {
        // ------------------------------------------------ producer: weights, src, parameter rows of a stage's groups
        if (ptx::elect_one()) {
            // (all parameters into registers before the wait: the first reads of the constant cache are slow)
            const int n0 = in_reg(tile * NB), ksteps = in_reg(p.ksteps), group_steps = in_reg(p.group_steps), stage_bytes = in_reg(p.stage_bytes);
            const uint32_t cols = (uint32_t)min((int64_t)NB, a.N - n0);
            const uint32_t sc_bytes = in_reg(cols * p.sc_bits / 8), zp_bytes = in_reg(cols * p.zp_bits / 8);
            const int sc_pitch = in_reg(NB * p.sc_bits / 8), zp_pitch = in_reg(NB * p.zp_bits / 8);
            const int off_sc = in_reg(p.off_sc), off_zp = in_reg(p.off_zp), stages = in_reg(p.stages);
            int first = st0 * (KS / 16);
            const int gi = first / group_steps;
            int r = first - gi * group_steps; // steps into the stage's first group
            const int64_t sc_ld = p.sc_grouped ? a.wei_scale.ld * p.sc_bits / 8 : 0, zp_ld = a.wei_zp.ld * p.zp_bits / 8;
            const char *sc_row = (const char *)a.wei_scale.ptr + gi * sc_ld + (int64_t)n0 * p.sc_bits / 8;
            const char *zp_row = (const char *)a.wei_zp.ptr + gi * zp_ld + (int64_t)n0 * p.zp_bits / 8;
            const uint64_t map_w = reinterpret_cast<uint64_t>(&tmW), map_s = reinterpret_cast<uint64_t>(&tmS);
            const uint32_t bars = ptx::smem_u32(full);
            uint32_t bar = bars, sw = ring;
            const uint32_t bars_end = bars + stages * 8;
            uint32_t ph = 1;
            ptx::grid_dependency_wait();
            for (int st = st0; st < st1; ++st) {
                if (!wait<200>(bar + MAX_STAGES * 8, ph)) { atomicExch(a.status, 5); break; }
                const int last = min(first + KS / 16, ksteps); // one past the stage's steps
                // rows of the groups that begin in the stage (of the one the CTA begins in, too)
                int rows = 0;
                if (st == st0 || r == 0 || r + (last - first) > group_steps)
                    rows = r + (last - first) <= group_steps ? 1 : (r + (last - first) + group_steps - 1) / group_steps;
                arrive_expect_tx(bar, W_BYTES + C::S_BYTES + rows * (sc_bytes + zp_bytes));
                tma_load(sw, map_w, bar, n0 / 2, st * KS);
                tma_load(sw + W_BYTES, map_s, bar, st * KS, m0);
                const char *sc = sc_row, *zp = zp_row;
                for (int i = 0; i < rows; ++i) {
                    bulk_load(sw + off_sc + i * sc_pitch, sc, sc_bytes, bar);
                    if (zp_bytes) bulk_load(sw + off_zp + i * zp_pitch, zp, zp_bytes, bar);
                    sc += sc_ld;
                    zp += zp_ld;
                }
                r += last - first;
                first = last;
                while (r >= group_steps) { r -= group_steps; sc_row += sc_ld; zp_row += zp_ld; }
                bar += 8;
                sw += stage_bytes;
                if (bar == bars_end) { bar = bars; sw = ring; ph ^= 1; }
            }
        }
        __syncwarp();
        asm volatile("griddepcontrol.launch_dependents;"); // the CTA's loads are all on their way
        ptx::grid_dependency_wait();
        if (splits > 1) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    } else {
        // ------------------------------------------------ consumers
        const int g = lane >> 2, t4 = lane & 3;
        const int stages = in_reg(p.stages), stage_bytes = in_reg(p.stage_bytes), group_steps = in_reg(p.group_steps);
        const int off_sc = in_reg(p.off_sc), off_zp = in_reg(p.off_zp);
        // the lane's 8 columns are one word of a k-row, at byte 32 * warp + 4 g; 128-byte swizzle: the 16-byte chunk
        // index is XORed with the row's low three bits.  Rows 2 t4, 2 t4 + 1 and 8 more of each k16 step: the 32 lanes
        // of a load hit 32 banks.
        const uint32_t chunk = (32 * warp + 4 * g) >> 4, within = (4 * g) & 15;
        const uint32_t lds0 = (2 * t4) * 128 + ((chunk ^ (uint32_t)(2 * t4)) << 4) + within;
        const uint32_t lds1 = (2 * t4 + 1) * 128 + ((chunk ^ (uint32_t)(2 * t4 + 1)) << 4) + within;
        // ldmatrix: lane l names row l % 8 of matrix l / 8; the matrices are the step's k-octets, of one block of 8 rows
        // or of two; 128-byte swizzle again: step q's octets are the chunks 2 q and 2 q + 1
        const uint32_t mrow = lane & 7, moct = (lane >> 3) & 1;
        const uint32_t lds_s = W_BYTES + (MT > 1 ? (lane >> 4) * 1024 : 0) + mrow * 128 + ((moct ^ mrow) << 4);
        const int col = 64 * warp + 8 * g; // in the tile
        // s4: the sign bit flipped, u = w + 8
        const uint32_t magic_lo = p.sgn4 ? 0x00080008u : 0u, magic_hi = p.sgn4 ? 0x00800080u : 0u;
        const uint32_t mul_lo = F16 ? 0x78007800u : 0x7F007F00u; // 2^15, 2^127
        const uint32_t mul_hi = F16 ? 0x68006800u : 0x7D007D00u; // 2^11, 2^123
        constexpr float UNIT = F16 ? 512.f : 64.f;
        const uint64_t unit2 = pack2(UNIT, UNIT);
        const float bias0 = p.sgn4 ? -8.f : 0.f;
        auto pack_const = [&](float v) -> uint32_t { // an integer / UNIT twice, exact in both types
            v *= 1.f / UNIT;
            if (F16) {
                const uint32_t h = __half_as_ushort(__float2half_rn(v));
                return h | (h << 16);
            }
            return perm(__float_as_uint(v), 0, 0x3232);
        };
        // a zero-point nibble z makes the constant zadd - z / UNIT: the subnormal z * 2^-133 (f16: 2^-24) times -2^127 (-2^15)
        const int zp_dt = in_reg(a.wei_zp.dt), sc_dt = in_reg(a.wei_scale.dt);
        const uint32_t zflip = zp_dt == DT_S4 ? 0x88888888u : 0u, zmul = mul_lo | 0x80008000u;
        const uint32_t zadd = pack_const(bias0 + (zp_dt == DT_S4 ? 8.f : 0.f));
        constexpr bool PER_COLUMN = ZPM >= 1 && ZPM <= 3;
        uint32_t zc[PER_COLUMN ? 8 : 1]; // -(bias + zero_point) / UNIT of the lane's columns
        if (!PER_COLUMN) zc[0] = pack_const(bias0);
        ptx::grid_dependency_wait();
        bool rest = false; // a zero-point was not exact
        if (ZPM == 4 && p.zp_common) {
            const int z = load_int(zp_dt, a.wei_zp.ptr, 0), exact = exact_part<F16>(z, p.sgn4);
            zc[0] = pack_const(bias0 - (float)exact);
            rest = z != exact;
        }
        uint64_t tot[4][MT][2]; // pairs of rows of the columns 2 j and 2 j + 1
        float acc[4][MT][4];
        auto clear = [&]() {
#pragma unroll
            for (int t = 0; t < MT; ++t) {
#pragma unroll
                for (int e = 0; e < 4; ++e) {
#pragma unroll
                    for (int j = 0; j < 4; ++j) acc[j][t][e] = 0.f;
                }
            }
        };
        clear();
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int t = 0; t < MT; ++t) tot[j][t][0] = tot[j][t][1] = 0ull;
        const int sc_pitch = NB * p.sc_bits / 8, zp_pitch = NB * p.zp_bits / 8;
        constexpr bool HELD = scales_held<MT, SC32>;
        const uint32_t held = ptx::smem_u32(smem + p.off_held) + 8 * (32 * warp + lane);
        uint32_t scales[SC32 ? 8 : 4]; // of the open group: f32 bits, or 16-bit pairs
        auto begin_group = [&](uint32_t so, int row) {
            uint32_t held_here[HELD ? 8 : 1];
            uint32_t *const scp = HELD ? held_here : scales;
            const uint32_t sc = ring + so + off_sc + row * sc_pitch;
            if constexpr (!SC32) {
                const uint4 v = lds128(sc + 2 * col);
                scp[0] = v.x; scp[1] = v.y; scp[2] = v.z; scp[3] = v.w;
            } else if (sc_dt == DT_F32) {
                const uint4 v = lds128(sc + 4 * col), w = lds128(sc + 4 * col + 16);
                scp[0] = v.x; scp[1] = v.y; scp[2] = v.z; scp[3] = v.w;
                scp[SC32 ? 4 : 0] = w.x; scp[SC32 ? 5 : 0] = w.y; scp[SC32 ? 6 : 0] = w.z; scp[SC32 ? 7 : 0] = w.w;
            } else if (sc_dt == DT_BF16 || sc_dt == DT_F16) {
                const uint4 v = lds128(sc + 2 * col);
                const uint32_t h[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const uint32_t b = i & 1 ? h[i / 2] >> 16 : h[i / 2] & 0xffffu;
                    scp[SC32 ? i : 0] = sc_dt == DT_BF16 ? b << 16 : __float_as_uint(__half2float(__ushort_as_half((unsigned short)b)));
                }
            } else {
                const uint32_t b[2] = {lds32(sc + col), lds32(sc + col + 4)};
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const unsigned char c = (unsigned char)(b[i / 4] >> (8 * (i & 3)));
                    scp[SC32 ? i : 0] = __float_as_uint(sc_dt == DT_F8_E4M3 ? e4m3_to_f32(c) : e5m2_to_f32(c));
                }
            }
            if constexpr (HELD) {
#pragma unroll
                for (int j = 0; j < 4; ++j) sts64(held + j * (8 * 32 * WARPS), held_here[HELD ? 2 * j : 0], held_here[HELD ? 2 * j + 1 : 0]);
            }
            if constexpr (ZPM == 2 || ZPM == 3) {
                const uint32_t zp = ring + so + off_zp + row * zp_pitch;
                const bool wide = ZPM == 3 && zp_dt == DT_S32;
                uint32_t b[2] = {0, 0};
                if (!wide) { b[0] = lds32(zp + col); b[1] = lds32(zp + col + 4); }
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const int u = (int)(b[i / 4] >> (8 * (i & 3))) & 255;
                    const int z = wide ? (int)lds32(zp + 4 * (col + i)) : zp_dt == DT_S8 ? (int)(signed char)u : u;
                    const int exact = ZPM == 3 ? exact_part<F16>(z, p.sgn4) : z;
                    zc[PER_COLUMN ? i : 0] = pack_const(bias0 - (float)exact);
                    rest |= z != exact;
                }
            }
            if constexpr (ZPM == 1) {
                const uint32_t zx = lds32(ring + so + off_zp + row * zp_pitch + (col >> 1)) ^ zflip;
                // two columns' constants at a time, like weights: the nibbles i and i + 4 in the halves of a word
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const uint32_t n2 = i ? zx >> (4 * i) : zx;
                    const uint32_t c2 = fma2<F16>(n2 & 0x000F000Fu, zmul, zadd);
                    zc[i] = perm(c2, 0, 0x1010);
                    zc[i + 4] = perm(c2, 0, 0x3232);
                }
            }
        };
        auto end_group = [&]() {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                float s0, s1; // columns col + 2 j and + 1
                if (HELD) {
                    const uint2 v = lds64(held + j * (8 * 32 * WARPS));
                    s0 = __uint_as_float(v.x);
                    s1 = __uint_as_float(v.y);
                } else if (SC32) {
                    s0 = __uint_as_float(scales[SC32 ? 2 * j : 0]);
                    s1 = __uint_as_float(scales[SC32 ? 2 * j + 1 : 0]);
                } else if (sc_dt == DT_BF16) {
                    s0 = __uint_as_float(scales[j] << 16);
                    s1 = __uint_as_float(scales[j] & 0xffff0000u);
                } else {
                    const float2 f = __half22float2(*reinterpret_cast<const __half2 *>(&scales[j]));
                    s0 = f.x;
                    s1 = f.y;
                }
                const uint64_t s02 = pack2(s0, s0), s12 = pack2(s1, s1);
#pragma unroll
                for (int t = 0; t < MT; ++t) {
#pragma unroll
                    for (int e = 0; e < 4; e += 2) {
                        uint64_t v = mul_f32x2(pack2(acc[j][t][e], acc[j][t][e + 1]), unit2);
                        tot[j][t][e / 2] = fma_f32x2(e < 2 ? s02 : s12, v, tot[j][t][e / 2]);
                    }
                }
            }
            clear();
        };
        // A k16 step in registers: the lane's words, one per row (rows beyond K are the zeros TMA filled in), and the src
        // fragments.  The steps are read one ahead of the one that is multiplied, and the next stage's barrier is asked a
        // step before its answer is used.
        struct Step {
            uint32_t w[4];
            uint32_t b[2 * MT];
        };
        auto load_step = [&](Step &x, uint32_t sw, int q) {
            x.w[0] = lds32(sw + lds0 + q * 2048);
            x.w[1] = lds32(sw + lds1 + q * 2048);
            x.w[2] = lds32(sw + lds0 + q * 2048 + 1024);
            x.w[3] = lds32(sw + lds1 + q * 2048 + 1024);
            const uint32_t bs = (sw + lds_s) ^ (q << 5); // (stages are multiples of 1024 bytes)
#pragma unroll
            for (int t = 0; t + 1 < MT; t += 2) ldsm_x4(x.b + 2 * t, bs + t * 1024);
            if (MT & 1) ldsm_x2(x.b + 2 * (MT - 1), bs + (MT - 1) * 1024);
        };
        auto multiply = [&](const Step &x) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const uint32_t sel = ((4 + j) << 12) | ((4 + j) << 8) | (j << 4) | j;
                // byte j of two k-rows, each in a 16-bit half: low nibble = column col + 2 j, high = + 1
                const uint32_t x01 = perm(x.w[0], x.w[1], sel), x23 = perm(x.w[2], x.w[3], sel);
                const uint32_t z0 = zc[PER_COLUMN ? 2 * j : 0], z1 = zc[PER_COLUMN ? 2 * j + 1 : 0];
                uint32_t w[4];
                w[0] = fma2<F16>(and_xor(x01, 0x000F000Fu, magic_lo), mul_lo, z0);
                w[1] = fma2<F16>(and_xor(x01, 0x00F000F0u, magic_hi), mul_hi, z1);
                w[2] = fma2<F16>(and_xor(x23, 0x000F000Fu, magic_lo), mul_lo, z0);
                w[3] = fma2<F16>(and_xor(x23, 0x00F000F0u, magic_hi), mul_hi, z1);
#pragma unroll
                for (int t = 0; t < MT; ++t) mma<F16>(acc[j][t], w, x.b[2 * t], x.b[2 * t + 1]);
            }
        };

        int left = group_steps - (st0 * (KS / 16)) % group_steps; // k16 steps left in the open group piece
        bool fresh = true; // the next step opens a piece
        uint32_t ph = 0, so = 0; // parity and offset of the stage
        const uint32_t bars = ptx::smem_u32(full), ring_bytes = stages * stage_bytes;
        uint32_t bar = bars; // the stage's full barrier
        Step x0, x1;
        ok = __all_sync(0xffffffffu, wait<20>(bar, 0));
        if (ok && st0 < st1) load_step(x0, ring, 0);
        for (int st = st0; st < st1 && ok; ++st) {
            const uint32_t sw = ring + so;
            uint32_t pn = ph, son = so + stage_bytes, barn = bar + 8;
            if (son == ring_bytes) { son = 0; barn = bars; pn ^= 1; }
            uint32_t ready = 1;
            int row = (STEPS != 4 && !fresh) ? 1 : 0; // parameter row of the next group that begins here (row 0: the one open already)
            const int nsteps = STEPS == 4 ? 4 : min(4, p.ksteps - st * 4);
            if (STEPS == 4 && fresh) begin_group(so, 0);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                Step &cur = q & 1 ? x1 : x0, &next = q & 1 ? x0 : x1;
                if (q < 3) {
                    load_step(next, sw, q + 1);
                    if (q == 2 && st + 1 < st1) ready = try_wait(barn, pn);
                } else {
                    if (STEPS == 4) { // everything of the stage is in registers
                        __syncwarp();
                        if (lane == 0) arrive(bar + MAX_STAGES * 8);
                    }
                    if (!__all_sync(0xffffffffu, ready)) ready = __all_sync(0xffffffffu, wait_long<20>(barn, pn));
                    load_step(next, ring + son, 0); // (after the last stage: what a stage holds by then, not used)
                }
                if (STEPS == 4 || q < nsteps) {
                    if (STEPS != 4 && q % STEPS == 0 && fresh) begin_group(so, row++);
                    multiply(cur);
                    if (q % STEPS == STEPS - 1) {
                        left -= STEPS; // (beyond K, in the last stage, everything read is zero)
                        fresh = left <= 0;
                        if (fresh) {
                            end_group();
                            left += group_steps;
                        }
                    }
                }
            }
            if (STEPS != 4) {
                __syncwarp();
                if (lane == 0) arrive(bar + MAX_STAGES * 8);
            }
            ok = ready;
            bar = barn;
            so = son;
            ph = pn;
        }
        if (!ok) atomicExch(a.status, 5);
        else if (!fresh) end_group(); // the share ends inside a group
        if (ZPM >= 3 && __any_sync(0xffffffffu, rest)) {
#pragma unroll
            for (int t = 0; t < MT; ++t) {
                float t0[8], t1[8];
                const int m = 8 * t + 2 * t4;
                if (m >= M) continue;
                rest_terms<F16>(a, p, m0 + m, (int64_t)tile * NB + col, st0 * KS, min(st1 * KS, (int)a.K), t0);
                rest_terms<F16>(a, p, m0 + min(m + 1, M - 1), (int64_t)tile * NB + col, st0 * KS, min(st1 * KS, (int)a.K), t1);
#pragma unroll
                for (int i = 0; i < 8; ++i) tot[i / 2][t][i & 1] = fma_f32x2(pack2(-1.f, -1.f), pack2(t0[i], t1[i]), tot[i / 2][t][i & 1]);
            }
        }

        // -------------------------------------------- the sums go to the cluster's CTAs, a slice of the columns to each
        // (asynchronous stores that count themselves at the receiver's barrier: no CTA waits for another to read)
        if (splits > 1) asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); // long since complete
        const int slice_log = NB_LOG - split_log, slice = 1 << slice_log;
        const int owner = col >> slice_log, c = col & (slice - 1);
        const uint32_t sums_at = map_rank(ptx::smem_u32(sums), owner), bar_at = map_rank(ptx::smem_u32(sums_bar), owner);
#pragma unroll
        for (int t = 0; t < MT; ++t)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int m = 8 * t + 2 * t4 + h;
                if (m >= M) continue;
                auto v = [&](int j, int e) { return (uint32_t)(tot[j][t][e] >> (32 * h)); };
                const uint32_t at = sums_at + (uint32_t)((rank * M + m) * slice + c) * 4;
                st_async_v4(at, v(0, 0), v(0, 1), v(1, 0), v(1, 1), bar_at);
                st_async_v4(at + 16, v(2, 0), v(2, 1), v(3, 0), v(3, 1), bar_at);
            }
    }

    // ---------------------------------------------------- this CTA's slice: the sum over the ranks, in order -> dst
    const int slice_log = NB_LOG - split_log, slice = 1 << slice_log;
    float ssc = 1.f;
    if (a.src_scale.ptr) ssc = load_float(a.src_scale.dt, a.src_scale.ptr, 0);
    else if (a.src_scale.on_host) ssc = a.src_scale.host_value;
    const bool late = !ptx::mbar_wait(sums_bar, 0);
    if (late) atomicExch(a.status, 5);
    if (__syncthreads_or(late)) {
        if (splits > 1) ptx::outlast_cluster(sums_bar);
        return;
    }
    const int nvec = M << (slice_log - 2);
    for (int i = threadIdx.x; i < nvec; i += THREADS) {
        const int m = i >> (slice_log - 2), c = (i << 2) & (slice - 1);
        const int64_t n = (int64_t)tile * NB + rank * slice + c;
        if (n >= a.N) continue;
        const float *at = sums + m * slice + c;
        float4 v = *reinterpret_cast<const float4 *>(at);
        for (int r = 1; r < splits; ++r) {
            const float4 w = *reinterpret_cast<const float4 *>(at + r * M * slice);
            v.x += w.x; v.y += w.y; v.z += w.z; v.w += w.w;
        }
        float d[4] = {v.x * ssc, v.y * ssc, v.z * ssc, v.w * ssc};
        if (p.fast_store) { // N is a multiple of 32: the four columns exist
            if (a.bias) {
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    d[e] = __fadd_rn(d[e], load_float(a.bias_dt, a.bias, (m0 + m) * a.bias_sm + (n + e) * a.bias_sn));
            }
            const int64_t o = (int64_t)(m0 + m) * a.dst_sm + n;
            if (a.dst_dt == DT_F32) {
                *reinterpret_cast<float4 *>((float *)a.dst + o) = make_float4(d[0], d[1], d[2], d[3]);
            } else if (a.dst_dt == DT_BF16) {
                uint2 pk;
                pk.x = (uint32_t)f32_to_bf16_bits(d[0]) | ((uint32_t)f32_to_bf16_bits(d[1]) << 16);
                pk.y = (uint32_t)f32_to_bf16_bits(d[2]) | ((uint32_t)f32_to_bf16_bits(d[3]) << 16);
                *reinterpret_cast<uint2 *>((unsigned short *)a.dst + o) = pk;
            } else {
                uint2 pk;
                pk.x = (uint32_t)__half_as_ushort(__float2half_rn(d[0])) | ((uint32_t)__half_as_ushort(__float2half_rn(d[1])) << 16);
                pk.y = (uint32_t)__half_as_ushort(__float2half_rn(d[2])) | ((uint32_t)__half_as_ushort(__float2half_rn(d[3])) << 16);
                *reinterpret_cast<uint2 *>((unsigned short *)a.dst + o) = pk;
            }
        } else {
#pragma unroll
            for (int e = 0; e < 4; ++e) finish_store_cold(a, d[e], m0 + m, n + e);
        }
    }
}

typedef CUresult (*encode_tiled_fn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
        const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
        CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

encode_tiled_fn wd_get_encode() {
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

int wd_bits(int dt) {
    switch (dt) {
        case DT_F32: case DT_S32: return 32;
        case DT_BF16: case DT_F16: return 16;
        case DT_S4: case DT_U4: return 4;
        default: return 8;
    }
}

// Parameter rows that one stage can need: the groups its four k16 steps touch.
int wd_rows_per_stage(int group_steps) {
    if (group_steps % 4 == 0) return 1;
    if (4 % group_steps == 0) return 4 / group_steps;
    return (4 + group_steps - 2) / group_steps + 1;
}

// log2 of the CTAs per tile: the number that gives the busiest SM the least to do.  In units of a stage's instructions: a
// CTA's start and end count as 2 + mt stages, and a stage that has the SM to itself takes as long as 2.75 - mt / 4 that
// share it.  us a call with 1 / 2 / 4 / 8 CTAs per tile: K = 8192, N = 28672, M = 1: 50.4 / 39.4 / 36.8 / 35.1 (8 chosen),
// M = 32: 106 / 82.4 / 87.2 / 91.0 (2); M = 13, 4096 x 11008: - / 17.5 / 16.3 / 11.7 (8); M = 8, 1280 x 7008: - / 7.2 / 5.9 / 6.2 (8).
int wd_split_log(int64_t ntiles, int kstages, int mt, int sm_count) {
    int best = 0;
    int64_t cost = INT64_MAX;
    for (int l = 0; 1 << l <= MAX_CLUSTER && 1 << l <= kstages; ++l) {
        const int64_t busiest = ((ntiles << l) + sm_count - 1) / sm_count;
        const int64_t share = 4 * busiest > 11 - mt ? 4 * busiest : 11 - mt; // in quarters
        const int64_t c = share * (((kstages + (1 << l) - 1) >> l) + 2 + mt);
        if (c < cost) { cost = c; best = l; }
    }
    return best;
}

template <int MT, bool F16, int ZPM, bool SC32, int STEPS>
int wd_launch(const CUtensorMap &tw, const CUtensorMap &ts, const MatmulArgs &a, WdParams p, int ntiles, cudaStream_t st) {
    using C = WdCfg<MT>;
    auto kern = woq_decode_kernel<MT, F16, ZPM, SC32, STEPS>;
    const int rb = wd_rows_per_stage(p.group_steps);
    auto up128 = [](int v) { return (v + 127) / 128 * 128; };
    p.off_sc = W_BYTES + C::S_BYTES;
    p.off_zp = p.off_sc + up128(rb * NB * p.sc_bits / 8);
    p.stage_bytes = (p.off_zp + up128(rb * NB * p.zp_bits / 8) + 1023) / 1024 * 1024;
    const int sums_bytes = p.rows * NB * 4;
    // as many stages as the CTA's share of the SM holds; four where wide parameter rows leave fewer (then fewer CTAs fit an SM)
    constexpr int held_bytes = scales_held<MT, SC32> ? HELD_BYTES : 0;
    p.stages = (C::SMEM - BAR_BYTES - sums_bytes - held_bytes) / p.stage_bytes;
    p.stages = p.stages > MAX_STAGES ? MAX_STAGES : p.stages < 4 ? 4 : p.stages;
    p.off_bars = p.stages * p.stage_bytes + sums_bytes;
    p.off_held = p.off_bars + BAR_BYTES;
    const int smem_bytes = p.off_held + held_bytes;
    if (smem_bytes > SMEM_PER_SM) return 3; // (not reached: woq_decode_fits)
    static std::atomic<unsigned long long> configured;
    if (!opt_in_dynamic_smem(kern, SMEM_PER_SM, configured)) return 5;
    cudaLaunchConfig_t cfg {};
    cfg.gridDim = dim3((unsigned)ntiles << p.split_log, (unsigned)((a.M + p.rows - 1) / p.rows));
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = (size_t)smem_bytes;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1u << p.split_log;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    cudaError_t e = cudaLaunchKernelEx(&cfg, kern, tw, ts, a, p);
    if (e != cudaSuccess) {
        (void)cudaGetLastError();
        set_last_error(std::string("cuda:tcgen05:woq4 launch: ") + cudaGetErrorString(e));
        return 5;
    }
    count_launch("woq_decode");
    return 0;
}

template <int MT, bool F16>
int wd_choose(const CUtensorMap &tw, const CUtensorMap &ts, const MatmulArgs &a, const WdParams &p, int zpm, int ntiles, cudaStream_t st) {
#define QMM_WD(Z, S) \
    (p.group_steps % 4 == 0 ? wd_launch<MT, F16, Z, S, 4>(tw, ts, a, p, ntiles, st) \
                    : p.group_steps % 2 == 0 ? wd_launch<MT, F16, Z, S, 2>(tw, ts, a, p, ntiles, st) \
                                             : wd_launch<MT, F16, Z, S, 1>(tw, ts, a, p, ntiles, st))
    switch (zpm) {
        // (more than 24 rows, the registers short: form 4 spills less, and is the faster one where groups end seldom.  us a call,
        // 0 / 4: 32 x 8192 x 28672 bf16 in groups of 128 84.2 / 78.4, of 64 91.3 / 92.0; 32 x 8192 x 1024 f16, of 64 17.3 / 18.4)
        case 0: return MT == 4 && p.group_steps % 4 == 0 && p.group_steps >= 8 ? QMM_WD(4, true) : QMM_WD(0, false);
        case 1: return p.sc_bits == 16 ? QMM_WD(1, false) : QMM_WD(1, true);
        case 2: return QMM_WD(2, true);
        case 3: return QMM_WD(3, true);
        default: return QMM_WD(4, true);
    }
#undef QMM_WD
}

} // namespace

bool woq_decode_pointers_ok(const MatmulArgs &a) {
    return (uintptr_t)a.wei % 16 == 0 && (uintptr_t)a.src % 16 == 0 && (uintptr_t)a.wei_scale.ptr % 16 == 0
            && (uintptr_t)a.wei_zp.ptr % 16 == 0;
}

// Whether the kernel takes the problem: for more than 16 rows, parameter rows as wide as the weights themselves (groups
// of 16 with 32-bit scales and zero-points) go to the next implementation.  `group`: K-group of the parameters (K when there
// is none); types as DT_* (zp_dt < 0: no zero-points per group).
bool woq_decode_fits(int64_t M, int64_t K, int64_t group, int scale_dt, int zp_dt) {
    const int64_t ksteps = (K + 15) / 16;
    int64_t gs = group / 16;
    if (gs < 1 || gs > ksteps) gs = ksteps;
    const int rb = wd_rows_per_stage((int)gs);
    return M <= 16 || rb * NB * (wd_bits(scale_dt) + (zp_dt < 0 ? 0 : wd_bits(zp_dt))) / 8 < W_BYTES;
}

// 16-bit scales, and no zero-points or 4-bit ones per group: what woq_decode_us was fitted to
bool woq_decode_common_form(const MatmulArgs &a) {
    return wd_bits(a.wei_scale.dt) == 16 && (!a.wei_zp.ptr || (a.wei_zp.mask && wd_bits(a.wei_zp.dt) == 4));
}

// Microseconds that a problem takes here, for the choice between this kernel and the one whose operand lies in tensor
// memory (woq_rows.cu) when there are more than 32 rows.  The busiest SM's stages, with its CTAs' starts and ends, at 0.42 (0.62 for
// more than 24 rows), more with groups below 64 (a fold of the sums at each end).  Fitted, with that kernel's model, to 156
// problems (33 to 512 rows, K 1024 to 8192, N 1024 to 28672, groups of 32 to 128) timed with both: within 25 % of the time (10 % for
// eight of ten), and the choice costs 0.03 % on average, 3 % at most.
float woq_decode_us(int64_t M, int64_t N, int64_t K, int64_t group, bool zero_points, int sm_count) {
    if (sm_count < 1) sm_count = 148;
    const int64_t blocks = (M + 31) / 32, rows = (M + blocks - 1) / blocks, mt = (rows + 7) / 8;
    const int64_t tiles = (N + NB - 1) / NB * blocks, kstages = (K + KS - 1) / KS;
    const int l = wd_split_log(tiles, (int)kstages, (int)mt, sm_count);
    const float busiest = (float)(((tiles << l) + sm_count - 1) / sm_count), share = (float)((kstages + (1 << l) - 1) >> l);
    const float stage = (mt > 3 ? 0.62f : 0.42f) * (group >= 64 ? 1.f : zero_points ? 1.71f : 1.35f);
    return 3.2f + stage * (busiest > 1.1f ? busiest : 1.1f) * (share + 1.9f + 0.64f * (float)mt);
}

int launch_woq_decode(const MatmulArgs &a, int sm_count, cudaStream_t st) {
    if (a.M == 0 || a.N == 0) return 0;
    encode_tiled_fn enc = wd_get_encode();
    if (!enc) return 5;
    // more than 32 rows: equal blocks of them, each with CTAs of its own that read the weights again (from L2)
    const int blocks = (int)((a.M + 31) / 32), rows = (int)((a.M + blocks - 1) / blocks), mt = (rows + 7) / 8;
    CUtensorMap tw, ts;
    {
        cuuint64_t dims[2] = {(cuuint64_t)(a.N / 2), (cuuint64_t)a.K};
        cuuint64_t strides[1] = {(cuuint64_t)(a.wei_sk / 2)};
        cuuint32_t box[2] = {NB / 2, KS};
        cuuint32_t estr[2] = {1, 1};
        if (enc(&tw, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void *>(a.wei), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE)
                != CUDA_SUCCESS)
            return 5;
    }
    {
        // src rows as 16-bit words; rows beyond M and k beyond K read as zeros
        cuuint64_t dims[2] = {(cuuint64_t)a.K, (cuuint64_t)a.M};
        cuuint64_t strides[1] = {(cuuint64_t)((a.M > 1 ? a.src_sm : a.K) * 2)};
        cuuint32_t box[2] = {KS, (cuuint32_t)(8 * mt)};
        cuuint32_t estr[2] = {1, 1};
        if (enc(&ts, CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, const_cast<void *>(a.src), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE)
                != CUDA_SUCCESS)
            return 5;
    }
    WdParams p {};
    p.ksteps = (int)((a.K + 15) / 16);
    p.kstages = (int)((a.K + KS - 1) / KS);
    p.rows = rows;
    p.sc_grouped = a.wei_scale.mask & 1;
    const bool zp_rows = a.wei_zp.ptr && a.wei_zp.mask;
    const int64_t group = p.sc_grouped ? a.wei_scale.g0 : (zp_rows && (a.wei_zp.mask & 1)) ? a.wei_zp.g0 : a.K;
    p.group_steps = (int)(group / 16);
    // one group: its end is the end of the CTA's share (a multiple of four steps, for the widest form of the loop)
    if (p.group_steps < 1 || p.group_steps >= p.ksteps) p.group_steps = p.kstages * (KS / 16);
    p.sgn4 = a.wei_dt == DT_S4;
    p.zp_common = a.wei_zp.ptr && !a.wei_zp.mask;
    p.sc_bits = wd_bits(a.wei_scale.dt);
    p.zp_bits = zp_rows ? wd_bits(a.wei_zp.dt) : 0;
    const bool inexact = a.wei_zp.dt == DT_S32 || (a.wei_zp.dt == DT_U8 && a.src_dt == DT_BF16 && a.wei_dt == DT_S4);
    const int zpm = zp_rows ? (p.zp_bits == 4 ? 1 : inexact ? 3 : 2) : p.zp_common || p.sc_bits != 16 ? 4 : 0;
    {
        const int es = a.dst_dt == DT_F32 ? 4 : 2;
        p.fast_store = a.n_po == 0 && !a.dst_scale.ptr && !a.dst_scale.on_host
                && (a.dst_dt == DT_F32 || a.dst_dt == DT_BF16 || a.dst_dt == DT_F16) && a.dst_sn == 1
                && (a.M == 1 || a.dst_sm % 4 == 0) && (uintptr_t)a.dst % (4 * es) == 0;
    }
    const int ntiles = (int)((a.N + NB - 1) / NB);
    p.split_log = wd_split_log(ntiles * blocks, p.kstages, mt, sm_count > 0 ? sm_count : 148);
    const bool f16 = a.src_dt == DT_F16;
#define QMM_WD(MT) (f16 ? wd_choose<MT, true>(tw, ts, a, p, zpm, ntiles, st) : wd_choose<MT, false>(tw, ts, a, p, zpm, ntiles, st))
    return mt == 1 ? QMM_WD(1) : mt == 2 ? QMM_WD(2) : mt == 3 ? QMM_WD(3) : QMM_WD(4);
#undef QMM_WD
}

} // namespace qmm
