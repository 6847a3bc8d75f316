// What the 8-bit GEMM kernels share: the epilogue's arithmetic (a thread owns one dst column and some consecutive rows)
// and the tensor maps of their operands.
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "device_math.cuh"
#include "launch.h"
// waits of these kernels are long (a tile's mainloop, a ring that is full): let the hardware hold the
// polling thread for up to this many nanoseconds per poll (measured: 3 % on the fp8 GEMM)
#define QMM_TRY_WAIT_HINT_NS 2000
#include "sm100_ptx.cuh"

namespace qmm {

struct TcParams {
    int num_m_tiles, num_n_tiles, num_k_blocks;
    uint32_t idesc;
    int w_kmajor; // weights are `ba` (K contiguous)
#ifdef QMM_PROFILE
    int mainloop_only; // 1 no epilogue, 2 TMEM reads only, 3 everything but the stores, 4 binary operands read from one address (wrong results)
#endif
    int after_prekernel; // launched as the programmatic dependent of the column / row sum kernel before it
    const int32_t *colsum; // sum_k w[k][n]       (src zero-point compensation)
    const int32_t *rowsum; // sum_k s[m][k]       (weights zero-point compensation)
};

namespace {

constexpr int BT_N = 128; // dst columns per tile = TMEM lanes = UMMA M
constexpr int BKB = 128; // bytes (= 8-bit elements) of K per stage: one swizzle row
constexpr int UMMA_K = 32; // K per tcgen05.mma for 8-bit operands

// Per-column terms of the epilogue, in registers of the thread that owns the column.
struct ColTerms {
    float wei_scale; // 1 when absent
    float bias; // bias[n] when the bias is a row vector, else 0
    int zs_colsum; // src_zp * colsum[n] - K * src_zp * wei_zp[n]
    int wei_zp; // wei_zp[n]
    float dst_zp; // dst_zp[n] when per-N
};

template <bool INT>
__device__ __forceinline__ ColTerms load_col_terms(const MatmulArgs &a, const TcParams &tp, int64_t n) {
    ColTerms c;
    c.wei_scale = 1.f;
    c.bias = 0.f;
    c.zs_colsum = 0;
    c.wei_zp = 0;
    c.dst_zp = 0.f;
    if (n >= a.N) return c;
    if (a.dst_zp.ptr && a.dst_zp.mask > 0) c.dst_zp = (float)((const int *)a.dst_zp.ptr)[n];
    if (a.wei_scale.ptr) c.wei_scale = load_float(a.wei_scale.dt, a.wei_scale.ptr, (a.wei_scale.mask & 2) ? n : 0);
    else if (a.wei_scale.on_host) c.wei_scale = a.wei_scale.host_value;
    if (a.bias && a.bias_sm == 0) c.bias = load_float(a.bias_dt, a.bias, n * a.bias_sn);
    if (INT) {
        if (a.wei_zp.ptr) c.wei_zp = load_int(a.wei_zp.dt, a.wei_zp.ptr, (a.wei_zp.mask & 2) ? n : 0);
        if (a.src_zp.ptr && tp.colsum) { // (else the kernel makes the sums itself)
            const int zs = ((const int *)a.src_zp.ptr)[0];
            c.zs_colsum = zs * ptx::ld_dependent(tp.colsum + n) - (int)a.K * zs * c.wei_zp;
        }
    }
    return c;
}

// Per-tensor terms of the epilogue, read once per thread.
struct TensorTerms {
    bool has_dst_scale, has_dst_zp, dst_zp_per_n, row_scale, row_sum, bias_by_row;
    float dst_scale, dst_rcp, dst_zp, src_scale;
};

template <bool INT>
__device__ __forceinline__ TensorTerms load_tensor_terms(const MatmulArgs &a, const TcParams &tp) {
    TensorTerms t;
    t.has_dst_scale = a.non_default_attr && (a.dst_scale.ptr || a.dst_scale.on_host);
    t.dst_scale = a.dst_scale.ptr ? load_float(a.dst_scale.dt, a.dst_scale.ptr, 0) : a.dst_scale.host_value;
    t.dst_rcp = __frcp_rn(t.dst_scale);
    // the floating-point reference path has no dst zero-point
    t.has_dst_zp = a.non_default_attr && INT && a.dst_zp.ptr;
    t.dst_zp_per_n = a.dst_zp.mask > 0;
    t.dst_zp = (t.has_dst_zp && !t.dst_zp_per_n) ? (float)((const int *)a.dst_zp.ptr)[0] : 0.f;
    t.row_scale = a.src_scale.ptr && (a.src_scale.mask & 1);
    t.src_scale = 1.f; // per-tensor src scale (1 when absent or per-row)
    if (a.src_scale.ptr && !t.row_scale) t.src_scale = load_float(a.src_scale.dt, a.src_scale.ptr, 0);
    else if (a.src_scale.on_host) t.src_scale = a.src_scale.host_value;
    t.row_sum = INT && tp.rowsum != nullptr;
    t.bias_by_row = a.bias && a.bias_sm != 0;
    return t;
}

// Typed store of one f32 value, saturating / rounding as the reference does
// (src/cpu/simple_q10n.hpp:41-81; src/common/bfloat16.cpp:22-47: f32
// subnormals flush to signed zero before the bf16 rounding).
template <int DST>
__device__ __forceinline__ uint32_t typed_bits(float v) {
    if constexpr (DST == DT_F32) {
        return __float_as_uint(v);
    } else if constexpr (DST == DT_BF16) {
        if (fabsf(v) < 1.17549435e-38f) v = copysignf(0.f, v);
        unsigned short b = __bfloat16_as_ushort(__float2bfloat16_rn(v));
        if (v != v) b = (unsigned short)((__float_as_uint(v) >> 16) | 0x40u); // NaN: payload kept, quiet bit set
        return b;
    } else if constexpr (DST == DT_F16) {
        return __half_as_ushort(__float2half_rn(v));
    } else if constexpr (DST == DT_S32) {
        v = fminf(fmaxf(v, -2147483648.f), 2147483520.f);
        return (uint32_t)__float2int_rn(v);
    } else if constexpr (DST == DT_S8) {
        return (uint32_t)(unsigned char)(signed char)__float2int_rn(fminf(fmaxf(v, -128.f), 127.f));
    } else {
        return (uint32_t)(unsigned char)__float2int_rn(fminf(fmaxf(v, 0.f), 255.f));
    }
}
template <int DST>
__device__ __forceinline__ void store_bits(void *p, uint32_t b) {
    if constexpr (DST == DT_F32 || DST == DT_S32) *(uint32_t *)p = b;
    else if constexpr (DST == DT_BF16 || DST == DT_F16) *(unsigned short *)p = (unsigned short)b;
    else *(unsigned char *)p = (unsigned char)b;
}
template <int DST>
__device__ __forceinline__ void store_typed(void *p, float v) {
    store_bits<DST>(p, typed_bits<DST>(v));
}
template <int DST>
struct dst_size {
    static constexpr int value = (DST == DT_F32 || DST == DT_S32) ? 4 : (DST == DT_BF16 || DST == DT_F16) ? 2 : 1;
};

// 32 consecutive dst rows of column n, accumulators in r[0..31].  Absent
// scales are 1 and an absent bias is 0, which leaves values unchanged.
// FULL: all R rows exist (m0 + R <= M): no clamped row indices, no predicated stores.
template <bool INT, bool CHAIN, int DST, int R, bool FULL = false>
__device__ __forceinline__ void epilogue_rows(const MatmulArgs &a, const TcParams &tp, const TensorTerms &t,
        const ColTerms &c, const uint32_t (&r)[R], int64_t m0, int64_t n) {
    if (n >= a.N) return;
    char *dptr = (char *)a.dst + (m0 * a.dst_sm + n * a.dst_sn) * dst_size<DST>::value;
    const int64_t dstep = a.dst_sm * dst_size<DST>::value;
    const int rows = FULL ? R : (int)min((int64_t)R, a.M - m0);
    // Phases of straight-line code over the R rows (uniform conditions are
    // tested once per phase, not per row), so the rows' dependency chains
    // interleave; only the stores are predicated on the M tail.
    float d[R];
    if constexpr (INT) {
        if (t.row_sum) {
#pragma unroll
            for (int j = 0; j < R; ++j)
                d[j] = (float)((int)r[j] - c.zs_colsum - c.wei_zp * ptx::ld_dependent(tp.rowsum + (FULL ? m0 + j : min(m0 + j, a.M - 1))));
        } else {
#pragma unroll
            for (int j = 0; j < R; ++j) d[j] = (float)((int)r[j] - c.zs_colsum);
        }
    } else {
#pragma unroll
        for (int j = 0; j < R; ++j) d[j] = __uint_as_float(r[j]);
    }
    if (t.row_scale) {
        if (FULL && a.src_scale.dt == DT_F32) {
            const float *ss = (const float *)a.src_scale.ptr + m0; // (not __ldg: the call before may have written them)
#pragma unroll
            for (int j = 0; j < R; ++j) d[j] = __fmul_rn(d[j], ss[j]);
        } else {
#pragma unroll
            for (int j = 0; j < R; ++j)
                d[j] = __fmul_rn(d[j], load_float(a.src_scale.dt, a.src_scale.ptr, FULL ? m0 + j : min(m0 + j, a.M - 1)));
        }
    } else {
#pragma unroll
        for (int j = 0; j < R; ++j) d[j] = __fmul_rn(d[j], t.src_scale);
    }
#pragma unroll
    for (int j = 0; j < R; ++j) d[j] = __fadd_rn(__fmul_rn(d[j], c.wei_scale), c.bias);
    if constexpr (CHAIN) {
        if (t.bias_by_row) {
#pragma unroll
            for (int j = 0; j < R; ++j)
                d[j] = __fadd_rn(d[j],
                        load_float(a.bias_dt, a.bias, (FULL ? m0 + j : min(m0 + j, a.M - 1)) * a.bias_sm + n * a.bias_sn));
        }
        apply_post_ops_rows<R, (DST == DT_S8 || DST == DT_U8), FULL>(a, d, m0, n);
    }
    if (t.has_dst_scale) { // the reference divides; the same quotient from a reciprocal taken once per thread
#pragma unroll
        for (int j = 0; j < R; ++j) d[j] = div_by_scale(d[j], t.dst_scale, t.dst_rcp);
    }
    if (t.has_dst_zp) {
        const float z = t.dst_zp_per_n ? c.dst_zp : t.dst_zp;
#pragma unroll
        for (int j = 0; j < R; ++j) d[j] = __fadd_rn(d[j], z);
    }
#ifdef QMM_PROFILE
    if (tp.mainloop_only == 3) { // everything but the stores
        float acc = 0.f;
#pragma unroll
        for (int j = 0; j < R; ++j) acc += d[j];
        if (acc == 123.456f) store_typed<DST>(dptr, acc);
        return;
    }
#endif
    // (kernels with a post-op chain have no replicated form: they are short of registers as it is)
    if (CHAIN || a.peers.count == 0) {
#pragma unroll
        for (int j = 0; j < R; ++j)
            if (FULL || j < rows) store_typed<DST>(dptr + j * dstep, d[j]);
    } else {
        // every rank's copy of dst: the value is converted once and stored count + 1 times (plain
        // stores through peer-mapped addresses; the kernel's last CTA publishes the flags)
        uint32_t b[R];
#pragma unroll
        for (int j = 0; j < R; ++j) b[j] = typed_bits<DST>(d[j]);
#pragma unroll
        for (int j = 0; j < R; ++j)
            if (FULL || j < rows) store_bits<DST>(dptr + j * dstep, b[j]);
        for (int q = 0; q < a.peers.count; ++q) {
            char *pp = dptr + a.peers.delta[q];
#pragma unroll
            for (int j = 0; j < R; ++j)
                if (FULL || j < rows) store_bits<DST>(pp + j * dstep, b[j]);
        }
    }
}

// DSTT: the dst data type when the kernel was instantiated for one (post-op chain kernels: a single
// copy of the chain's code in the instruction stream), -1 to choose at run time.
template <bool INT, bool CHAIN, int R, int DSTT = -1>
__device__ __forceinline__ void epilogue_rows_any(const MatmulArgs &a, const TcParams &tp, const TensorTerms &t,
        const ColTerms &c, const uint32_t (&r)[R], int64_t m0, int64_t n) {
    if constexpr (DSTT >= 0) {
        // whole pieces (all but the last rows of a ragged M) take the straight path
        if (m0 + R <= a.M) epilogue_rows<INT, CHAIN, DSTT, R, true>(a, tp, t, c, r, m0, n);
        else epilogue_rows<INT, CHAIN, DSTT, R, false>(a, tp, t, c, r, m0, n);
        return;
    }
    switch (a.dst_dt) {
        case DT_BF16: epilogue_rows<INT, CHAIN, DT_BF16, R>(a, tp, t, c, r, m0, n); break;
        case DT_F32: epilogue_rows<INT, CHAIN, DT_F32, R>(a, tp, t, c, r, m0, n); break;
        case DT_S8: epilogue_rows<INT, CHAIN, DT_S8, R>(a, tp, t, c, r, m0, n); break;
        case DT_S32: epilogue_rows<INT, CHAIN, DT_S32, R>(a, tp, t, c, r, m0, n); break;
        case DT_F16: epilogue_rows<INT, CHAIN, DT_F16, R>(a, tp, t, c, r, m0, n); break;
        default: epilogue_rows<INT, CHAIN, DT_U8, R>(a, tp, t, c, r, m0, n); break;
    }
}

typedef CUresult (*encode_tiled_fn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
        const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
        CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

encode_tiled_fn get_encode() {
    static encode_tiled_fn fn = nullptr;
    if (!fn) {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess
                && q == cudaDriverEntryPointSuccess)
            fn = (encode_tiled_fn)p;
    }
    return fn;
}

// 2D map over a byte matrix [rows, cols] with row pitch `pitch` bytes; box =
// [box_rows, 128 bytes], 128-byte swizzle, out-of-bounds reads give zeros.
bool make_map_2d(CUtensorMap *map, const void *base, uint64_t cols, uint64_t rows, uint64_t pitch, uint32_t box_rows) {
    encode_tiled_fn enc = get_encode();
    if (!enc) return false;
    cuuint64_t dims[2] = {cols, rows};
    cuuint64_t strides[1] = {pitch};
    cuuint32_t box[2] = {128, box_rows};
    cuuint32_t estr[2] = {1, 1};
    return enc(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void *>(base), dims, strides, box, estr,
                   CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                   CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE)
            == CUDA_SUCCESS;
}

} // namespace

} // namespace qmm
