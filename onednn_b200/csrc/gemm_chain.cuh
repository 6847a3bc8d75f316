// Defines launch_gemm_chain_* of one dst data type.
#pragma once
#include "gemm_tc.cuh"

#define QMM_GEMM_CHAIN(NAME, DSTT) \
    int launch_gemm_chain_##NAME(QMM_GEMM_CHAIN_ARGS) { \
        if (sp) return int_path ? launch_split_cfg<1, true, DSTT>(mw, ms, a, tp, *sp, st) : launch_split_cfg<0, true, DSTT>(mw, ms, a, tp, *sp, st); \
        if (int_path) \
            return bt == 256 ? launch_cfg<1, 256, 4, true, DSTT>(mw, ms, a, tp, sm_count, st) : launch_cfg<1, 128, 6, true, DSTT>(mw, ms, a, tp, sm_count, st); \
        return bt == 256 ? launch_cfg<0, 256, 4, true, DSTT>(mw, ms, a, tp, sm_count, st) : launch_cfg<0, 128, 6, true, DSTT>(mw, ms, a, tp, sm_count, st); \
    }
