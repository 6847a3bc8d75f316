"""Performance cases of the quantized matmul library.

Each case is one call that a program linked against the library makes over and
over: one execution of a prepared ``dnnl::matmul`` (or ``dnnl::reorder``)
primitive on the caller's CUDA stream, with the caller's device buffers behind
the memory objects.  The five matmul families and their sizes are the ones
``bench.py`` and the tests use; the ranges around them are those of the layers of
a language model served with 8-bit or 4-bit weights: any number of rows M, K and
N from a narrow layer to a wide one.

``kind`` of a case
  int8    u8 / s8 activations x s8 weights, with a src zero-point (u8) or per-row
          scales (s8) and per-column weight scales
  chain   s8 x s8 with bias, gelu_tanh, a residual and requantization to s8
  fp8     8-bit float activations and weights, per-tensor scales, bf16 bias
  woq4    bf16 / f16 activations x 4-bit weights, scales and zero-points per K-group
  woq8    bf16 activations x s8 weights, per-column scales
  moe     the grouped form of woq8: rows of several experts in one call
  reorder f32 / bf16 matrix quantized to s8 with per-column scales
"""
import math

import torch

from onednn_b200 import api
from onednn_b200 import workloads as W

_TORCH_DT = {W.S32: torch.int32, W.F32: torch.float32, W.BF16: torch.bfloat16, W.F16: torch.float16,
             W.S8: torch.int8, W.U8: torch.uint8}
_DT = {name: code for code, name in W.DT_NAME.items()}


def listed():
    return [
        # a small int8 layer with a u8 activation zero-point and exact s32 sums: launch latency
        {"name": "int8_small_zp", "kind": "int8", "M": 256, "K": 1024, "N": 1024, "src": "u8", "dst": "s32",
         "runtime_m": False},
        # token generation with int8 weights: a ragged batch of 17 rows; the program made one
        # primitive with M left open for every batch size
        {"name": "int8_decode_m17", "kind": "int8", "M": 17, "K": 4096, "N": 11008, "src": "s8", "dst": "bf16",
         "runtime_m": True},
        # prompt processing: the up-projection of an int8 MLP with its whole post-op chain
        {"name": "int8_chain", "kind": "chain", "M": 2048, "K": 4096, "N": 11008},
        # prompt processing in fp8, a full batch: the largest dense call
        {"name": "fp8_prefill", "kind": "fp8", "M": 4096, "K": 4096, "N": 14336, "src": "f8_e4m3"},
        # a short ragged prompt in fp8
        {"name": "fp8_chunk_m509", "kind": "fp8", "M": 509, "K": 4096, "N": 4096, "src": "f8_e4m3"},
        # token generation with 4-bit weights, one sequence
        {"name": "int4_decode_m1", "kind": "woq4", "M": 1, "K": 8192, "N": 28672, "src": "bf16", "wei": "s4",
         "group": 128, "zp": True},
        # token generation, thirteen sequences, a narrower f16 model, symmetric weights
        {"name": "int4_decode_m13", "kind": "woq4", "M": 13, "K": 4096, "N": 11008, "src": "f16", "wei": "u4",
         "group": 64, "zp": False},
        # the prompt of the same kind of model: 4-bit weights against a few hundred rows
        {"name": "int4_prefill_m300", "kind": "woq4", "M": 300, "K": 4096, "N": 4096, "src": "bf16", "wei": "s4",
         "group": 128, "zp": True},
        # mixture of experts, a full batch (row counts per expert follow Zipf's law)
        {"name": "moe_prefill", "kind": "moe", "M": 8192, "K": 4096, "N": 14336, "experts": 64},
        # mixture of experts, token generation on the 8 experts one GPU holds
        {"name": "moe_decode", "kind": "moe", "M": 37, "K": 4096, "N": 14336, "experts": 8},
        # dense s8 weight decompression, a medium prompt
        {"name": "woq8_m777", "kind": "woq8", "M": 777, "K": 4096, "N": 4096},
        # a weight matrix quantized when a model is loaded or updated
        {"name": "reorder_quantize", "kind": "reorder", "M": 4096, "N": 14336, "src": "f32"},
    ]


def _log_int(rng, lo, hi, step=1):
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(lo, min(hi, int(round(v / step)) * step))


def draw(rng):
    """One more case of the listed kinds: M is any number, K and N multiples of 16 (of 32 for 4-bit
    weights, whose K is also a multiple of the scale group), from 1/8 to twice a common layer."""
    kind = rng.choice(["int8", "chain", "fp8", "woq4", "woq4", "woq8", "moe", "reorder"])
    if kind == "reorder":
        return {"kind": kind, "M": _log_int(rng, 512, 8192), "N": _log_int(rng, 512, 14336, 8),
                "src": rng.choice(["f32", "bf16"])}
    if kind == "moe":
        return {"kind": kind, "M": _log_int(rng, 8, 8192), "K": _log_int(rng, 1024, 4096, 64),
                "N": _log_int(rng, 1024, 14336, 64), "experts": rng.choice([8, 16, 32, 64])}
    if kind == "woq4":
        group = rng.choice([32, 64, 128])
        c = {"kind": kind, "M": _log_int(rng, 1, 512), "K": _log_int(rng, 1024, 8192, 128),
             "N": _log_int(rng, 1024, 28672, 32), "src": rng.choice(["bf16", "f16"]), "wei": rng.choice(["s4", "u4"]),
             "group": group, "zp": rng.random() < 0.5}
        while c["M"] * c["K"] * c["N"] > 12e9:
            c["M"] = max(1, c["M"] // 2)
        return c
    c = {"kind": kind, "M": _log_int(rng, 1, 4096), "K": _log_int(rng, 512, 8192, 16), "N": _log_int(rng, 512, 16384, 16)}
    if kind == "int8":
        c.update(src=rng.choice(["u8", "s8"]), dst=rng.choice(["s32", "f32", "bf16"]), runtime_m=rng.random() < 0.25)
    if kind == "fp8":
        c.update(src=rng.choice(["f8_e4m3", "f8_e5m2"]))
    while c["M"] * c["K"] * c["N"] > 2.4e11:
        c["M"] = max(1, c["M"] // 2)
    return c


class _Call:
    """The handles a program keeps for one primitive: engine, stream, primitive and the memory objects
    that wrap its device buffers."""

    def __init__(self):
        self.eng = api.engine(api.engine.kind.gpu, torch.cuda.current_device())
        self.strm = api.stream(self.eng, torch.cuda.current_stream().cuda_stream)
        self.keep, self.args = [], {}

    def tensor(self, arg, t, dims, dt, fmt=api.tag.ab):
        md = api.memory.desc(dims, dt, fmt)
        self.args[arg] = api.memory(md, self.eng, t.data_ptr())
        self.keep.append(t)
        return md

    def finish(self, prim, dst):
        self.prim, self.dst = prim, dst
        return self


def _randint(g, lo, hi, shape, dtype):
    return torch.randint(lo, hi, shape, generator=g, device="cuda", dtype=dtype)


def _uniform(g, lo, hi, shape):
    return torch.rand(shape, generator=g, device="cuda") * (hi - lo) + lo


def _randn(g, shape):
    return torch.randn(shape, generator=g, device="cuda")


def _fp8(g, shape, dt):
    # N(0, 1) spread over the e4m3 range
    x = _randn(g, shape) * (448.0 / 6.0)
    return x.clamp_(-448.0, 448.0).to(torch.float8_e4m3fn if dt == W.F8_E4M3 else torch.float8_e5m2)


def prepare(case, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    call = _Call()
    if case["kind"] == "reorder":
        return _prepare_reorder(case, g, call)
    if case["kind"] == "moe":
        return _prepare_moe(case, seed, g, call)
    M, K, N, kind = case["M"], case["K"], case["N"], case["kind"]
    attr = api.primitive_attr()
    scales, zps = [], []  # (arg, buffer, mask, groups, data type)
    bias_md = None
    post_ops = None
    if kind in ("int8", "chain"):
        src_dt = _DT[case.get("src", "s8")]
        dst_dt = W.S8 if kind == "chain" else _DT[case["dst"]]
        wei, wei_dt = _randint(g, -127, 128, (K, N), torch.int8), W.S8
        if src_dt == W.U8:
            src = _randint(g, 0, 256, (M, K), torch.uint8)
            zps.append((api.ARG_SRC, torch.full((1,), 128, dtype=torch.int32, device="cuda"), 0, (), W.S32))
        else:
            src = _randint(g, -64, 64, (M, K), torch.int8)
            if dst_dt != W.S32:
                scales.append((api.ARG_SRC, _uniform(g, 0.001, 0.01, (M, 1)), 1, (), W.F32))
        if dst_dt != W.S32:
            scales.append((api.ARG_WEIGHTS, _uniform(g, 0.001, 0.01, (1, N)), 2, (), W.F32))
        if kind == "chain":
            scales.append((api.ARG_DST, torch.full((1,), 0.06 * math.sqrt(K / 4096.0), device="cuda"), 0, (), W.F32))
            bias_md = call.tensor(api.ARG_BIAS, _randn(g, (1, N)), (1, N), W.F32)
            resid = _randn(g, (M, N))
            po_md = call.tensor(api.ARG_ATTR_MULTIPLE_POST_OP(1) | api.ARG_SRC_1, resid, (M, N), W.F32)
            post_ops = api.post_ops()
            post_ops.append_eltwise(W.ELTWISE["gelu_tanh"], 0.0, 0.0)
            post_ops.append_binary(W.BINARY["add"], po_md)
    elif kind == "fp8":
        src_dt, wei_dt, dst_dt = _DT[case["src"]], W.F8_E4M3, W.BF16
        src, wei = _fp8(g, (M, K), src_dt), _fp8(g, (K, N), wei_dt)
        for arg in (api.ARG_SRC, api.ARG_WEIGHTS):
            scales.append((arg, torch.full((1,), 6.0 / 448.0, device="cuda"), 0, (), W.F32))
        bias_md = call.tensor(api.ARG_BIAS, _randn(g, (1, N)).bfloat16(), (1, N), W.BF16)
    elif kind == "woq4":
        src_dt, wei_dt = _DT[case["src"]], _DT[case["wei"]]
        dst_dt = src_dt
        src = _randn(g, (M, K)).to(_TORCH_DT[src_dt])
        wei = _randint(g, 0, 256, (K, N // 2), torch.uint8)  # two uniform nibbles per byte
        groups = (case["group"], 1)
        G = K // case["group"]
        scales.append((api.ARG_WEIGHTS, _uniform(g, 0.005, 0.02, (G, N)).to(_TORCH_DT[src_dt]), 3, groups, src_dt))
        if case["zp"]:
            zps.append((api.ARG_WEIGHTS, _randint(g, 0, 256, (G, N // 2), torch.uint8), 3, groups, W.U4))
        attr.set_fpmath_mode(api.fpmath_mode.bf16 if src_dt == W.BF16 else api.fpmath_mode.f16, True)
    else:  # woq8
        src_dt, wei_dt, dst_dt = W.BF16, W.S8, W.BF16
        src, wei = _randn(g, (M, K)).bfloat16(), _randint(g, -127, 128, (K, N), torch.int8)
        scales.append((api.ARG_WEIGHTS, _uniform(g, 0.001, 0.01, (1, N)), 2, (), W.F32))
        attr.set_fpmath_mode(api.fpmath_mode.bf16, True)
    dst = torch.empty((M, N), dtype=_TORCH_DT[dst_dt], device="cuda")

    for arg, _, mask, groups, dt in scales:
        attr.set_scales(arg, mask, groups, dt)
    for arg, _, mask, groups, dt in zps:
        attr.set_zero_points(arg, mask, groups, dt)
    if post_ops is not None:
        attr.set_post_ops(post_ops)
    src_md = call.tensor(api.ARG_SRC, src, (M, K), src_dt)
    wei_md = call.tensor(api.ARG_WEIGHTS, wei, (K, N), wei_dt)
    dst_md = call.tensor(api.ARG_DST, dst, (M, N), dst_dt)
    if case.get("runtime_m"):
        src_md = api.memory.desc((api.RUNTIME_DIM_VAL, K), src_dt, (K, 1))
        dst_md = api.memory.desc((api.RUNTIME_DIM_VAL, N), dst_dt, (N, 1))
    for base, entries in ((api.ARG_ATTR_SCALES, scales), (api.ARG_ATTR_ZERO_POINTS, zps)):
        for arg, t, mask, groups, dt in entries:
            dims = tuple(t.shape[:-1]) + (t.shape[-1] * (2 if dt == W.U4 else 1),)
            call.tensor(base | arg, t, dims, dt, api.tag.a if len(dims) == 1 else api.tag.ab)
    return call.finish(api.matmul(api.matmul.primitive_desc(call.eng, src_md, wei_md, dst_md, bias_md, attr)), dst)


def _prepare_moe(case, seed, g, call):
    M, K, N, E = case["M"], case["K"], case["N"], case["experts"]
    sizes = W.zipf_group_sizes(M, E, seed=seed)
    offsets = torch.from_numpy(sizes).cumsum(0).to(torch.int32).cuda()
    src = _randn(g, (M, K)).bfloat16()
    wei = torch.empty((E, K, N), dtype=torch.int8, device="cuda")
    for e in range(E):
        wei[e] = _randint(g, -127, 128, (K, N), torch.int8)
    wei_scale = _uniform(g, 0.001, 0.01, (E, 1, N))
    dst = torch.empty((M, N), dtype=torch.bfloat16, device="cuda")
    attr = api.primitive_attr()
    attr.set_fpmath_mode(api.fpmath_mode.bf16, True)
    attr.set_scales(api.ARG_WEIGHTS, 0b101, (), W.F32)
    src_md = api.memory.desc.grouped((M, K), W.BF16, 0, E)
    dst_md = api.memory.desc.grouped((M, N), W.BF16, 0, E)
    call.args[api.ARG_SRC] = api.memory(src_md, call.eng, handles=[src.data_ptr(), offsets.data_ptr()])
    call.args[api.ARG_DST] = api.memory(dst_md, call.eng, handles=[dst.data_ptr(), offsets.data_ptr()])
    call.keep += [src, dst, offsets]
    wei_md = call.tensor(api.ARG_WEIGHTS, wei, (E, K, N), W.S8, api.tag.abc)
    call.tensor(api.ARG_ATTR_SCALES | api.ARG_WEIGHTS, wei_scale, (E, 1, N), W.F32, api.tag.abc)
    call.finish(api.matmul(api.matmul.primitive_desc(call.eng, src_md, wei_md, dst_md, None, attr)), dst)
    run(call)  # servers of such models execute every expert layer once when the weights have been loaded
    return call


def _prepare_reorder(case, g, call):
    M, N, src_dt = case["M"], case["N"], _DT[case["src"]]
    src = (_randn(g, (M, N)) * 0.05).to(_TORCH_DT[src_dt])
    scale = (src.float().abs().amax(0, keepdim=True) / 127.0).contiguous()
    dst = torch.empty((M, N), dtype=torch.int8, device="cuda")
    attr = api.primitive_attr()
    attr.set_scales(api.ARG_DST, 2, (), W.F32)
    src_md = call.tensor(api.ARG_FROM, src, (M, N), src_dt)
    dst_md = call.tensor(api.ARG_TO, dst, (M, N), W.S8)
    call.tensor(api.ARG_ATTR_SCALES | api.ARG_DST, scale, (1, N), W.F32)
    return call.finish(api.reorder(api.reorder.primitive_desc(call.eng, src_md, call.eng, dst_md, attr)), dst)


def run(state):
    state.prim.execute(state.strm, state.args)
    return state.dst


def _rows_used(case):
    """Experts with at least one row, in expectation: only their weights have to be read."""
    p = [1.0 / r ** 1.1 for r in range(1, case["experts"] + 1)]
    t = sum(p)
    return sum(1.0 - (1.0 - x / t) ** case["M"] for x in p)


def work(case):
    M, N, kind = case["M"], case["N"], case["kind"]
    if kind == "reorder":
        return {"bytes": M * N * ((4 if case["src"] == "f32" else 2) + 1) + 4 * N, "flops": M * N}
    K = case["K"]
    flops = 2 * M * K * N
    if kind == "moe":
        e = _rows_used(case)
        return {"bytes": 2 * M * K + e * (K * N + 4 * N) + 2 * M * N + 4 * case["experts"], "flops": flops}
    if kind == "int8":
        b = M * K + K * N + M * N * {"s32": 4, "f32": 4, "bf16": 2}[case["dst"]]
        if case["dst"] != "s32":
            b += 4 * N + (4 * M if case["src"] == "s8" else 0)
    elif kind == "chain":
        b = M * K + K * N + 4 * M + 8 * N + M * N * (4 + 1)
    elif kind == "fp8":
        b = M * K + K * N + 2 * N + 2 * M * N
    elif kind == "woq4":
        b = 2 * M * K + K * N // 2 + K // case["group"] * N * 2 + 2 * M * N
        if case["zp"]:
            b += K // case["group"] * N // 2
    else:
        b = 2 * M * K + K * N + 4 * N + 2 * M * N
    return {"bytes": b, "flops": flops}


def tolerance(case):
    """Four times the largest difference seen between the library's results and the same products summed
    in 64 bits and rounded to the result's type (sums in another order move single roundings)."""
    kind = case["kind"]
    if kind == "reorder" or (kind == "int8" and case["dst"] == "s32"):
        return "exact"  # integer sums; one IEEE division and one rounding
    if kind == "chain":
        return {"rel": 0.0, "differ": 5e-5}  # values that lie on a rounding boundary of the requantization
    if kind == "int8" and case["dst"] == "f32":
        return {"rel": 4e-7, "max": 1e-6}
    if kind == "woq4" and case["src"] == "f16":
        return {"rel": 1e-4, "max": 4e-3}  # f16 results
    return {"rel": 5e-4, "max": 3.2e-2}  # bf16 results
