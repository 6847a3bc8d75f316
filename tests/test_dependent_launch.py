"""Kernels that start before their predecessor on the stream has ended (programmatic dependent launch).

They wait for that end (griddepcontrol.wait) before they read anything, and what they read then may be what the
predecessor wrote: tensors, scales, zero-points, offsets.  A load that says its memory is constant while the kernel runs
(__ldg, ld.global.nc, a __restrict__ pointer) may be moved above the wait by the compiler or served from a path that is
not coherent, so no such load may stand in these kernels or in the functions they use.  Whether a given compiler moves
one cannot be seen from results, so the CPU test reads the sources; the GPU tests chain calls in which every kind of
input is written by the call before."""
import os
import re

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "onednn_b200", "csrc")
NON_COHERENT = re.compile(r"__ldg|\.global\.nc|__restrict__|__ldcs|__ldlu")


def _source(name):
    text = open(os.path.join(CSRC, name)).read()
    text = re.sub(r"/\*.*?\*/", "", text, flags=re.S)
    text = re.sub(r"//[^\n]*", "", text)
    return re.sub(r"__launch_bounds__\((?:[^()]|\([^()]*\))*\)", "", text)


def _functions(text):
    """{name: body} of every function of a source (the definitions' braces matched), overloads joined."""
    out = {}
    for m in re.finditer(r"(\w+)\s*\((?:[^;{}()]|\([^;{}()]*\))*\)\s*(?:const\s*)?\{", text):
        at, depth = m.end(), 1
        while depth:
            depth += {"{": 1, "}": -1}.get(text[at], 0)
            at += 1
        if m.group(1) not in ("if", "for", "while", "switch"):
            out[m.group(1)] = out.get(m.group(1), "") + text[m.end():at]
    return out


def _reachable(file):
    """{kernel: text} of the dependent kernels of a file: their bodies and those of every function reached from them."""
    names, todo = set(), [file]
    while todo:
        f = todo.pop()
        if f in names or not os.path.exists(os.path.join(CSRC, f)):
            continue
        names.add(f)
        todo += re.findall(r'#include "([^"]+)"', open(os.path.join(CSRC, f)).read())
    functions = {}
    for f in names:
        for n, b in _functions(_source(f)).items():
            functions[n] = functions.get(n, "") + b
    kernels = {n: b for n, b in _functions(_source(file)).items()
               if n.endswith("_kernel") and "grid_dependency_wait()" in b}
    out = {}
    for k in kernels:
        seen, queue = {k}, [k]
        while queue:
            for n in set(re.findall(r"\b(\w+)\s*(?:<[^<>;]*>)?\s*\(", functions[queue.pop()])):
                if n in functions and n not in seen:
                    seen.add(n)
                    queue.append(n)
        out[k] = "".join(functions[n] for n in seen)
    return out


@pytest.mark.parametrize("file", ["reorder.cu", "gemm_split.cuh", "gemm_tc.cuh", "grouped_tc.cu", "woq_decode.cu", "woq8_decode.cu", "woq_rows.cu"])
def test_dependent_kernels_read_with_coherent_loads(file):
    kernels = _reachable(file)
    assert kernels, "no kernel with a wait in " + file
    for name, text in kernels.items():
        assert not NON_COHERENT.findall(text), "%s: %s" % (name, sorted(set(NON_COHERENT.findall(text))))


@pytest.mark.parametrize("file", ["gemm_split.cuh", "woq_decode.cu", "woq8_decode.cu"])
def test_a_cta_whose_peers_are_late_outlasts_them(file):
    """The CTAs of a cluster send their sums into each other's shared memory.  One whose bounded wait for them ran out may
    not end while a slower one can still send there: that store would go to memory that is gone.  A wait that runs out
    cannot be staged on a GPU without breaking the kernel, so the test reads the sources: the wait's result is kept, and
    the whole CTA is held on it."""
    (name, body), = [(n, b) for n, b in _functions(_source(file)).items() if n.endswith("_kernel")]
    assert re.search(r"st_async_v4\(|send_v4\(", body)
    wait = re.search(r"\blate = !ptx::mbar_wait\((\w+), 0\);", body)
    assert wait, name + " drops the result of its wait for the other CTAs' sums"
    tail = body[wait.end():]
    if "some_late" in tail:  # at the kernel's end, where a barrier of the CTA stands anyway; nothing returns before it
        assert "some_late = __syncthreads_or(late);" in tail
        assert re.search(r"if \(some_late && splits > 1\) ptx::outlast_cluster\(%s\);\s*\}\s*$" % wait.group(1), tail)
        assert "return" not in re.sub(r"\[[^\]]*\]\s*\([^()]*\)\s*\{[^{}]*\}", "", tail)  # (lambdas aside)
    else:  # right behind the wait, before anything is stored
        assert re.match(r"\s*if \(late\) atomicExch\(a\.status, 5\);\s*if \(__syncthreads_or\(late\)\) \{"
                        r"\s*if \(splits > 1\) ptx::outlast_cluster\(%s\);\s*return;" % wait.group(1), tail)


class _Device:
    """Device buffers (torch tensors) behind memory objects of this library, and a stream of its own for the calls."""

    def __init__(self, eng):
        import torch
        self.torch, self.eng, self.keep = torch, eng, []

    def put(self, a):
        t = self.torch.from_numpy(np.ascontiguousarray(a).view(np.uint8).reshape(-1).copy()).to("cuda:0")
        self.keep.append(t)
        return t

    def empty(self, nbytes):
        t = self.torch.zeros(nbytes, dtype=self.torch.uint8, device="cuda:0")
        self.keep.append(t)
        return t

    def mem(self, dims, dt, t):
        from onednn_b200 import api
        return api.memory(api.memory.desc(dims, dt, api.tag.a if len(dims) == 1 else api.tag.ab), self.eng, t.data_ptr())


def _in_a_row(dev, strm, calls, outputs, repeats=8):
    """Runs the calls one at a time, then all of them without a wait between, the outputs cleared each time: same bits."""
    dev.torch.cuda.synchronize()
    for prim, args in calls:
        prim.execute(strm, args)
        strm.wait()
    want = [t.cpu().numpy().copy() for t in outputs]
    for _ in range(repeats):
        for t in outputs:
            t.zero_()
        dev.torch.cuda.synchronize()
        for prim, args in calls:
            prim.execute(strm, args)
        strm.wait()
        for t, w in zip(outputs, want):
            assert np.array_equal(t.cpu().numpy(), w)
    return want


def _reorder(eng, dims, src_dt, dst_dt, **scales):
    from onednn_b200 import api, workloads as W
    attr = api.primitive_attr()
    for arg, mask in scales.items():
        attr.set_scales(api.ARG_DST if arg == "dst" else api.ARG_SRC, mask, (), W.F32)
    md = lambda dt: api.memory.desc(dims, dt, api.tag.ab)
    return api.reorder(api.reorder.primitive_desc(eng, md(src_dt), eng, md(dst_dt), attr))


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(8, 128), (512, 1024), (300, 4100)])
def test_reorders_of_a_matrix_and_scales_that_the_calls_before_wrote(gpu, shape):
    """bf16 -> f32 matrix, f32 scales brought over from another place, then the quantization of the one by the others, to s8
    and, from the 16-bit matrix that a third call wrote, to u8: each call's inputs are the outputs of those before."""
    from onednn_b200 import api, workloads as W
    eng, strm = gpu
    M, N = shape
    r = np.random.Generator(np.random.PCG64(31))
    d = _Device(eng)
    x16 = W.f32_to_bf16(r.standard_normal((M, N), dtype=np.float32))
    src, sc0 = d.put(x16), d.put(r.uniform(0.01, 0.05, (1, N)).astype(np.float32))
    x32, h16, sc, q8, qu = d.empty(4 * M * N), d.empty(2 * M * N), d.empty(4 * N), d.empty(M * N), d.empty(M * N)
    quant = api.ARG_ATTR_SCALES | api.ARG_DST
    calls = [
        (_reorder(eng, (M, N), W.BF16, W.F32), {api.ARG_FROM: d.mem((M, N), W.BF16, src), api.ARG_TO: d.mem((M, N), W.F32, x32)}),
        (_reorder(eng, (1, N), W.F32, W.F32), {api.ARG_FROM: d.mem((1, N), W.F32, sc0), api.ARG_TO: d.mem((1, N), W.F32, sc)}),
        (_reorder(eng, (M, N), W.F32, W.S8, dst=2), {api.ARG_FROM: d.mem((M, N), W.F32, x32), api.ARG_TO: d.mem((M, N), W.S8, q8),
                                                     quant: d.mem((1, N), W.F32, sc)}),
        (_reorder(eng, (M, N), W.F32, W.F16), {api.ARG_FROM: d.mem((M, N), W.F32, x32), api.ARG_TO: d.mem((M, N), W.F16, h16)}),
        (_reorder(eng, (M, N), W.F16, W.U8, dst=2), {api.ARG_FROM: d.mem((M, N), W.F16, h16), api.ARG_TO: d.mem((M, N), W.U8, qu),
                                                     quant: d.mem((1, N), W.F32, sc)}),
    ]
    want = _in_a_row(d, strm, calls, [x32, sc, q8, h16, qu])
    x = W.bf16_to_f32(x16)
    scale = sc0.cpu().numpy().view(np.float32)
    assert np.array_equal(want[2].view(np.int8).reshape(M, N), np.clip(np.rint(x / scale), -128, 127).astype(np.int8))
    assert np.array_equal(want[4].reshape(M, N), np.clip(np.rint(x.astype(np.float16).astype(np.float32) / scale), 0, 255).astype(np.uint8))


@pytest.mark.gpu
@pytest.mark.parametrize("shape", [(33, 256, 512), (40, 512, 1024), (1900, 256, 1536)])
def test_int8_layer_after_the_calls_that_quantize_its_src_and_write_its_parameters(gpu, shape):
    """The src, its per-row scales, the weight scales and the residual of an int8 matmul with a post-op chain are each the
    output of a call right before it (reorders), and its result is the input of a reorder: the split and the persistent
    kernel, rows that fill the pieces of eight and rows that do not."""
    from onednn_b200 import api, workloads as W
    eng, strm = gpu
    M, K, N = shape
    r = np.random.Generator(np.random.PCG64(32))
    d = _Device(eng)
    f32 = lambda lo, hi, dims: r.uniform(lo, hi, dims).astype(np.float32)
    x, xs = f32(-1, 1, (M, K)), f32(0.01, 0.02, (1, K))
    given = [(x, (M, K)), (f32(0.001, 0.01, (M, 1)), (M, 1)), (f32(0.001, 0.01, (1, N)), (1, N)), (f32(-3, 3, (M, N)), (M, N))]
    src8, row_scale, col_scale, resid = d.empty(M * K), d.empty(4 * M), d.empty(4 * N), d.empty(4 * M * N)
    dst8, back = d.empty(M * N), d.empty(4 * M * N)
    one = d.put(np.full(1, 0.06, np.float32))
    wei = d.put(r.integers(-127, 128, (K, N), dtype=np.int8))
    quant = api.ARG_ATTR_SCALES
    calls = [(_reorder(eng, (M, K), W.F32, W.S8, dst=2), {api.ARG_FROM: d.mem((M, K), W.F32, d.put(x)), api.ARG_TO: d.mem((M, K), W.S8, src8),
                                                          quant | api.ARG_DST: d.mem((1, K), W.F32, d.put(xs))})]
    for (a, dims), t in zip(given[1:], (row_scale, col_scale, resid)):
        calls.append((_reorder(eng, dims, W.F32, W.F32), {api.ARG_FROM: d.mem(dims, W.F32, d.put(a)), api.ARG_TO: d.mem(dims, W.F32, t)}))
    attr = api.primitive_attr()
    attr.set_scales(api.ARG_SRC, 1, (), W.F32)
    attr.set_scales(api.ARG_WEIGHTS, 2, (), W.F32)
    attr.set_scales(api.ARG_DST, 0, (), W.F32)
    md = lambda dims, dt: api.memory.desc(dims, dt, api.tag.ab)
    po = api.post_ops()
    po.append_eltwise(W.ELTWISE["relu"], 0.0, 0.0)
    po.append_binary(W.BINARY["add"], md((M, N), W.F32))
    attr.set_post_ops(po)
    pd = api.matmul.primitive_desc(eng, md((M, K), W.S8), md((K, N), W.S8), md((M, N), W.S8), None, attr)
    assert pd.impl_info_str() == "cuda:tcgen05:int8"
    calls.append((api.matmul(pd), {
        api.ARG_SRC: d.mem((M, K), W.S8, src8), api.ARG_WEIGHTS: d.mem((K, N), W.S8, wei), api.ARG_DST: d.mem((M, N), W.S8, dst8),
        quant | api.ARG_SRC: d.mem((M, 1), W.F32, row_scale), quant | api.ARG_WEIGHTS: d.mem((1, N), W.F32, col_scale),
        quant | api.ARG_DST: d.mem((1,), W.F32, one),
        api.ARG_ATTR_MULTIPLE_POST_OP(1) | api.ARG_SRC_1: d.mem((M, N), W.F32, resid)}))
    calls.append((_reorder(eng, (M, N), W.S8, W.F32), {api.ARG_FROM: d.mem((M, N), W.S8, dst8), api.ARG_TO: d.mem((M, N), W.F32, back)}))
    want = _in_a_row(d, strm, calls, [src8, row_scale, col_scale, resid, dst8, back])
    s8 = np.clip(np.rint(x / xs), -128, 127).astype(np.int8)
    assert np.array_equal(want[0].view(np.int8).reshape(M, K), s8)
    assert np.unique(want[4]).size > 20  # (not a constant result)


@pytest.mark.gpu
@pytest.mark.parametrize("M", [5, 40, 2000])
def test_int4_layer_after_the_calls_that_write_its_src_and_parameters(gpu, M):
    """The src, the group scales and the group zero-points of an int4 matmul are each the output of a call right before it
    (4-bit zero-points, which no reorder copies, as eight 8-bit halves): the decode kernel, the same in blocks of rows, and
    the kernel for many rows."""
    from onednn_b200 import api, workloads as W
    eng, strm = gpu
    K, N, G = 512, 1056, 64
    r = np.random.Generator(np.random.PCG64(33))
    d = _Device(eng)
    f32 = lambda lo, hi, dims: r.uniform(lo, hi, dims).astype(np.float32)
    zp_bytes = r.integers(0, 256, (K // G, N // 2), dtype=np.uint8)
    wei = d.put(r.integers(0, 256, (K, N // 2), dtype=np.uint8))
    src, scale, zp, dst, back = d.empty(2 * M * K), d.empty(2 * (K // G) * N), d.empty(zp_bytes.size), d.empty(4 * M * N), d.empty(2 * M * N)
    copy = lambda dims, sdt, ddt, a, t: (_reorder(eng, dims, sdt, ddt), {api.ARG_FROM: d.mem(dims, sdt, a), api.ARG_TO: d.mem(dims, ddt, t)})
    calls = [copy((M, K), W.F32, W.BF16, d.put(f32(-1, 1, (M, K))), src),
             copy((K // G, N), W.F32, W.BF16, d.put(f32(0.005, 0.02, (K // G, N))), scale),
             copy(zp_bytes.shape, W.U8, W.U8, d.put(zp_bytes), zp)]
    attr = api.primitive_attr()
    attr.set_fpmath_mode(api.fpmath_mode.bf16, True)
    attr.set_scales(api.ARG_WEIGHTS, 3, (G, 1), W.BF16)
    attr.set_zero_points(api.ARG_WEIGHTS, 3, (G, 1), W.U4)
    md = lambda dims, dt: api.memory.desc(dims, dt, api.tag.ab)
    pd = api.matmul.primitive_desc(eng, md((M, K), W.BF16), md((K, N), W.U4), md((M, N), W.F32), None, attr)
    assert pd.impl_info_str() == ("cuda:tcgen05:woq4" if M <= 32 else "cuda:tcgen05:woq4_rows")
    calls.append((api.matmul(pd), {
        api.ARG_SRC: d.mem((M, K), W.BF16, src), api.ARG_WEIGHTS: d.mem((K, N), W.U4, wei), api.ARG_DST: d.mem((M, N), W.F32, dst),
        api.ARG_ATTR_SCALES | api.ARG_WEIGHTS: d.mem((K // G, N), W.BF16, scale),
        api.ARG_ATTR_ZERO_POINTS | api.ARG_WEIGHTS: d.mem((K // G, N), W.U4, zp)}))
    calls.append(copy((M, N), W.F32, W.BF16, dst, back))
    want = _in_a_row(d, strm, calls, [src, scale, zp, dst, back])
    # against f64
    nib = lambda b: np.stack([b & 15, b >> 4], -1).reshape(b.shape[0], -1).astype(np.float64)
    w = nib(wei.cpu().numpy().reshape(K, N // 2)) - np.repeat(nib(zp_bytes), G, 0)
    w *= np.repeat(W.bf16_to_f32(want[1].view(np.uint16)).reshape(K // G, N), G, 0)
    x = W.bf16_to_f32(want[0].view(np.uint16)).reshape(M, K).astype(np.float64)
    got = want[3].view(np.float32).reshape(M, N)
    assert np.all(np.abs(got - x @ w) <= K * 2.0 ** -24 * (np.abs(x) @ np.abs(w)))  # f32 sums of K exact products, any order


@pytest.mark.gpu
@pytest.mark.parametrize("M,experts", [(24, 8), (50, 200), (700, 8)])
def test_grouped_and_dense_s8_layers_after_the_calls_that_write_their_inputs(gpu, M, experts):
    """Weight scales, src and the row offsets of a grouped s8-weight matmul are each the output of a call right before it,
    and its result is the src of a dense s8-weight matmul: few rows and many."""
    from onednn_b200 import api, workloads as W
    eng, strm = gpu
    K, N = 256, 320
    r = np.random.Generator(np.random.PCG64(34))
    d = _Device(eng)
    f32 = lambda lo, hi, dims: r.uniform(lo, hi, dims).astype(np.float32)
    ends = np.cumsum(r.multinomial(M, np.full(experts, 1.0 / experts))).astype(np.int32)
    wei = r.integers(-127, 128, (experts, K, N), dtype=np.int8)
    wei2 = r.integers(-127, 128, (N, K), dtype=np.int8)
    src, offs, scale, scale2 = d.empty(2 * M * K), d.empty(4 * experts), d.empty(4 * experts * N), d.empty(4 * K)
    mid, out = d.empty(2 * M * N), d.empty(4 * M * K)
    copy = lambda dims, sdt, ddt, a, t: (_reorder(eng, dims, sdt, ddt), {api.ARG_FROM: d.mem(dims, sdt, a), api.ARG_TO: d.mem(dims, ddt, t)})
    calls = [copy((M, K), W.F32, W.BF16, d.put(f32(-1, 1, (M, K))), src),
             copy((experts, N), W.F32, W.F32, d.put(f32(0.001, 0.01, (experts, N))), scale),
             copy((1, K), W.F32, W.F32, d.put(f32(0.001, 0.01, (1, K))), scale2),
             copy((1, experts), W.S32, W.S32, d.put(ends), offs)]
    attr = api.primitive_attr()
    attr.set_fpmath_mode(api.fpmath_mode.bf16, True)
    attr.set_scales(api.ARG_WEIGHTS, 0b101, (), W.F32)
    grouped = lambda dims: api.memory.desc.grouped(dims, W.BF16, 0, experts)
    abc = lambda dims, dt: api.memory.desc(dims, dt, api.tag.abc)
    put = lambda md, t: api.memory(md, eng, t.data_ptr())
    pd = api.matmul.primitive_desc(eng, grouped((M, K)), abc((experts, K, N), W.S8), grouped((M, N)), None, attr)
    assert pd.impl_info_str() == "cuda:tcgen05:grouped"
    calls.append((api.matmul(pd), {
        api.ARG_SRC: api.memory(grouped((M, K)), eng, handles=[src.data_ptr(), offs.data_ptr()]),
        api.ARG_DST: api.memory(grouped((M, N)), eng, handles=[mid.data_ptr(), offs.data_ptr()]),
        api.ARG_WEIGHTS: put(abc((experts, K, N), W.S8), d.put(wei)),
        api.ARG_ATTR_SCALES | api.ARG_WEIGHTS: put(abc((experts, 1, N), W.F32), scale)}))
    attr2 = api.primitive_attr()
    attr2.set_fpmath_mode(api.fpmath_mode.bf16, True)
    attr2.set_scales(api.ARG_WEIGHTS, 2, (), W.F32)
    md = lambda dims, dt: api.memory.desc(dims, dt, api.tag.ab)
    pd2 = api.matmul.primitive_desc(eng, md((M, N), W.BF16), md((N, K), W.S8), md((M, K), W.F32), None, attr2)
    assert pd2.impl_info_str() == "cuda:tcgen05:woq8"
    calls.append((api.matmul(pd2), {
        api.ARG_SRC: d.mem((M, N), W.BF16, mid), api.ARG_WEIGHTS: d.mem((N, K), W.S8, d.put(wei2)), api.ARG_DST: d.mem((M, K), W.F32, out),
        api.ARG_ATTR_SCALES | api.ARG_WEIGHTS: d.mem((1, K), W.F32, scale2)}))
    # (the offsets are cleared by hand to zeros between the runs: no rows, a valid call)
    want = _in_a_row(d, strm, calls, [src, scale, scale2, offs, mid, out])
    assert np.array_equal(want[3].view(np.int32), ends)
    x = W.bf16_to_f32(want[0].view(np.uint16)).reshape(M, K).astype(np.float64)
    sc = want[1].view(np.float32).reshape(experts, N)
    got = W.bf16_to_f32(want[4].view(np.uint16)).reshape(M, N)
    for e, (b, t) in enumerate(zip(np.concatenate([[0], ends[:-1]]), ends)):
        exact = x[b:t] @ wei[e].astype(np.float64) * sc[e]
        terms = np.abs(x[b:t]) @ np.abs(wei[e].astype(np.float64)) * sc[e]
        assert np.all(np.abs(got[b:t] - exact) <= 2.0 ** -8 * np.abs(exact) + K * 2.0 ** -24 * terms)  # bf16 rounding, f32 sums
