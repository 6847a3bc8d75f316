"""8-bit GEMM of few tiles (K split over the CTAs of a cluster, column sums from the GEMM itself) and calls in a row:
edges of row pieces, column tiles and K stages."""
import numpy as np
import pytest

from onednn_b200 import api
from onednn_b200 import workloads as W
from onednn_b200.runner import run_problem
from oracle import oracle as O
from test_parity_gpu import _ba, _wei_zp
from util import assert_parity, summation_slack

pytestmark = pytest.mark.gpu

# (M, K, N): one piece of 8 rows and its neighbours, two row tiles, one K stage and ragged ones, one column group of 16
SHAPES = [(1, 16, 16), (8, 128, 128), (9, 2064, 144), (17, 4096, 1040), (31, 1152, 272), (33, 656, 400), (64, 8192, 256),
          (65, 1296, 528), (127, 992, 1808), (200, 3216, 96)]


@pytest.mark.parametrize("shape", SHAPES)
def test_int8_src_zero_point_is_exact(gpu, shape):
    eng, strm = gpu
    p = W.int8_zp(*shape)
    got, impl = run_problem(p, eng, strm)
    assert impl == "cuda:tcgen05:int8"
    assert np.array_equal(got, O.run_port(p))


@pytest.mark.parametrize("shape", SHAPES[1::2])
def test_int8_both_zero_points_per_column_scales(gpu, shape):
    eng, strm = gpu
    p = W.int8_zp(*shape, per_n_scales=True)
    r = np.random.Generator(np.random.PCG64(5))
    p.quant["wei_zp"] = W.Quant(r.integers(-9, 10, (1, p.N)).astype(np.int8), W.S8, 2)
    got, impl = run_problem(p, eng, strm)
    assert impl == "cuda:tcgen05:int8"
    assert_parity(got, O.run_port(p), p.dst_dt, str(shape), None)


@pytest.mark.parametrize("shape", SHAPES)
def test_post_op_chain(gpu, shape):
    eng, strm = gpu
    p = W.int8_postops(*shape)
    got, impl = run_problem(p, eng, strm)
    assert impl == "cuda:tcgen05:int8"
    assert_parity(got, O.run_port(p), p.dst_dt, str(shape), None)


@pytest.mark.parametrize("shape", SHAPES)
def test_fp8(gpu, shape):
    eng, strm = gpu
    p = W.fp8_prefill(*shape)
    got, impl = run_problem(p, eng, strm)
    assert impl == "cuda:tcgen05:fp8"
    assert_parity(got, O.run_port(p), p.dst_dt, str(shape), summation_slack(p))
    got2, _ = run_problem(p, eng, strm)  # the shares are added in the same order every time
    assert np.array_equal(got, got2)


def _chain_to(p, dst_dt):
    """The chain's problem with another result type.  Floating-point results: relu instead of gelu, for the device's tanhf and the
    host's differ by units in the last place, which shows where the residual cancels it (4 ulp of bf16 in 3 of 2.9 million)."""
    p.dst_dt = dst_dt
    if dst_dt not in (W.S8, W.U8):
        p.post_ops[0] = W.PostOp(W.PO_ELTWISE, W.ELTWISE["relu"], 0.0, 0.0, 1.0)
    if dst_dt not in (W.S8, W.U8):
        p.quant.pop("dst_scale", None)
    return p


# problems of enough tiles for the persistent kernel: ragged ends of rows, columns and K; zero-points of one and of both
# sides with either layout of the weights (the column sums come from a kernel of their own there, the row sums in both)
PERSISTENT = {
    "chain_ragged": lambda: W.int8_postops(700, 400, 4112),
    "chain_short_k": lambda: W.int8_postops(2000, 144, 1040),
    "chain_f32": lambda: _chain_to(W.int8_postops(700, 400, 4112), W.F32),
    "chain_bf16": lambda: _chain_to(W.int8_postops(700, 400, 4112), W.BF16),
    "chain_u8": lambda: _chain_to(W.int8_postops(700, 400, 4112), W.U8),
    "src_zp": lambda: W.int8_zp(520, 528, 4112),
    "src_zp_ba": lambda: _ba(W.int8_zp(520, 528, 4112)),
    "both_zp": lambda: _wei_zp(W.int8_zp(520, 528, 4112, per_n_scales=True), True),
    "both_zp_ba": lambda: _wei_zp(_ba(W.int8_zp(520, 528, 4112)), False),
    "fp8": lambda: W.fp8_prefill(1030, 272, 4112),
}


@pytest.mark.parametrize("name", sorted(PERSISTENT))
def test_persistent_kernel_on_ragged_problems(gpu, name):
    eng, strm = gpu
    p = PERSISTENT[name]()
    got, impl = run_problem(p, eng, strm)
    assert impl == ("cuda:tcgen05:fp8" if name == "fp8" else "cuda:tcgen05:int8")
    assert api.last_kernel() == "gemm_tc"
    assert_parity(got, O.run_port(p), p.dst_dt, name, summation_slack(p) if name == "fp8" else None)


@pytest.mark.parametrize("make", [lambda: W.int8_zp(65, 1296, 528), lambda: W.fp8_prefill(127, 992, 1808), lambda: W.int8_postops(31, 1152, 272)],
                         ids=["int8_zp", "fp8", "chain"])
def test_few_tiles_take_the_split_kernel(gpu, make):
    eng, strm = gpu
    run_problem(make(), eng, strm)
    assert api.last_kernel() == "gemm_split"


def test_calls_in_a_row_see_each_other_s_results(gpu):
    """Kernels that start before their predecessor on the stream has ended: a chain of s8 layers, each reading what the
    one before it wrote, gives what the layers give one at a time."""
    import torch
    from onednn_b200.runner import Prepared
    eng, strm = gpu
    M, n = 40, 512
    p = W.int8_postops(M, n, n)
    dev = torch.device("cuda:0")
    put = lambda a: torch.from_numpy(np.ascontiguousarray(a).view(np.uint8).reshape(-1).copy()).to(dev)
    first = Prepared(p, eng).upload()
    bufs = [put(p.src.data)] + [torch.zeros(M * n, dtype=torch.uint8, device=dev) for _ in range(6)]
    args = []
    for i in range(6):
        a = dict(first.args)
        a[api.ARG_SRC] = api.memory(api.memory.desc((M, n), W.S8, api.tag.ab), eng, bufs[i].data_ptr())
        a[api.ARG_DST] = api.memory(api.memory.desc((M, n), W.S8, api.tag.ab), eng, bufs[i + 1].data_ptr())
        args.append(a)
    torch.cuda.synchronize()
    for a in args:
        first.prim.execute(strm, a)
        strm.wait()
    want = [b.cpu().numpy().copy() for b in bufs[1:]]
    assert np.unique(want[-1]).size > 2
    for _ in range(5):
        for b in bufs[1:]:
            b.zero_()
        torch.cuda.synchronize()
        for a in args:
            first.prim.execute(strm, a)
        strm.wait()
        for b, w in zip(bufs[1:], want):
            assert np.array_equal(b.cpu().numpy(), w)
