"""s8 weight decompression for few rows, dense and grouped: edges of row blocks, column tiles, K stages and experts."""
import numpy as np
import pytest

from onednn_b200 import workloads as W
from onednn_b200.runner import run_problem
from oracle import oracle as O
from util import assert_parity, summation_slack, summation_slack_grouped

pytestmark = pytest.mark.gpu


def _dense(M, K, N, dst_dt=W.BF16, per_tensor=False):
    p = W.int4_decode(M, K, N, group=K, wei_dt=W.S8, with_zp=False, dst_dt=dst_dt)
    r = np.random.Generator(np.random.PCG64(3))
    p.quant["wei_scale"] = W.Quant(r.uniform(0.001, 0.01, (1,) if per_tensor else (1, N)).astype(np.float32), W.F32, 0 if per_tensor else 2)
    return p


def _bias_relu(p):
    r = np.random.Generator(np.random.PCG64(9))
    p.bias = W.QTensor(W.f32_to_bf16(r.standard_normal((1, p.N), dtype=np.float32)), W.BF16, (1, p.N))
    p.post_ops.append(W.PostOp(W.PO_ELTWISE, W.ELTWISE["relu"], 0.0, 0.0, 1.0))
    return p


DENSE = {
    "one_stage": lambda: _dense(1, 16, 16),
    "m8_tail_columns": lambda: _dense(8, 512, 144),
    "m9_k_tail": lambda: _dense(9, 1040, 272, dst_dt=W.F32),
    "m24_long_k": lambda: _dense(24, 8192, 128, dst_dt=W.F16),
    "m33_two_blocks": lambda: _dense(33, 2048, 400),
    "m100_four_blocks_per_tensor": lambda: _dense(100, 1024, 528, per_tensor=True),
    "bias_relu": lambda: _bias_relu(_dense(19, 768, 336)),
}
GROUPED = {
    "one_row": lambda: W.moe_grouped(1, 256, 128, 4, sizes=[0, 0, 1, 0]),
    "block_edges": lambda: W.moe_grouped(64, 320, 272, 5, sizes=[32, 0, 7, 25, 0]),
    "two_blocks_of_an_expert": lambda: W.moe_grouped(50, 1088, 160, 3, sizes=[1, 41, 8]),
    "many_experts": lambda: W.moe_grouped(40, 128, 64, 70),
}


@pytest.mark.parametrize("name", sorted(DENSE))
def test_dense_matches_oracle(gpu, name):
    eng, strm = gpu
    p = DENSE[name]()
    got, impl = run_problem(p, eng, strm)
    assert impl == "cuda:tcgen05:woq8"
    assert_parity(got, O.run_port(p), p.dst_dt, name, summation_slack(p))
    got2, _ = run_problem(p, eng, strm)
    assert np.array_equal(got, got2)


@pytest.mark.parametrize("name", sorted(GROUPED))
def test_grouped_matches_oracle(gpu, name):
    eng, strm = gpu
    p = GROUPED[name]()
    got, impl = run_problem(p, eng, strm)
    assert impl == "cuda:tcgen05:grouped"
    assert_parity(got, O.run_port(p), p.dst_dt, name, summation_slack_grouped(p))
