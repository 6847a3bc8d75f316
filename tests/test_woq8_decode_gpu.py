"""s8 weight decompression for few rows, dense and grouped: edges of row blocks, column tiles, K stages and experts."""
import numpy as np
import pytest

from onednn_b200 import api
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
    # blocks found across the 32s of experts that a warp looks through; experts of one, two and no blocks; as many experts as
    # the kernel takes, and one more
    "second_32_of_experts": lambda: W.moe_grouped(64, 96, 80, 41, sizes=[0] * 30 + [1, 0, 33, 0, 0, 0, 0, 0, 0, 1, 29]),
    "all_rows_last": lambda: W.moe_grouped(64, 64, 32, 65, sizes=[0] * 64 + [64]),
    "one_row_each": lambda: W.moe_grouped(64, 64, 48, 64, sizes=[1] * 64),
    "1024_experts": lambda: W.moe_grouped(63, 32, 32, 1024),
    "1025_experts": lambda: W.moe_grouped(63, 32, 32, 1025),
}


# enough rows for the other kernel, whose tile plan for a dense problem comes from the host
DENSE_ROWS = {
    "full_blocks": lambda: _dense(2900, 200, 1168),  # 14 x 10 tiles of up to 208 rows in one wave, 16 x 10 of up to 192 in two
    "low_blocks": lambda: _dense(3000, 128, 1040, dst_dt=W.F32),  # one wave either way
    "several_waves": lambda: _dense(3328, 136, 4112, per_tensor=True),
    "bias_relu": lambda: _bias_relu(_dense(3100, 144, 1056)),
}


@pytest.mark.parametrize("name", sorted(DENSE_ROWS))
def test_dense_many_rows_match_oracle(gpu, name):
    eng, strm = gpu
    p = DENSE_ROWS[name]()
    got, impl = run_problem(p, eng, strm)
    assert (impl, api.last_kernel()) == ("cuda:tcgen05:woq8", "grouped_tc")
    assert_parity(got, O.run_port(p), p.dst_dt, name, summation_slack(p))


@pytest.mark.parametrize("name", sorted(DENSE))
def test_dense_matches_oracle(gpu, name):
    eng, strm = gpu
    p = DENSE[name]()
    got, impl = run_problem(p, eng, strm)
    assert (impl, api.last_kernel()) == ("cuda:tcgen05:woq8", "woq8_decode")
    assert_parity(got, O.run_port(p), p.dst_dt, name, summation_slack(p))
    got2, _ = run_problem(p, eng, strm)
    assert np.array_equal(got, got2)


@pytest.mark.parametrize("name", sorted(GROUPED))
def test_grouped_matches_oracle(gpu, name):
    eng, strm = gpu
    p = GROUPED[name]()
    got, impl = run_problem(p, eng, strm)
    assert (impl, api.last_kernel()) == ("cuda:tcgen05:grouped", "grouped_tc" if name == "1025_experts" else "woq8_decode")
    assert_parity(got, O.run_port(p), p.dst_dt, name, summation_slack_grouped(p))


BAD_OFFSETS = {
    # (src ends, dst ends or None for the same): a step back, an end beyond the rows, fewer dst rows than src rows, a negative end
    "step_back": (lambda M: [10, 5, M - 3, M], None),
    "beyond_the_rows": (lambda M: [2, 7, M - 1, M + 1], None),
    "last_of_many": (lambda M: list(range(1, 21)) + [M] * 178 + [M - 1], None),
    "dst_rows_differ": (lambda M: [4, 9, 20, M], lambda M: [4, 10, 20, M]),
    "negative": (lambda M: [-1, 3, 8, M], None),
}


@pytest.mark.parametrize("M", [40, 64, 65, 300])
@pytest.mark.parametrize("name", sorted(BAD_OFFSETS))
def test_grouped_bad_offsets_write_nothing(gpu, name, M):
    """One wrong offset: the call reports invalid_arguments and dst stays as it was, for few rows (whose kernel reads the
    offsets itself) as for many (which have a planning kernel)."""
    from onednn_b200.runner import Prepared
    eng, strm = gpu
    ends, dst_ends = (f(M) if f else None for f in BAD_OFFSETS[name])
    n = len(ends)
    p = W.moe_grouped(M, 128, 160, n, sizes=[M] + [0] * (n - 1))
    p.offsets = np.array(ends, np.int32)
    p.dst_init = np.full((M, p.N), 0x4242, np.uint16)
    r = Prepared(p, eng).upload()
    if dst_ends:
        r.args[api.ARG_DST].write(np.array(dst_ends, np.int32), 1)
    for _ in range(2):
        r.execute(strm)
        with pytest.raises(api.error) as ei:
            strm.wait()
        assert ei.value.status == api.invalid_arguments
        assert np.array_equal(r.download(), p.dst_init)
    strm.wait()  # the status word is cleared: the stream stays usable
