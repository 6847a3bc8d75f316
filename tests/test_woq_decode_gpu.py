"""int4 weight decompression: the edges of the decode kernel's row blocks, column tiles, K stages and groups, and, for more than
32 rows, both kernels that the choice falls on."""
import numpy as np
import pytest

from onednn_b200 import api
from onednn_b200 import workloads as W
from onednn_b200.runner import run_problem
from oracle import oracle as O
from test_parity_gpu import _requantized, _src_scale, _with_bias_relu
from util import assert_parity, summation_slack

pytestmark = pytest.mark.gpu


def _scales(p, dt):
    q = p.quant["wei_scale"]
    p.quant["wei_scale"] = W.Quant(W.to_storage(W.to_f32(q.data, q.dt), dt), dt, q.mask, q.groups)
    return p


def _common_zp(p, value, dt):
    p.quant["wei_zp"] = W.Quant(W.to_storage(np.array([value]), dt), dt, 0)
    return p


def _wide_zp(p, dt, lo, hi):
    """Zero-points per (group, column) of another type, in [lo, hi)."""
    q = p.quant["wei_zp"]
    r = np.random.Generator(np.random.PCG64(17))
    p.quant["wei_zp"] = W.Quant(W.to_storage(r.integers(lo, hi, (p.K // q.groups[0], p.N)), dt), dt, 3, q.groups)
    return p


def _one_scale_row(p):
    q = p.quant["wei_scale"]
    p.quant["wei_scale"] = W.Quant(np.ascontiguousarray(q.data.reshape(-1, p.N)[:1]), q.dt, 2)
    p.quant.pop("wei_zp", None)
    return p


def _large_scales():
    """f32 scales just below the type's range against src values as far below 1: all products and sums are finite."""
    p = W.int4_decode(6, 256, 160, with_zp=False, dst_dt=W.F32)
    r = np.random.Generator(np.random.PCG64(11))
    p.src = W.QTensor(W.f32_to_bf16(W.bf16_to_f32(p.src.data) * np.float32(2.0 ** -100)), W.BF16, p.src.dims)
    q = p.quant["wei_scale"]
    p.quant["wei_scale"] = W.Quant((r.uniform(1.0, 1.99, q.data.shape) * 2.0 ** 123).astype(np.float32), W.F32, 3, q.groups)
    return p


CASES = {
    "one_step_one_column_piece": lambda: W.int4_decode(1, 16, 32, group=16),
    "m9_two_blocks": lambda: W.int4_decode(9, 512, 288),
    "m24_three_blocks": lambda: W.int4_decode(24, 1024, 544, group=64),
    "m25_four_blocks_f16": lambda: W.int4_decode(25, 768, 256, wei_dt=W.U4, src_dt=W.F16, dst_dt=W.F16, with_zp=False, group=64),
    "m17_group32": lambda: W.int4_decode(17, 416, 320, group=32),
    "m16_group48_across_stages": lambda: W.int4_decode(16, 1104, 256, group=48),
    "m32_group16": lambda: W.int4_decode(32, 272, 160, group=16, zp_dt=W.S4),
    "k_tail_group16": lambda: W.int4_decode(3, 1040, 96, group=16, wei_dt=W.U4),
    "k_tail_one_group": lambda: _one_scale_row(W.int4_decode(11, 1072, 288, group=16)),
    "shares_cut_groups": lambda: W.int4_decode(2, 4096, 256, group=512),
    "eight_shares_ring_turns": lambda: W.int4_decode(5, 8192, 256),
    "many_tiles": lambda: W.int4_decode(1, 256, 40992),
    "f16_s4_s4zp": lambda: W.int4_decode(13, 1024, 288, zp_dt=W.S4, src_dt=W.F16, dst_dt=W.F32),
    "u8_zp_m20": lambda: W.int4_decode(20, 512, 288, zp_dt=W.U8),
    "s8_zp_f16_m30": lambda: W.int4_decode(30, 512, 288, wei_dt=W.U4, zp_dt=W.S8, src_dt=W.F16, dst_dt=W.F16),
    "u8_zp_f32_scales_group32": lambda: _scales(W.int4_decode(9, 544, 160, group=32, zp_dt=W.U8), W.F32),
    "s8_zp_group16_m27": lambda: W.int4_decode(27, 272, 288, group=16, wei_dt=W.U4, zp_dt=W.S8),
    "f32_scales_m32_group16": lambda: _scales(W.int4_decode(32, 272, 160, group=16), W.F32),
    "f32_scales_no_zp_m24": lambda: _scales(W.int4_decode(24, 1024, 288, group=64, with_zp=False), W.F32),
    "u8_zp_u4_weights_up_to_255": lambda: _wide_zp(W.int4_decode(6, 512, 160, wei_dt=W.U4), W.U8, 200, 256),
    "common_s8_zp_m32_group32": lambda: _common_zp(W.int4_decode(32, 512, 160, group=32), -128, W.S8),
    "u8_zp_m32_group64_f16": lambda: _wide_zp(W.int4_decode(32, 1024, 288, group=64, src_dt=W.F16, dst_dt=W.F16), W.U8, 0, 256),
    # zero-points of which a rest has to come off the sums: some columns of some groups, all of them, groups across stages
    "u8_zp_above_248": lambda: _wide_zp(W.int4_decode(5, 2048, 288, group=64), W.U8, 230, 256),
    "u8_zp_above_248_m32_group48": lambda: _wide_zp(W.int4_decode(32, 1104, 160, group=48), W.U8, 240, 256),
    "s32_zp_mixed_m20": lambda: _wide_zp(W.int4_decode(20, 640, 160, group=32, wei_dt=W.U4), W.S32, -400, 300),
    "s32_zp_f16_m3": lambda: _wide_zp(W.int4_decode(3, 512, 160, src_dt=W.F16, dst_dt=W.F32), W.S32, -1100, 1100),
    "common_s32_zp": lambda: _common_zp(W.int4_decode(18, 512, 160), -7, W.S32),
    "common_s32_zp_large": lambda: _common_zp(W.int4_decode(7, 1040, 160, group=16), 3000, W.S32),
    "common_u8_zp_255_per_n_scale": lambda: _common_zp(_one_scale_row(W.int4_decode(11, 1072, 288, group=16)), 255, W.U8),
    "common_zp": lambda: _common_zp(W.int4_decode(7, 512, 160), -77, W.S8),
    "f32_scales_u4_zp": lambda: _scales(W.int4_decode(12, 640, 160, group=64), W.F32),
    "f16_scales": lambda: _scales(W.int4_decode(8, 640, 160), W.F16),
    "f8_scales": lambda: _scales(W.int4_decode(3, 512, 160, with_zp=False), W.F8_E4M3),
    "large_f32_scales": _large_scales,
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_matches_oracle(gpu, name):
    eng, strm = gpu
    p = CASES[name]()
    got, impl = run_problem(p, eng, strm)
    assert impl == "cuda:tcgen05:woq4"
    assert_parity(got, O.run_port(p), p.dst_dt, name, summation_slack(p))
    got2, _ = run_problem(p, eng, strm)  # the shares are added in the same order every time
    assert np.array_equal(got, got2)


ROWS_CASES = {
    # blocks of rows of the decode kernel: 2 x 17, 2 x 32, 3 x 22 with a short last one, ...
    "m33": ("woq_decode", lambda: W.int4_decode(33, 1024, 288)),
    "m64_group32": ("woq_decode", lambda: W.int4_decode(64, 512, 160, group=32)),
    "m65_f16": ("woq_decode", lambda: W.int4_decode(65, 768, 544, wei_dt=W.U4, src_dt=W.F16, dst_dt=W.F16, group=64)),
    "m97_k_tail": ("woq_decode", lambda: W.int4_decode(97, 1104, 96, group=16)),
    # enough tiles and short K for the kernel with the operand in tensor memory
    "m1000_group128": ("woq_rows", lambda: W.int4_decode(1000, 512, 1056)),
    "m2040_group64": ("woq_rows", lambda: W.int4_decode(2040, 256, 1024, group=64)),
    "m2048_group32_u4": ("woq_rows", lambda: W.int4_decode(2048, 256, 1024, group=32, wei_dt=W.U4)),
    "m2000_group48": ("woq_rows", lambda: W.int4_decode(2000, 288, 1024, group=48)),
    "m1024_f16_u8zp": ("woq_rows", lambda: W.int4_decode(1024, 512, 1024, group=256, zp_dt=W.U8, src_dt=W.F16, dst_dt=W.F16)),
    "m1024_no_zp": ("woq_rows", lambda: W.int4_decode(1024, 528, 1024, group=528, with_zp=False, dst_dt=W.F32)),
    "m1024_f16_group64": ("woq_rows", lambda: W.int4_decode(1024, 768, 1056, group=64, wei_dt=W.U4, src_dt=W.F16, dst_dt=W.F16, with_zp=False)),
    "m1000_group64_ring_turns": ("woq_rows", lambda: W.int4_decode(1000, 1536, 1056, group=64)),
    "m1024_one_scale_row": ("woq_rows", lambda: _one_scale_row(W.int4_decode(1024, 384, 1056))),
    # that kernel takes scales of other types at any size: long K (the ten stages of weights turn twice), several tiles per
    # CTA, groups of every kind, options of the epilogue
    "f32_scales_32_groups": ("woq_rows", lambda: _scales(W.int4_decode(70, 4096, 256), W.F32)),
    "f32_scales_long_k_tail": ("woq_rows", lambda: _scales(W.int4_decode(50, 2896, 160, group=16), W.F32)),
    "f32_scales_group64_s4zp": ("woq_rows", lambda: _scales(W.int4_decode(129, 3072, 160, group=64, wei_dt=W.U4, zp_dt=W.S4), W.F32)),
    "f32_scales_group256": ("woq_rows", lambda: _scales(W.int4_decode(48, 4096, 128, group=256), W.F32)),
    "f32_scales_two_tiles_per_cta": ("woq_rows", lambda: _scales(W.int4_decode(33, 2816, 19072), W.F32)),
    "f32_scales_bias_relu": ("woq_rows", lambda: _with_bias_relu(_scales(W.int4_decode(48, 512, 256), W.F32))),
    "f32_scales_src_scale": ("woq_rows", lambda: _src_scale(_scales(W.int4_decode(72, 384, 160), W.F32))),
    "f32_scales_requantized_s8": ("woq_rows", lambda: _requantized(_scales(W.int4_decode(55, 256, 160, dst_dt=W.S8), W.F32))),
    "f8_scales": ("woq_rows", lambda: _scales(W.int4_decode(38, 512, 160, with_zp=False), W.F8_E4M3)),
    "common_zp_f16": ("woq_rows", lambda: _common_zp(W.int4_decode(64, 2944, 160, src_dt=W.F16, dst_dt=W.F32), -128, W.S8)),
    "u8_zp_f16_long_k": ("woq_rows", lambda: W.int4_decode(80, 2944, 256, zp_dt=W.U8, src_dt=W.F16, dst_dt=W.F32)),
}


@pytest.mark.parametrize("name", sorted(ROWS_CASES))
def test_more_rows_match_oracle(gpu, name):
    eng, strm = gpu
    kernel, make = ROWS_CASES[name]
    p = make()
    got, impl = run_problem(p, eng, strm)
    assert impl == "cuda:tcgen05:woq4_rows"
    assert api.last_kernel() == kernel  # (both report that name: a change of the choice would move cases unnoticed)
    assert_parity(got, O.run_port(p), p.dst_dt, name, summation_slack(p))
    got2, _ = run_problem(p, eng, strm)
    assert np.array_equal(got, got2)


@pytest.mark.parametrize("src_dt,M", [(W.F16, 4), (W.F16, 32), (W.BF16, 4), (W.BF16, 32), (W.F16, 40), (W.F16, 300)],
                         ids=["f16_m4", "f16_m32", "bf16_m4", "bf16_m32", "f16_m40", "f16_m300"])
@pytest.mark.parametrize("zp", ["common_u8", "u8_per_group", "u4_per_group"])
def test_zero_points_come_off_the_weights(gpu, src_dt, M, zp):
    """Activations of one sign: w - zero_point is taken exactly before the products are summed.  Summing over w and taking
    zero_point * sum(src) off afterwards cancels: it costs a factor of twenty and more in accuracy here."""
    eng, strm = gpu
    p = W.int4_decode(M, 4096, 160, group=512, wei_dt=W.U4, zp_dt=W.U4 if zp == "u4_per_group" else W.U8, src_dt=src_dt, dst_dt=W.F32)
    p.src = W.QTensor(p.src.data & 0x7fff, src_dt, p.src.dims)  # |src|
    r = np.random.Generator(np.random.PCG64(21))
    if zp == "common_u8":
        _common_zp(p, 8, W.U8)
    else:
        p.quant["wei_zp"] = W.Quant(W.to_storage(r.integers(7, 10, (8, 160)), p.quant["wei_zp"].dt), p.quant["wei_zp"].dt, 3, (512, 1))
    got, impl = run_problem(p, eng, strm)
    assert impl == ("cuda:tcgen05:woq4" if M <= 32 else "cuda:tcgen05:woq4_rows")
    zq = p.quant["wei_zp"]
    z = np.broadcast_to(W.to_f32(zq.data, zq.dt).astype(np.float64).reshape(-1, 160 if zp != "common_u8" else 1), (8, 160))
    w = W.to_f32(p.wei.data, W.U4).astype(np.float64).reshape(4096, 160) - np.repeat(z, 512, 0)
    q = p.quant["wei_scale"]
    w *= np.repeat(W.to_f32(q.data, q.dt).astype(np.float64).reshape(8, 160), 512, 0)
    exact = W.to_f32(p.src.data, src_dt).astype(np.float64).reshape(M, 4096) @ w
    err = np.linalg.norm(got - exact) / np.linalg.norm(exact)
    # a group's 32 blocks of 16 exact products are added in f32 one after another; the tensor cores cut each sum off, by up to
    # 2^-23 of it, 2^-24 on average, and the running sum is half the last one on average: 32 * 2^-24 / 2 = 9.5e-7 at most where
    # all errors have one sign (measured: 1.0e-7 to 1.8e-7; 3.7e-6 to 4.2e-6 with the zero-points taken off afterwards)
    assert err < 1e-6, err


def test_calls_in_a_row_see_each_other_s_results(gpu):
    """The kernel starts before its predecessor on the stream has ended: a chain of calls, each reading what the one
    before it wrote, gives what the calls give one at a time."""
    import torch
    from onednn_b200.runner import Prepared
    eng, strm = gpu
    n = 1024
    p = W.int4_decode(4, n, n)
    first = Prepared(p, eng)
    dev = torch.device("cuda:0")
    put = lambda a: torch.from_numpy(np.ascontiguousarray(a).view(np.uint8).reshape(-1).copy()).to(dev)
    fixed = {"wei": put(p.wei.data), **{k: put(q.data) for k, q in p.quant.items()}}
    # small weights keep the values of the chain in range
    bufs = [put(p.src.data)] + [torch.zeros(4 * n * 2, dtype=torch.uint8, device=dev) for _ in range(6)]

    def bound(i):
        r = first if i == 0 else Prepared(p, eng)
        r.bind_device({"src": bufs[i].data_ptr(), "dst": bufs[i + 1].data_ptr(), **{k: t.data_ptr() for k, t in fixed.items()}})
        return r

    calls = [bound(i) for i in range(6)]
    torch.cuda.synchronize()
    for r in calls:
        r.execute(strm)
        strm.wait()
    want = [b.cpu().numpy().copy() for b in bufs[1:]]
    for _ in range(5):
        for b in bufs[1:]:
            b.zero_()
        torch.cuda.synchronize()
        for r in calls:
            r.execute(strm)
        strm.wait()
        for b, w in zip(bufs[1:], want):
            assert np.array_equal(b.cpu().numpy(), w)
