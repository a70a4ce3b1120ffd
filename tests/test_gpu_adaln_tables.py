"""The adaLN tables that feed the fused norm: launch_adaln_expand (bit-exact) and the fp32-compute Linear."""
import ctypes as C

import numpy as np
import pytest
import torch

import oracle
import slopfab_b200 as sfq
from helpers import RefWeight, dev, ref_check, ref_weight_from

pytestmark = pytest.mark.gpu


def _ref():
    ref = oracle.ref
    if ref is None:
        return None
    V, I = C.c_void_p, C.c_int
    ref.ref_dev_adaln_expand.argtypes = [V, V, V, V, I, I, I, I, I]
    ref.ref_dev_linear_forward_f32.argtypes = [C.POINTER(RefWeight), V, I, V]
    ref.ref_last_error.restype = C.c_char_p
    return ref


@pytest.mark.parametrize("num_t,modalities,params,channels,rank", [(1, 3, 6, 64, 16), (3, 3, 6, 320, 64), (2, 1, 2, 5120, 256)])
def test_adaln_expand_is_bit_exact(num_t, modalities, params, channels, rank):
    features = modalities * params * channels
    w = oracle.make_data(features * rank, 41, 0.2).reshape(features, rank)
    bias = oracle.make_data(features, 42, 0.5)
    code = oracle.make_data(num_t * rank, 43, 1.0).reshape(num_t, rank)
    want = oracle.adaln_expand(w, bias, code, modalities, params, channels)
    dw, db, dc = dev(w), dev(bias), dev(code)
    out = torch.empty(want.shape, dtype=torch.float32, device="cuda")
    sfq.check(sfq.lib.sfq_adaln_expand(sfq.ptr(dw), sfq.ptr(db), sfq.ptr(dc), sfq.ptr(out), num_t, modalities, params, channels, rank,
                                       sfq.stream_ptr()))
    got = out.cpu().numpy()
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
    # row p = (modality * params + param) * channels + channel of the Linear lands at [param, t, modality, channel]
    p = (1 % modalities * params + 1) * channels + 5
    acc = np.float32(bias[p])
    for k in range(rank):
        acc = np.float32(np.float64(w[p, k]) * np.float64(code[0, k]) + np.float64(acc))  # fma: one rounding
    assert got[1, 0, 1 % modalities, 5] == acc
    ref = _ref()
    if ref is not None:
        rout = torch.empty_like(out)
        ref_check(ref, ref.ref_dev_adaln_expand(sfq.ptr(dw), sfq.ptr(db), sfq.ptr(dc), sfq.ptr(rout), num_t, modalities, params,
                                                channels, rank))
        assert torch.equal(rout, out)


def test_adaln_expand_refusals():
    t = torch.zeros(16, dtype=torch.float32, device="cuda")
    for args in [(0, 1, 1, 4, 4), (1, 1, 1, 4, 0), (70000, 1, 1, 4, 4)]:
        with pytest.raises(sfq.SfqError, match="launch_adaln_expand"):
            sfq.check(sfq.lib.sfq_adaln_expand(sfq.ptr(t), sfq.ptr(t), sfq.ptr(t), sfq.ptr(t), *args, None))


@pytest.mark.parametrize("fmt", ["f32", "bf16"])
@pytest.mark.parametrize("rows,n,k", [(1, 192, 64), (3, 1000, 256), (70, 130, 100)])
def test_forward_f32_against_the_fp64_product(fmt, rows, n, k):
    rng = np.random.default_rng(rows + n)
    x = rng.standard_normal((rows, k)).astype(np.float32)
    w = (0.05 * rng.standard_normal((n, k))).astype(np.float32)
    bias = rng.standard_normal(n).astype(np.float32)
    if fmt == "bf16":
        wbits = oracle.to_bf16(w)
        w = oracle.from_bf16(wbits)
        dw = dev(wbits)
        weight = sfq.new_weight(format=sfq.BF16, data=sfq.ptr(dw), out_features=n, in_features=k)
    else:
        dw = dev(w)
        weight = sfq.new_weight(format=sfq.F32, data=sfq.ptr(dw), out_features=n, in_features=k)
    db = dev(bias)
    weight.bias = sfq.ptr(db)
    weight.bias_format = sfq.F32
    runner = sfq.LinearRunner()
    dx = dev(x)
    got = runner.forward_f32(weight, dx).cpu().numpy()
    want = x.astype(np.float64) @ w.astype(np.float64).T + bias
    # fp32 accumulation over k terms of magnitude ~|x||w|: a few ulps of the largest partial sum
    assert np.abs(got - want).max() <= 2e-6 * k * np.abs(x).max() * np.abs(w).max() + 1e-6
    ref = _ref()
    if ref is not None:
        ry = torch.empty((rows, n), dtype=torch.float32, device="cuda")
        rw = ref_weight_from(weight)
        ref_check(ref, ref.ref_dev_linear_forward_f32(C.byref(rw), sfq.ptr(dx), rows, sfq.ptr(ry)))
        assert np.abs(ry.cpu().numpy() - got).max() <= 2e-6 * k * np.abs(x).max() * np.abs(w).max() + 1e-6


@pytest.mark.parametrize("fmt", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows,n,k", [(1, 5, 4), (3, 2368, 516), (4, 2371, 5120), (5, 3000, 1000), (8, 30, 512), (9, 2400, 516), (16, 2369, 2052),
                                      (17, 2500, 132), (64, 2500, 1024), (65, 300, 256), (3, 300, 258)])
def test_forward_f32_row_tiles(fmt, rows, n, k):
    """Every row tile (1, 4, 8, 16), one and four features per CTA, ragged ends of all three extents, and the tiled kernel behind
    them (K not in fours). Bound: (K / 256 + 16) additions of fp32 terms, each rounding by 2^-24 of the sum of
    the terms' magnitudes at most."""
    g = torch.Generator("cuda").manual_seed(rows + n)
    x = torch.randn((rows, k), device="cuda", generator=g)
    w = torch.randn((n, k), device="cuda", generator=g).mul_(0.05).to(fmt)
    bias = torch.randn(n, device="cuda", generator=g)
    weight = sfq.new_weight(format=sfq.F32 if fmt == torch.float32 else sfq.BF16, data=sfq.ptr(w), out_features=n, in_features=k,
                            bias=sfq.ptr(bias), bias_format=sfq.F32)
    got = sfq.LinearRunner().forward_f32(weight, x)
    want = x.double() @ w.double().T + bias.double()
    terms = x.double().abs() @ w.double().abs().T + bias.double().abs()
    steps = (k / 256 + 16) if k % 4 == 0 else k + 1
    assert bool(((got.double() - want).abs() <= steps * 2.0 ** -24 * terms).all())


@pytest.mark.parametrize("fmt", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("rows,n,k", [(64, 30720, 256), (33, 5120, 64), (513, 2560, 512), (3000, 512, 512), (600, 9000, 1024)])
def test_forward_f32_of_many_rows_or_short_sums(fmt, rows, n, k):
    """Where the tiled kernel is the faster one it runs whatever the alignment allows: the bits of a call are those of the same call
    with an x that only the tiled kernel can read. Bound: one fp32 rounding per term, by 2^-24 of the terms' magnitudes at most."""
    g = torch.Generator("cuda").manual_seed(rows + n)
    x = torch.randn((rows, k), device="cuda", generator=g)
    w = torch.randn((n, k), device="cuda", generator=g).mul_(0.05).to(fmt)
    weight = sfq.new_weight(format=sfq.F32 if fmt == torch.float32 else sfq.BF16, data=sfq.ptr(w), out_features=n, in_features=k)
    runner = sfq.LinearRunner()
    got = runner.forward_f32(weight, x)
    shifted = torch.empty(rows * k + 1, device="cuda")[1:].view(rows, k)
    shifted.copy_(x)
    assert torch.equal(got, runner.forward_f32(weight, shifted))
    want = x.double() @ w.double().T
    terms = x.double().abs() @ w.double().abs().T
    assert bool(((got.double() - want).abs() <= (k + 1) * 2.0 ** -24 * terms).all())


def test_forward_f32_refuses_what_it_does_not_build():
    t = torch.zeros(256 * 256, dtype=torch.float32, device="cuda")
    runner = sfq.LinearRunner()
    w = sfq.new_weight(format=sfq.W4A8, data=sfq.ptr(t), out_features=256, in_features=256)
    with pytest.raises(sfq.SfqError, match="BF16 activations"):
        runner.forward_f32(w, t.view(256, 256))
