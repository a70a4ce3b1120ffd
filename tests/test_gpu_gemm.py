"""GPU parity of the tcgen05 GEMMs and of the LinearRunner, through the C ABI.

int8: accumulators exact, so the bf16 output must equal the oracle's bit for bit (the reference's own
bar for W4A8/W6A8). nvfp4: fp32 accumulation order is the tensor core's, so the bar is the tolerance the
task states -- max-abs 2e-2 and relative-L2 1e-3 against the fp4-activation oracle rounded to bf16 --
plus the reference tests' wrong-layout controls. bf16: 1e-3 abs / 1e-2 rel as in linear_nvfp4.
"""
import ctypes as C

import numpy as np
import pytest
import torch

import oracle
import slopfab_b200 as sfq
from slopfab_b200.block import BlockWeights, Nvfp4Block, Nvfp4Linear
from helpers import (P, bf16_tensor, bits, dev, gaussian_bf16, pack_nvfp4, pack_w4a8, pack_w6a8, ref_check, ref_dev,
                     ref_weight_from, synthetic_packed_int8)

pytestmark = pytest.mark.gpu
S = None


def _status_clean():
    assert sfq.device_status() == 0, "a kernel abandoned a bounded wait"


@pytest.mark.parametrize("tile_n", [0, 256, 128])
@pytest.mark.parametrize("M,N,K", [(128, 256, 128), (1, 128, 256), (200, 384, 512), (129, 34, 256), (300, 520, 1280),
                                   (257, 1024, 5120)])
def test_gemm_int8_bit_exact(M, N, K, tile_n):
    rng = np.random.default_rng(M * 7 + N + K)
    a = rng.integers(-128, 128, size=(M, K), dtype=np.int8)
    w = rng.integers(-127, 128, size=(N, K), dtype=np.int8)
    rs = (rng.random(M, dtype=np.float32) * 0.05 + 1e-3).astype(np.float32)
    cs = (rng.random(N, dtype=np.float32) * 0.01 + 1e-4).astype(np.float32)
    bias = (0.01 * rng.standard_normal(N)).astype(np.float32)
    da, dw, drs, dcs, db = dev(a), dev(w), dev(rs), dev(cs), dev(bias)
    acc = oracle.int8_gemm(a, w)
    sfq.lib.sfq_test_gemm_variant(tile_n, 0, 0)
    try:
        for use_bias, act in ((False, sfq.ACT_NONE), (True, sfq.ACT_NONE), (True, sfq.ACT_GELU_TANH)):
            y = torch.full((M, N), float("nan"), dtype=torch.bfloat16, device="cuda")
            ep = sfq.Epilogue(sfq.ptr(drs), sfq.ptr(dcs), 1.0, sfq.ptr(db) if use_bias else None, sfq.F32, act)
            sfq.check(sfq.lib.sfq_gemm_int8(sfq.ptr(da), sfq.ptr(dw), C.byref(ep), sfq.ptr(y), M, N, K, S))
            _status_clean()
            want = np.empty((M, N), np.uint16)
            oracle.lib.orc_w4a8_output_bf16(P(acc), P(rs), P(cs), M, N, P(want))
            if use_bias:
                oracle.lib.orc_add_bias_bf16(P(want), P(bias), 0, M, N)
            got = bits(y)
            if act == sfq.ACT_GELU_TANH:
                oracle.lib.orc_gelu_tanh_bf16(P(want), want.size)
                worst = np.abs(got.astype(np.int32) - want.astype(np.int32)).max()
                assert worst <= 1, f"GELU epilogue off by {worst} bf16 ulps"
            else:
                bad = int((got != want).sum())
                assert bad == 0, f"{bad} of {M * N} outputs differ (bias={use_bias}); first at {np.argwhere(got != want)[:4]}"
    finally:
        sfq.lib.sfq_test_gemm_variant(0, 0, 0)


@pytest.mark.parametrize("M,N,K", [(128, 256, 128), (300, 512, 1024), (257, 384, 2048), (1000, 5120, 5120), (4096, 1280, 13824)])
def test_w4a8_expanded_inside_the_gemm_equals_unpack_then_gemm(M, N, K):
    """The int8 weight rows produced in shared memory inside the GEMM are those of the stand-alone unpacker, so the int32
    accumulators and every output bit agree with unpack + GEMM (which the tests above pin to the oracle); the oracle's own
    decode is checked directly on a sample of rows."""
    packed, s_rel, s_ch, book = synthetic_packed_int8(4, 16, N, K, seed=M + N + K)
    rng = np.random.default_rng(M * 3 + K)
    a = rng.integers(-128, 128, size=(M, K), dtype=np.int8)
    rs = (rng.random(M, dtype=np.float32) * 0.05 + 1e-3).astype(np.float32)
    bias = (0.01 * rng.standard_normal(N)).astype(np.float32)
    da, dp, dg, dbk, drs, dcs, db = dev(a), dev(packed), dev(s_rel), dev(book), dev(rs), dev(s_ch), dev(bias)
    w8 = torch.empty((N, K), dtype=torch.int8, device="cuda")
    sfq.check(sfq.lib.sfq_unpack_w4a8_int8(sfq.ptr(dp), sfq.ptr(dg), sfq.ptr(dbk), sfq.ptr(w8), N, K, 16, S))
    for use_bias, act in ((False, sfq.ACT_NONE), (True, sfq.ACT_GELU_TANH)):
        ep = sfq.Epilogue(sfq.ptr(drs), sfq.ptr(dcs), 1.0, sfq.ptr(db) if use_bias else None, sfq.F32, act)
        want = torch.full((M, N), float("nan"), dtype=torch.bfloat16, device="cuda")
        sfq.check(sfq.lib.sfq_gemm_int8(sfq.ptr(da), sfq.ptr(w8), C.byref(ep), sfq.ptr(want), M, N, K, S))
        for rep in range(2):  # twice: the second launch starts from warm barriers' other phase
            got = torch.full((M, N), float("nan"), dtype=torch.bfloat16, device="cuda")
            sfq.check(sfq.lib.sfq_gemm_w4a8_fused(sfq.ptr(da), sfq.ptr(dp), sfq.ptr(dg), sfq.ptr(dbk), C.byref(ep), sfq.ptr(got), M, N, K, S))
            _status_clean()
            bad = int((got.view(torch.int16) != want.view(torch.int16)).sum())
            assert bad == 0, f"{bad} of {M * N} outputs differ (bias={use_bias}, launch {rep})"
    # against the oracle's decode and integer product on a few rows of the activation
    rows = np.unique(np.concatenate([[0, M - 1], rng.integers(0, M, size=6)]))
    w_ref = w8.cpu().numpy()
    acc = oracle.int8_gemm(np.ascontiguousarray(a[rows]), w_ref)
    out = np.empty((len(rows), N), np.uint16)
    oracle.lib.orc_w4a8_output_bf16(P(acc), P(np.ascontiguousarray(rs[rows])), P(s_ch), len(rows), N, P(out))
    ep = sfq.Epilogue(sfq.ptr(drs), sfq.ptr(dcs), 1.0, None, sfq.F32, sfq.ACT_NONE)
    got = torch.empty((M, N), dtype=torch.bfloat16, device="cuda")
    sfq.check(sfq.lib.sfq_gemm_w4a8_fused(sfq.ptr(da), sfq.ptr(dp), sfq.ptr(dg), sfq.ptr(dbk), C.byref(ep), sfq.ptr(got), M, N, K, S))
    assert np.array_equal(bits(got)[rows], out)


def test_w4a8_fused_refuses_what_it_does_not_cover():
    M, N, K = 128, 256, 192  # K is not a multiple of 128
    z = torch.zeros(1 << 16, dtype=torch.uint8, device="cuda")
    y = torch.empty((M, N), dtype=torch.bfloat16, device="cuda")
    ep = sfq.Epilogue(sfq.ptr(z), sfq.ptr(z), 1.0, None, sfq.F32, sfq.ACT_NONE)
    assert sfq.lib.sfq_gemm_w4a8_fused(sfq.ptr(z), sfq.ptr(z), sfq.ptr(z), sfq.ptr(z), C.byref(ep), sfq.ptr(y), M, N, K, S) != 0
    assert sfq.lib.sfq_gemm_w4a8_fused(None, sfq.ptr(z), sfq.ptr(z), sfq.ptr(z), C.byref(ep), sfq.ptr(y), M, N, 256, S) != 0


def test_gemm_int8_multi_tile_persistence():
    # more tiles than SMs, ragged M, several raster bands: every CTA walks several tiles through both accumulators
    M, N, K = 128 * 37 - 8, 1536, 512
    rng = np.random.default_rng(5)
    a = rng.integers(-128, 128, size=(M, K), dtype=np.int8)
    w = rng.integers(-127, 128, size=(N, K), dtype=np.int8)
    rs = np.full(M, 2.0 ** -6, np.float32)
    cs = np.full(N, 2.0 ** -7, np.float32)
    y = torch.empty((M, N), dtype=torch.bfloat16, device="cuda")
    da, dw, drs, dcs = dev(a), dev(w), dev(rs), dev(cs)
    ep = sfq.Epilogue(sfq.ptr(drs), sfq.ptr(dcs), 1.0, None, sfq.F32, sfq.ACT_NONE)
    sfq.check(sfq.lib.sfq_gemm_int8(sfq.ptr(da), sfq.ptr(dw), C.byref(ep), sfq.ptr(y), M, N, K, S))
    _status_clean()
    want = (da.float() @ dw.float().T) * (2.0 ** -13)  # exact in fp32: |acc| < 2^24
    assert torch.equal(y, want.to(torch.bfloat16))


@pytest.mark.parametrize("M,N,K", [(128, 256, 128), (300, 512, 520), (77, 128, 5120), (2500, 768, 1032)])
def test_gemm_bf16_within_reference_tolerance(M, N, K):
    x = bf16_tensor(gaussian_bf16((M, K), seed=M))
    w = bf16_tensor(gaussian_bf16((N, K), seed=N + 1, sigma=0.02))
    y = torch.empty((M, N), dtype=torch.bfloat16, device="cuda")
    ep = sfq.Epilogue(None, None, 1.0, None, sfq.F32, sfq.ACT_NONE)
    sfq.check(sfq.lib.sfq_gemm_bf16(sfq.ptr(x), sfq.ptr(w), C.byref(ep), sfq.ptr(y), M, N, K, S))
    _status_clean()
    want = x.float() @ w.float().T
    assert torch.all((y.float() - want).abs() <= 1e-3 + 1e-2 * want.abs())


@pytest.mark.parametrize("kind", ["int8", "bf16", "nvfp4"])
@pytest.mark.parametrize("M,N,slabs", [
    (1, 128, 32),      # one tile, K four ways
    (77, 136, 35),     # ragged N, unequal shares of K
    (128, 4736, 33),   # the most tiles that K is still split four ways for on 148 SMs
    (128, 4864, 17),   # two ways
    (100, 9472, 16),   # the most tiles with two ways
    (128, 9600, 16),   # 128-wide tiles, no split
    (64, 640, 9),      # too few slabs for a split
    (33, 18944, 3),    # the most 128-wide tiles
    (33, 19072, 3),    # 256-wide tiles
])
def test_gemm_of_few_rows_equals_the_256_wide_kernel(M, N, slabs, kind):
    """At most 128 rows: narrower tiles and K divided over a cluster. int8 sums are exact; in fp32 only the order of the sums
    differs, which moves at most the last bit of the bf16 result."""
    rng = np.random.default_rng(M + N + slabs)
    bias = dev((0.01 * rng.standard_normal(N)).astype(np.float32))
    if kind == "nvfp4":
        N = (N + 127) // 128 * 128
        K = slabs * 256 - 64  # the last slab is not full
        a = dev(rng.integers(0, 256, size=(M, K // 2), dtype=np.uint8))
        w = dev(rng.integers(0, 256, size=(N, K // 2), dtype=np.uint8))
        rows = (M + 127) // 128 * 128
        sa, sw = (dev(rng.integers(0x30, 0x40, size=n * K // 16, dtype=np.uint8)) for n in (rows, N))
        bias = dev((0.01 * rng.standard_normal(N)).astype(np.float32))
        run = lambda y, ep: sfq.lib.sfq_gemm_nvfp4(sfq.ptr(a), sfq.ptr(sa), sfq.ptr(w), sfq.ptr(sw), C.byref(ep), sfq.ptr(y), M, N, K, S)  # noqa: E731
        ep = sfq.Epilogue(None, None, 0.001, sfq.ptr(bias), sfq.F32, sfq.ACT_NONE)
    elif kind == "int8":
        K = slabs * 128 - 48
        a = dev(rng.integers(-128, 128, size=(M, K), dtype=np.int8))
        w = dev(rng.integers(-127, 128, size=(N, K), dtype=np.int8))
        rs, cs = dev((rng.random(M) * 0.05 + 1e-3).astype(np.float32)), dev((rng.random(N) * 0.01 + 1e-4).astype(np.float32))
        run = lambda y, ep: sfq.lib.sfq_gemm_int8(sfq.ptr(a), sfq.ptr(w), C.byref(ep), sfq.ptr(y), M, N, K, S)  # noqa: E731
        ep = sfq.Epilogue(sfq.ptr(rs), sfq.ptr(cs), 1.0, sfq.ptr(bias), sfq.F32, sfq.ACT_NONE)
    else:
        K = slabs * 64 - 8
        a = bf16_tensor(gaussian_bf16((M, K), seed=M))
        w = torch.randn((N, K), device="cuda", generator=torch.Generator("cuda").manual_seed(N)).mul_(0.02).to(torch.bfloat16)
        run = lambda y, ep: sfq.lib.sfq_gemm_bf16(sfq.ptr(a), sfq.ptr(w), C.byref(ep), sfq.ptr(y), M, N, K, S)  # noqa: E731
        ep = sfq.Epilogue(None, None, 1.0, sfq.ptr(bias), sfq.F32, sfq.ACT_NONE)
    got = []
    for tile_n in (0, 0, 256):
        y = torch.full((M, N), float("nan"), dtype=torch.bfloat16, device="cuda")
        sfq.lib.sfq_test_gemm_variant(tile_n, 0, 0)
        try:
            sfq.check(run(y, ep))
        finally:
            sfq.lib.sfq_test_gemm_variant(0, 0, 0)
        _status_clean()
        got.append(y)
    assert torch.equal(got[0], got[1])  # the order of the sums is fixed
    if kind == "int8":
        assert torch.equal(got[0], got[2])
    else:
        f, want = got[0].float(), got[2].float()
        # fp32 sums a few ulps apart, rounded to bf16 twice: the product (|product| <= |result| + |bias|) and the sum with the bias may
        # each land one bf16 step (2^-7 of the value at most) apart
        assert bool(((f - want).abs() <= 2.0 ** -7 * (2 * want.abs() + bias.abs()) + 1e-5 * want.abs().max()).all())


@pytest.mark.parametrize("M,N,K", [(77, 512, 8192), (128, 4864, 4096), (300, 512, 1024)])  # four ways, two ways, CTA pairs
def test_gemm_on_a_device_without_clusters(M, N, K):
    """Where clusters cannot be scheduled every plain GEMM runs as single CTAs: the bits are those of the one-CTA kernel."""
    rng = np.random.default_rng(M + N)
    a, w = dev(rng.integers(-128, 128, size=(M, K), dtype=np.int8)), dev(rng.integers(-127, 128, size=(N, K), dtype=np.int8))
    rs, cs = dev((rng.random(M) * 0.05 + 1e-3).astype(np.float32)), dev((rng.random(N) * 0.01 + 1e-4).astype(np.float32))
    x, v = bf16_tensor(gaussian_bf16((M, K), seed=M)), torch.randn((N, K), device="cuda").mul_(0.02).to(torch.bfloat16)
    ep8, ep16 = sfq.Epilogue(sfq.ptr(rs), sfq.ptr(cs), 1.0, None, sfq.F32, sfq.ACT_NONE), sfq.Epilogue(None, None, 1.0, None, sfq.F32, sfq.ACT_NONE)

    def run():
        y8, y16 = (torch.full((M, N), float("nan"), dtype=torch.bfloat16, device="cuda") for _ in range(2))
        sfq.check(sfq.lib.sfq_gemm_int8(sfq.ptr(a), sfq.ptr(w), C.byref(ep8), sfq.ptr(y8), M, N, K, S))
        sfq.check(sfq.lib.sfq_gemm_bf16(sfq.ptr(x), sfq.ptr(v), C.byref(ep16), sfq.ptr(y16), M, N, K, S))
        _status_clean()
        return y8, y16

    plain = run()
    sfq.lib.sfq_test_gemm_variant(128 if M <= 128 else 256, 0, 0)
    single = run()
    sfq.lib.sfq_test_gemm_variant(0, 0, 0)
    sfq.lib.sfq_test_gemm_no_clusters(1)
    try:
        alone = run()
        y = torch.empty((M, N // 2), dtype=torch.bfloat16, device="cuda")
        ep = sfq.Epilogue(sfq.ptr(rs), sfq.ptr(cs), 1.0, None, sfq.F32, sfq.ACT_SWIGLU)
        assert sfq.lib.sfq_gemm_int8(sfq.ptr(a), sfq.ptr(w), C.byref(ep), sfq.ptr(y), M, N, K, S) == sfq.ERR_RUNTIME  # needs pairs, as ever
    finally:
        sfq.lib.sfq_test_gemm_no_clusters(0)
    assert torch.equal(alone[0], plain[0]) and torch.equal(alone[0], single[0]) and torch.equal(alone[1], single[1])
    assert M > 128 or not torch.equal(alone[1], plain[1])  # with clusters the sums of few rows are divided: another order


def _nvfp4_case(M, N, K, seed):
    rng = np.random.default_rng(seed)
    w = (0.02 * rng.standard_normal((N, K))).astype(np.float32)
    data, scale, g = pack_nvfp4(w)
    x = gaussian_bf16((M, K), seed=seed + 1)
    return x, data, scale, g


def _run_nvfp4(x, data, scale, g, M, N, K, bias=None, act=sfq.ACT_NONE):
    dx = bf16_tensor(x)
    xq = torch.empty((M, K // 2), dtype=torch.uint8, device="cuda")
    xs = torch.empty(sfq.lib.sfq_nvfp4_act_scale_bytes(M, K), dtype=torch.uint8, device="cuda")
    sfq.check(sfq.lib.sfq_quantize_nvfp4_block(sfq.ptr(dx), None, sfq.ptr(xq), sfq.ptr(xs), None, M, K,
                                               sfq.NVFP4_ACT_GEMM_FEED, S))
    dd, ds = dev(data), dev(scale)
    y = torch.full((M, N), float("nan"), dtype=torch.bfloat16, device="cuda")
    db = dev(bias) if bias is not None else None
    ep = sfq.Epilogue(None, None, g, sfq.ptr(db), sfq.F32, act)
    sfq.check(sfq.lib.sfq_gemm_nvfp4(sfq.ptr(xq), sfq.ptr(xs), sfq.ptr(dd), sfq.ptr(ds), C.byref(ep), sfq.ptr(y),
                                     M, N, K, S))
    _status_clean()
    return y


@pytest.mark.parametrize("tile_n", [0, 256, 128])
@pytest.mark.parametrize("M,N,K", [(1, 128, 64), (17, 128, 128), (128, 256, 192), (200, 128, 320), (129, 256, 64),
                                   (256, 1024, 1024), (300, 384, 5120)])
def test_gemm_nvfp4_matches_fp4_activation_oracle(M, N, K, tile_n):
    # shapes of nvfp4_gemm_matches_cpu_reference (tests/test_nn_kernels_nvfp4_synthetic.cu:455-480) plus config 1
    x, data, scale, g = _nvfp4_case(M, N, K, seed=M + N + K)
    sfq.lib.sfq_test_gemm_variant(tile_n, 0, 0)
    try:
        y = _run_nvfp4(x, data, scale, g, M, N, K)
    finally:
        sfq.lib.sfq_test_gemm_variant(0, 0, 0)
    want = oracle.nvfp4_linear(x, data, scale, g, N, K)
    max_abs, rel_l2, corr = oracle.compare_bf16(want, bits(y))
    assert max_abs <= 2e-2 and rel_l2 <= 1e-3 and corr > 0.999, (max_abs, rel_l2, corr)
    # the reference's own bar for this comparison
    got, ref_ = oracle.from_bf16(bits(y)), oracle.from_bf16(want)
    assert np.all(np.abs(got - ref_) <= 1e-3 + 1e-2 * np.abs(ref_))


@pytest.mark.parametrize("act", [sfq.ACT_NONE, sfq.ACT_GELU_TANH, sfq.ACT_SWIGLU])
@pytest.mark.parametrize("M,N,K", [(1, 256, 64), (128, 256, 128), (129, 512, 320), (300, 384, 1024), (1000, 1280, 512), (4747, 2560, 256),
                                   (2600, 4992, 192)])
def test_gemm_nvfp4_quantized_result_equals_gemm_then_quantizer(M, N, K, act):
    """Codes and scales byte for byte, the zero scales of the padding rows included; bytes past the outputs stay as they were."""
    if act == sfq.ACT_SWIGLU and N % 256:
        N += 128
    g = torch.Generator("cuda").manual_seed(M + N + K)
    a = torch.randint(0, 256, (M, K // 2), dtype=torch.uint8, device="cuda", generator=g)
    w = torch.randint(0, 256, (N, K // 2), dtype=torch.uint8, device="cuda", generator=g)
    pad = (M + 127) // 128 * 128
    sa = torch.randint(0x30, 0x40, (pad * K // 16,), dtype=torch.uint8, device="cuda", generator=g)
    sw = torch.randint(0x30, 0x40, (N * K // 16,), dtype=torch.uint8, device="cuda", generator=g)
    bias = 0.01 * torch.randn(N, device="cuda", generator=g)
    cols = N // 2 if act == sfq.ACT_SWIGLU else N
    for db in (None, bias):
        ep = sfq.Epilogue(None, None, 0.002, sfq.ptr(db) if db is not None else None, sfq.F32, act)
        y = torch.empty((M, cols), dtype=torch.bfloat16, device="cuda")
        sfq.check(sfq.lib.sfq_gemm_nvfp4(sfq.ptr(a), sfq.ptr(sa), sfq.ptr(w), sfq.ptr(sw), C.byref(ep), sfq.ptr(y), M, N, K, S))
        want_q = torch.empty((M, cols // 2), dtype=torch.uint8, device="cuda")
        want_s = torch.empty(sfq.lib.sfq_nvfp4_act_scale_bytes(M, cols), dtype=torch.uint8, device="cuda")
        sfq.check(sfq.lib.sfq_quantize_nvfp4_block(sfq.ptr(y), None, sfq.ptr(want_q), sfq.ptr(want_s), None, M, cols, sfq.NVFP4_ACT_GEMM_FEED, S))
        got_q = torch.full((M * cols // 2 + 256,), 0xA5, dtype=torch.uint8, device="cuda")
        got_s = torch.full((want_s.numel() + 256,), 0xA5, dtype=torch.uint8, device="cuda")
        sfq.check(sfq.lib.sfq_gemm_nvfp4_quantized(sfq.ptr(a), sfq.ptr(sa), sfq.ptr(w), sfq.ptr(sw), C.byref(ep), sfq.ptr(got_q), sfq.ptr(got_s),
                                                   M, N, K, S))
        _status_clean()
        assert torch.equal(got_q[:-256].view(M, cols // 2), want_q) and torch.equal(got_s[:-256], want_s)
        assert bool((got_q[-256:] == 0xA5).all()) and bool((got_s[-256:] == 0xA5).all())


@pytest.mark.parametrize("M", [77, 300])
def test_gemm_nvfp4_quantized_result_on_a_device_without_clusters(M):
    """The result goes through bf16 scratch and the stand-alone quantizer there; eagerly and captured, and in a block, which used to
    run on such devices in its GELU form. SwiGLU is refused, as in the GEMM itself."""
    N, K = 512, 1024
    g = torch.Generator("cuda").manual_seed(M)
    x = torch.randn((M, K), device="cuda", generator=g).to(torch.bfloat16)
    data, scale, top = pack_nvfp4((0.02 * np.random.default_rng(1).standard_normal((N, K))).astype(np.float32))
    w, sw = dev(data), dev(scale)
    a = torch.empty((M, K // 2), dtype=torch.uint8, device="cuda")
    sa = torch.empty(sfq.lib.sfq_nvfp4_act_scale_bytes(M, K), dtype=torch.uint8, device="cuda")
    sfq.check(sfq.lib.sfq_quantize_nvfp4_block(sfq.ptr(x), None, sfq.ptr(a), sfq.ptr(sa), None, M, K, sfq.NVFP4_ACT_GEMM_FEED, S))
    q = torch.zeros((M, N // 2), dtype=torch.uint8, device="cuda")
    s = torch.zeros(sfq.lib.sfq_nvfp4_act_scale_bytes(M, N), dtype=torch.uint8, device="cuda")
    ep = lambda act: sfq.Epilogue(None, None, top, None, sfq.F32, act)  # noqa: E731
    run = lambda act: sfq.lib.sfq_gemm_nvfp4_quantized(sfq.ptr(a), sfq.ptr(sa), sfq.ptr(w), sfq.ptr(sw), C.byref(ep(act)), sfq.ptr(q), sfq.ptr(s),  # noqa: E731
                                                       M, N, K, sfq.stream_ptr())
    hidden, heads, ffn = 1024, 8, 2048
    lin = lambda n, k: Nvfp4Linear(*(dev(t) for t in pack_nvfp4((0.02 * np.random.default_rng(n).standard_normal((n, k))).astype(np.float32))[:2]), 1e-5, n, k)  # noqa: E731
    ones = torch.ones(hidden, dtype=torch.bfloat16, device="cuda")
    weights = BlockWeights(lin(3 * hidden, hidden), lin(hidden, hidden), lin(ffn, hidden), lin(hidden, ffn), ones, ones)
    mod = {name: 0.1 * torch.randn((3, hidden), device="cuda", generator=g) for name in ("scale_msa", "shift_msa", "gate_msa", "scale_mlp", "shift_mlp", "gate_mlp")}
    index = torch.zeros(M, dtype=torch.int32, device="cuda")
    block = Nvfp4Block(M, hidden, heads, ffn)
    want_x = block.forward(x.clone(), weights, mod, index)
    sfq.lib.sfq_test_gemm_no_clusters(1)
    try:
        for act in (sfq.ACT_NONE, sfq.ACT_GELU_TANH):
            y = torch.empty((M, N), dtype=torch.bfloat16, device="cuda")
            sfq.check(sfq.lib.sfq_gemm_nvfp4(sfq.ptr(a), sfq.ptr(sa), sfq.ptr(w), sfq.ptr(sw), C.byref(ep(act)), sfq.ptr(y), M, N, K, S))
            want_q, want_s = torch.empty_like(q), torch.empty_like(s)
            sfq.check(sfq.lib.sfq_quantize_nvfp4_block(sfq.ptr(y), None, sfq.ptr(want_q), sfq.ptr(want_s), None, M, N, sfq.NVFP4_ACT_GEMM_FEED, S))
            sfq.check(run(act))
            assert torch.equal(q, want_q) and torch.equal(s, want_s)
            graph = torch.cuda.CUDAGraph()
            torch.cuda.synchronize()
            with torch.cuda.graph(graph):
                sfq.check(run(act))
            q.zero_(), s.zero_()
            for _ in range(2):
                graph.replay()
            torch.cuda.synchronize()
            assert torch.equal(q, want_q) and torch.equal(s, want_s)
        assert run(sfq.ACT_SWIGLU) == sfq.ERR_RUNTIME
        got_x = block.forward(x.clone(), weights, mod, index)
    finally:
        sfq.lib.sfq_test_gemm_no_clusters(0)
    # another order of fp32 sums at most, i.e. a last bf16 bit here and there that the fp4 codes behind it amplify
    assert float((got_x.float() - want_x.float()).norm() / want_x.float().norm()) < 2e-2
    _status_clean()


def test_gemm_nvfp4_quantized_refusals():
    z = torch.zeros(1 << 16, dtype=torch.uint8, device="cuda")
    o = torch.zeros(1 << 16, dtype=torch.uint8, device="cuda")
    f = torch.zeros(256, dtype=torch.float32, device="cuda")
    run = lambda ep, q, s: sfq.lib.sfq_gemm_nvfp4_quantized(sfq.ptr(z), sfq.ptr(z), sfq.ptr(z), sfq.ptr(z), C.byref(ep), q, s, 128, 256, 64, S)  # noqa: E731
    plain = sfq.Epilogue(None, None, 1.0, None, sfq.F32, sfq.ACT_NONE)
    assert run(plain, None, sfq.ptr(o)) != 0 and run(plain, sfq.ptr(o), None) != 0
    assert run(plain, sfq.ptr(z), sfq.ptr(o)) != 0  # over its own operand
    assert run(plain, sfq.ptr(o) + 8, sfq.ptr(o)) != 0
    assert run(sfq.Epilogue(None, None, 1.0, None, sfq.F32, sfq.ACT_NONE, sfq.ptr(f), sfq.ptr(f)), sfq.ptr(o), sfq.ptr(o)) != 0


@pytest.mark.parametrize("tile_n", [0, 256])
@pytest.mark.parametrize("M,N,K", [(300, 512, 256), (129, 34, 256), (1000, 1280, 512)])
def test_gemm_gated_residual_epilogue(M, N, K, tile_n):
    # x += gate[a[r]] * (q w^T scaled + bias) in the epilogue == the plain GEMM followed by add_gated
    # (src/cuda/nn_pointwise.cu:16-37), bit for bit, on the vectorised and the ragged store paths
    rng = np.random.default_rng(M + N)
    a = rng.integers(-128, 128, size=(M, K), dtype=np.int8)
    w = rng.integers(-127, 128, size=(N, K), dtype=np.int8)
    rs = (rng.random(M, dtype=np.float32) * 0.05 + 1e-3).astype(np.float32)
    cs = (rng.random(N, dtype=np.float32) * 0.01 + 1e-4).astype(np.float32)
    bias = (0.01 * rng.standard_normal(N)).astype(np.float32)
    gate = (0.5 * rng.standard_normal((5, N))).astype(np.float32)
    idx = rng.integers(0, 5, size=M).astype(np.int32)
    x = gaussian_bf16((M, N), seed=M)
    da, dw, drs, dcs, db, dg, di = dev(a), dev(w), dev(rs), dev(cs), dev(bias), dev(gate), dev(idx)
    sfq.lib.sfq_test_gemm_variant(tile_n, 0, 0)
    try:
        branch = torch.empty((M, N), dtype=torch.bfloat16, device="cuda")
        ep = sfq.Epilogue(sfq.ptr(drs), sfq.ptr(dcs), 1.0, sfq.ptr(db), sfq.F32, sfq.ACT_NONE)
        sfq.check(sfq.lib.sfq_gemm_int8(sfq.ptr(da), sfq.ptr(dw), C.byref(ep), sfq.ptr(branch), M, N, K, S))
        y = bf16_tensor(x)
        ep2 = sfq.Epilogue(sfq.ptr(drs), sfq.ptr(dcs), 1.0, sfq.ptr(db), sfq.F32, sfq.ACT_NONE, sfq.ptr(dg), sfq.ptr(di))
        sfq.check(sfq.lib.sfq_gemm_int8(sfq.ptr(da), sfq.ptr(dw), C.byref(ep2), sfq.ptr(y), M, N, K, S))
        _status_clean()
    finally:
        sfq.lib.sfq_test_gemm_variant(0, 0, 0)
    want = x.copy()
    bb = bits(branch)
    oracle.lib.orc_add_gated_bf16(P(want), P(bb), P(gate), P(idx), M, N)
    assert np.array_equal(bits(y), want)
    # a gate without its index (or the other way round) is refused
    bad = sfq.Epilogue(sfq.ptr(drs), sfq.ptr(dcs), 1.0, None, sfq.F32, sfq.ACT_NONE, sfq.ptr(dg), None)
    assert sfq.lib.sfq_gemm_int8(sfq.ptr(da), sfq.ptr(dw), C.byref(bad), sfq.ptr(y), M, N, K, S) == sfq.ERR_INVALID_ARGUMENT


@pytest.mark.parametrize("kind", ["int8", "nvfp4"])
@pytest.mark.parametrize("M,N,K,bias", [(200, 512, 256, True), (1, 256, 128, False), (700, 1536, 512, True)])
def test_gemm_swiglu_epilogue(kind, M, N, K, bias):
    # weight rows [gate | up]: the fused epilogue equals the plain GEMM followed by swiglu_kernel
    # (src/cuda/nn_pointwise.cu:44-64), bit for bit
    rng = np.random.default_rng(M + N + K)
    b = (0.05 * rng.standard_normal(N)).astype(np.float32)
    db = dev(b)
    if kind == "int8":
        a = rng.integers(-128, 128, size=(M, K), dtype=np.int8)
        w = rng.integers(-127, 128, size=(N, K), dtype=np.int8)
        rs = (rng.random(M, dtype=np.float32) * 0.02 + 1e-3).astype(np.float32)
        cs = (rng.random(N, dtype=np.float32) * 0.01 + 1e-4).astype(np.float32)
        keep = [dev(a), dev(w), dev(rs), dev(cs)]

        def run(act, y):
            ep = sfq.Epilogue(sfq.ptr(keep[2]), sfq.ptr(keep[3]), 1.0, sfq.ptr(db) if bias else None, sfq.F32, act)
            return sfq.lib.sfq_gemm_int8(sfq.ptr(keep[0]), sfq.ptr(keep[1]), C.byref(ep), sfq.ptr(y), M, N, K, S)
    else:
        x, data, scale, g = _nvfp4_case(M, N, K, seed=M + 3)
        dx = bf16_tensor(x)
        xq = torch.empty((M, K // 2), dtype=torch.uint8, device="cuda")
        xs = torch.empty(sfq.lib.sfq_nvfp4_act_scale_bytes(M, K), dtype=torch.uint8, device="cuda")
        sfq.check(sfq.lib.sfq_quantize_nvfp4_block(sfq.ptr(dx), None, sfq.ptr(xq), sfq.ptr(xs), None, M, K,
                                                   sfq.NVFP4_ACT_GEMM_FEED, S))
        keep = [dev(data), dev(scale)]

        def run(act, y):
            ep = sfq.Epilogue(None, None, g, sfq.ptr(db) if bias else None, sfq.F32, act)
            return sfq.lib.sfq_gemm_nvfp4(sfq.ptr(xq), sfq.ptr(xs), sfq.ptr(keep[0]), sfq.ptr(keep[1]), C.byref(ep), sfq.ptr(y),
                                          M, N, K, S)
    fused_in = torch.empty((M, N), dtype=torch.bfloat16, device="cuda")
    sfq.check(run(sfq.ACT_NONE, fused_in))
    want = torch.empty((M, N // 2), dtype=torch.bfloat16, device="cuda")
    sfq.check(sfq.lib.sfq_swiglu(sfq.ptr(fused_in), sfq.ptr(want), M, N // 2, S))
    got = torch.full((M, N // 2), float("nan"), dtype=torch.bfloat16, device="cuda")
    sfq.check(run(sfq.ACT_SWIGLU, got))
    _status_clean()
    assert np.array_equal(bits(got), bits(want))


def test_gemm_swiglu_contract():
    y = torch.empty((4, 64), dtype=torch.bfloat16, device="cuda")
    a = torch.zeros((4, 64), dtype=torch.int8, device="cuda")
    w = torch.zeros((128, 64), dtype=torch.int8, device="cuda")  # N = 128 is not a multiple of 256
    s = torch.ones(128, device="cuda")
    ep = sfq.Epilogue(sfq.ptr(s), sfq.ptr(s), 1.0, None, sfq.F32, sfq.ACT_SWIGLU)
    assert sfq.lib.sfq_gemm_int8(sfq.ptr(a), sfq.ptr(w), C.byref(ep), sfq.ptr(y), 4, 128, 64, S) == sfq.ERR_INVALID_ARGUMENT


def test_gemm_nvfp4_multi_tile_persistence():
    # more 256x256 tiles than CTA pairs, ragged M, ragged last K stage: every pair walks several tiles through the one
    # accumulator and wraps the stage ring (and its scale slots) many times
    M, N, K = 256 * 41 - 24, 2048, 448
    x, data, scale, g = _nvfp4_case(M, N, K, seed=11)
    y = _run_nvfp4(x, data, scale, g, M, N, K)
    want = oracle.nvfp4_linear(x, data, scale, g, N, K)
    max_abs, rel_l2, corr = oracle.compare_bf16(want, bits(y))
    assert max_abs <= 2e-2 and rel_l2 <= 1e-3 and corr > 0.999, (max_abs, rel_l2, corr)


def test_gemm_nvfp4_wrong_layouts_are_far_away():
    # nvfp4_gemm_disk_layout (tests/test_nn_kernels_nvfp4_synthetic.cu:482-520): each plausible wrong form of
    # the stored weight must give rms_rel > 0.2 against the right answer, or the match above proves nothing.
    M, N, K = 64, 256, 512
    x, data, scale, g = _nvfp4_case(M, N, K, seed=99)
    right = oracle.from_bf16(bits(_run_nvfp4(x, data, scale, g, M, N, K)))
    swapped = ((data << 4) | (data >> 4)).astype(np.uint8)
    plain = np.zeros_like(scale)
    kb = K // 16
    for r in range(N):
        for b in range(kb):
            plain[r * kb + b] = scale[oracle.lib.orc_nvfp4_scale_slot(r, b, kb)]
    for name, d, s in (("nibbles swapped", swapped, scale), ("row-major scales", data, plain)):
        wrong = oracle.from_bf16(bits(_run_nvfp4(x, d, s, g, M, N, K)))
        rms = np.sqrt(((wrong - right) ** 2).sum() / (right ** 2).sum())
        assert rms > 0.2, (name, rms)
    # the global scale is applied exactly once (nvfp4_gemm_global_scale)
    doubled = oracle.from_bf16(bits(_run_nvfp4(x, data, scale, 2 * g, M, N, K)))
    assert np.allclose(doubled, 2 * right, rtol=2 ** -7, atol=1e-6)


def test_gemm_nvfp4_exact_grid_activations():
    # nvfp4_gemm_exact_fp4_activations: inputs already on the fp4 grid with unit scales make every product
    # exact, so the result must equal the integer-valued dot product.
    M, N, K = 128, 128, 256
    rng = np.random.default_rng(3)
    grid = np.array([0, .5, 1, 1.5, 2, 3, 4, 6, -.5, -1, -1.5, -2, -3, -4, -6], np.float32)
    x = grid[rng.integers(0, len(grid), size=(M, K))]
    x[:, ::16] = 6.0  # pins every block's amax to 6 -> scale 1.0
    w = grid[rng.integers(0, len(grid), size=(N, K))]
    w[:, ::16] = 6.0
    data = np.zeros((N, K // 2), np.uint8)
    scale = np.zeros(N * K // 16, np.uint8)
    sfq.check(sfq.lib.sfq_pack_nvfp4(P(w), N, K, 1.0, P(data), P(scale)))
    y = _run_nvfp4(oracle.to_bf16(x), data, scale, 1.0, M, N, K)
    want = torch.from_numpy(x.astype(np.float64) @ w.astype(np.float64).T).to(torch.bfloat16)
    assert torch.equal(y.cpu(), want)


def test_nvfp4_config1_bias_and_distance_to_dequantize_path():
    # benchmark config 1: M=256, K=N=1024, bias ~ N(0, 0.01), seed 0
    M, N, K = 256, 1024, 1024
    rng = np.random.default_rng(0)
    x = oracle.to_bf16(rng.standard_normal((M, K)).astype(np.float32))
    w = (0.02 * rng.standard_normal((N, K))).astype(np.float32)
    bias = (0.01 * rng.standard_normal(N)).astype(np.float32)
    data, scale, g = pack_nvfp4(w)
    y = _run_nvfp4(x, data, scale, g, M, N, K, bias=bias)
    want = oracle.nvfp4_linear(x, data, scale, g, N, K, bias=bias)
    max_abs, rel_l2, corr = oracle.compare_bf16(want, bits(y))
    assert max_abs <= 2e-2 and rel_l2 <= 1e-3, (max_abs, rel_l2)
    # against the bf16-activation (dequantize-then-GEMM) result the fp4 activation costs about 9 % rms
    # with correlation ~0.995 (src/cuda/nvfp4_gemm.cu:41-45): reported by the reference, checked loosely here
    dq = oracle.nvfp4_linear_dequant(x, data, scale, g, N, K, bias=bias)
    _, rel_a, corr_a = oracle.compare_bf16(dq, bits(y))
    assert 0.04 < rel_a < 0.16 and corr_a > 0.98, (rel_a, corr_a)
