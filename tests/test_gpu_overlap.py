"""Kernels that may start before the one in front of them has finished: each waits for it before it touches what it writes.

The kernel in front is one of the library's own that lets its successor start at once, runs for some tens of microseconds and
writes the operand under test last: a rotation of a large matrix whose last rows are that operand. Every operand that a kernel
reads is put there once, the tables and weights as well as the activation, holding stale values until the rotation overwrites
them. The answer has to be that of the same two calls with a synchronisation between them.
"""
import ctypes as C

import numpy as np
import pytest
import torch

import slopfab_b200 as sfq
from helpers import pack_nvfp4, synthetic_packed_int8
from slopfab_b200.block import BlockWeights, Nvfp4Block, Nvfp4Linear

pytestmark = pytest.mark.gpu
lib, ptr = sfq.lib, sfq.ptr
ROWS, DIM = 4096, 5120  # 84 MB: below the size from which launches are plain


class Front:
    """`tail` is the operand: the last bytes of the rotation's result (bf16 values, or zeros for tables of fp32 / int32)."""

    def __init__(self, nbytes, zeros=False, offset=0, rows=ROWS):
        g = torch.Generator("cuda").manual_seed(nbytes + offset)
        self.rows = rows
        self.x = torch.randn((rows, DIM), device="cuda", generator=g).to(torch.bfloat16)
        lines = -(-(nbytes + 64) // (2 * DIM))
        assert lines < rows // 2
        if zeros:
            self.x[rows - lines:] = 0
        self.out = torch.empty_like(self.x)
        flat = self.out.view(-1).view(torch.uint8)
        start = flat.numel() - lines * 2 * DIM + offset
        self.tail = flat[start:start + nbytes]

    def view(self, dtype, *shape):
        return self.tail.view(dtype).view(*shape)

    def launch(self):
        sfq.check(lib.sfq_convrot(ptr(self.x), ptr(self.out), self.rows, DIM, 256, sfq.stream_ptr()))


def agrees(front, stale, call, repeats=8):
    """call() -> tensors; the same behind the front kernel, with and without a synchronisation between."""
    def fill():
        front.tail.copy_(stale)
        torch.cuda.synchronize()

    fill()
    old = [t.clone() for t in call()]
    fill()
    front.launch()
    torch.cuda.synchronize()
    want = [t.clone() for t in call()]
    assert any(not torch.equal(a.view(torch.uint8), b.view(torch.uint8)) for a, b in zip(old, want)), "the operand does not matter"
    for _ in range(repeats):
        fill()
        front.launch()
        for a, b in zip(want, call()):
            assert torch.equal(a.view(torch.uint8), b.view(torch.uint8))
    assert sfq.device_status() == 0


def random_bytes(front, like):
    g = torch.Generator("cuda").manual_seed(3)
    return torch.randn(front.tail.numel() // 2, device="cuda", generator=g).to(torch.bfloat16).view(torch.uint8) if like == "bf16" else \
        torch.ones(front.tail.numel() // 4, device="cuda", dtype=like).view(torch.uint8)


def bf16(shape, seed, scale=1.0):
    return (scale * torch.randn(shape, device="cuda", generator=torch.Generator("cuda").manual_seed(seed))).to(torch.bfloat16)


@pytest.mark.parametrize("rows,dim", [(64, 5120), (400, 5120), (200, 7168)])
@pytest.mark.parametrize("operand", ["x", "weight", "scale", "shift", "index"])
@pytest.mark.parametrize("kind", ["norm", "fp4", "int8"])
def test_norms(kind, operand, rows, dim):
    sizes = {"x": 2 * rows * dim, "weight": 2 * dim, "scale": 12 * dim, "shift": 12 * dim, "index": 4 * rows}
    front = Front(sizes[operand], zeros=operand in ("scale", "shift", "index"))
    t = {"x": bf16((rows, dim), 1), "weight": bf16((dim,), 2), "scale": bf16((3, dim), 3).float(), "shift": bf16((3, dim), 4).float(),
         "index": torch.arange(rows, device="cuda", dtype=torch.int32) % 3}
    dtype = {"x": "bf16", "weight": "bf16", "scale": torch.float32, "shift": torch.float32, "index": torch.int32}[operand]
    t[operand] = front.view(torch.bfloat16 if dtype == "bf16" else dtype, *t[operand].shape)
    norm = sfq.Norm(ptr(t["weight"]), ptr(t["scale"]), ptr(t["shift"]), ptr(t["index"]), 1e-5)
    out = torch.empty((rows, dim), dtype=torch.bfloat16, device="cuda")
    q = torch.empty((rows, dim), dtype=torch.uint8, device="cuda")
    s = torch.zeros(lib.sfq_nvfp4_act_scale_bytes(rows, dim), dtype=torch.uint8, device="cuda")
    rs = torch.zeros(rows, device="cuda")

    def call():
        if kind == "norm":
            sfq.check(lib.sfq_rmsnorm(ptr(t["x"]), C.byref(norm), ptr(out), rows, dim, sfq.stream_ptr()))
            return [out]
        if kind == "fp4":
            sfq.check(lib.sfq_quantize_nvfp4_block(ptr(t["x"]), C.byref(norm), ptr(q), ptr(s), None, rows, dim, sfq.NVFP4_ACT_GEMM_FEED, sfq.stream_ptr()))
            return [q.view(-1)[:rows * dim // 2], s]
        sfq.check(lib.sfq_quantize_int8_token(ptr(t["x"]), C.byref(norm), ptr(q), ptr(rs), None, rows, dim, 1, sfq.stream_ptr()))
        return [q, rs]

    agrees(front, random_bytes(front, dtype), call)


@pytest.mark.parametrize("rows,dim,kind", [(300, 5120, "fp4"), (301, 5120, "int8"), (200, 13824, "int8"), (150, 6400, "int8"), (77, 5120, "rot"), (300, 5120, "rot")])
def test_quantizers(rows, dim, kind):
    front = Front(2 * rows * dim)
    x = front.view(torch.bfloat16, rows, dim)
    q = torch.empty((rows, 2 * dim), dtype=torch.uint8, device="cuda")
    s = torch.zeros(lib.sfq_nvfp4_act_scale_bytes(rows, dim), dtype=torch.uint8, device="cuda")
    rs = torch.zeros(rows, device="cuda")

    def call():
        if kind == "fp4":
            sfq.check(lib.sfq_quantize_nvfp4_block(ptr(x), None, ptr(q), ptr(s), None, rows, dim, sfq.NVFP4_ACT_GEMM_FEED, sfq.stream_ptr()))
            return [q.view(-1)[:rows * dim // 2], s]
        if kind == "rot":
            sfq.check(lib.sfq_convrot(ptr(x), ptr(q), rows, dim, 256, sfq.stream_ptr()))
            return [q]
        sfq.check(lib.sfq_quantize_int8_token(ptr(x), None, ptr(q), ptr(rs), None, rows, dim, 1, sfq.stream_ptr()))
        return [q.view(-1)[:rows * dim], rs]

    agrees(front, random_bytes(front, "bf16"), call)


@pytest.mark.parametrize("operand", ["x", "weight", "cos", "sin"])
def test_head_norm_and_rope(operand):
    rows, heads = 300, 12
    sizes = {"x": 256 * rows * heads, "weight": 256, "cos": 384 * rows, "sin": 384 * rows}
    front = Front(sizes[operand], zeros=operand in ("cos", "sin"))
    t = {"x": bf16((rows, heads * 128), 1), "weight": bf16((128,), 2), "cos": bf16((rows, 96), 3).float(), "sin": bf16((rows, 96), 4).float()}
    dtype = "bf16" if operand in ("x", "weight") else torch.float32
    t[operand] = front.view(torch.bfloat16 if dtype == "bf16" else dtype, *t[operand].shape)
    source = t["x"].clone()

    def call():
        if operand != "x":
            t["x"].copy_(source)
            torch.cuda.synchronize()
            front.tail.copy_(stale)
            torch.cuda.synchronize()
            if call.fresh:
                front.launch()
        sfq.check(lib.sfq_head_norm_rope(ptr(t["x"]), heads * 128, ptr(t["weight"]), ptr(t["cos"]), ptr(t["sin"]), rows, heads, 128, 1e-6, sfq.stream_ptr()))
        return [t["x"]]

    stale = random_bytes(front, dtype)
    if operand == "x":
        agrees(front, stale, call)
        return
    call.fresh = False  # the kernel works in place, so its own input is put back in front of the front kernel
    old = call()[0].clone()
    call.fresh = True
    got = [call()[0].clone() for _ in range(8)]
    t["x"].copy_(source)
    torch.cuda.synchronize()
    sfq.check(lib.sfq_head_norm_rope(ptr(t["x"]), heads * 128, ptr(t["weight"]), ptr(t["cos"]), ptr(t["sin"]), rows, heads, 128, 1e-6, sfq.stream_ptr()))
    assert not torch.equal(old, t["x"]) and all(torch.equal(g, t["x"]) for g in got)


@pytest.mark.parametrize("rows", [300, 1500])  # launched overlapped and plainly
@pytest.mark.parametrize("operand", ["x", "branch", "gate", "index"])
def test_gated_residual(operand, rows):
    dim = 5120
    sizes = {"x": 2 * rows * dim, "branch": 2 * rows * dim, "gate": 12 * dim, "index": 4 * rows}
    front = Front(sizes[operand], zeros=operand in ("gate", "index"))
    t = {"x": bf16((rows, dim), 1), "branch": bf16((rows, dim), 2), "gate": bf16((3, dim), 3).float(),
         "index": torch.arange(rows, device="cuda", dtype=torch.int32) % 3}
    dtype = {"x": "bf16", "branch": "bf16", "gate": torch.float32, "index": torch.int32}[operand]
    t[operand] = front.view(torch.bfloat16 if dtype == "bf16" else dtype, *t[operand].shape)
    source = t["x"].clone()

    def call():
        sfq.check(lib.sfq_add_gated(ptr(t["x"]), ptr(t["branch"]), ptr(t["gate"]), ptr(t["index"]), rows, dim, sfq.stream_ptr()))
        out = t["x"].clone()
        if operand != "x":
            t["x"].copy_(source)  # the kernel works in place
        return [out]

    agrees(front, random_bytes(front, dtype), call)


@pytest.mark.parametrize("operand,offset", [("q", 0), ("k", 0), ("v", 0), ("v", 6)])
@pytest.mark.parametrize("seq,heads", [(300, 4), (513, 40)])
def test_attention(operand, offset, seq, heads):
    front = Front(256 * seq * heads, offset=offset)
    t = {n: bf16((seq, heads * 128), i) for i, n in enumerate("qkv")}
    t[operand] = front.view(torch.bfloat16, seq, heads * 128)
    out = torch.empty((seq, heads * 128), dtype=torch.bfloat16, device="cuda")
    n = C.c_size_t()
    sfq.check(lib.sfq_attention_workspace_bytes(seq, heads, 128, C.byref(n)))
    ws = torch.empty(n.value, dtype=torch.uint8, device="cuda")

    def call():
        sfq.check(lib.sfq_attention_forward(t["q"].data_ptr(), heads * 128, t["k"].data_ptr(), t["v"].data_ptr(), heads * 128, ptr(out), heads * 128,
                                            seq, seq, heads, heads, 128, 0.0, ptr(ws), n.value, sfq.stream_ptr()))
        return [out]

    agrees(front, random_bytes(front, "bf16"), call)


@pytest.mark.parametrize("operand", ["x", "bias", "row_scale", "col_scale", "gate", "gate_index"])
@pytest.mark.parametrize("rows", [77, 300])  # K divided over a cluster; CTA pairs
def test_gemm_operands(operand, rows):
    """Everything a GEMM reads but its weight: int8 for the scales, bf16 for the rest."""
    n, k = 512, 4096
    int8 = operand in ("row_scale", "col_scale")
    sizes = {"x": 2 * rows * k, "bias": 4 * n, "row_scale": 4 * rows, "col_scale": 4 * n, "gate": 12 * n, "gate_index": 4 * rows}
    front = Front(sizes[operand], zeros=operand != "x")
    t = {"x": bf16((rows, k), 1), "bias": bf16((n,), 2).float(), "row_scale": torch.rand(rows, device="cuda"), "col_scale": torch.rand(n, device="cuda"),
         "gate": bf16((3, n), 3).float(), "gate_index": torch.arange(rows, device="cuda", dtype=torch.int32) % 3}
    dtype = "bf16" if operand == "x" else (torch.int32 if operand == "gate_index" else torch.float32)
    t[operand] = front.view(torch.bfloat16 if dtype == "bf16" else dtype, *t[operand].shape)
    w = bf16((n, k), 5, 0.02)
    a8 = torch.randint(-127, 128, (rows, k), device="cuda", dtype=torch.int8)
    w8 = torch.randint(-127, 128, (n, k), device="cuda", dtype=torch.int8)
    gated = operand.startswith("gate")
    y = torch.zeros((rows, n), dtype=torch.bfloat16, device="cuda")
    ep = sfq.Epilogue(ptr(t["row_scale"]), ptr(t["col_scale"]), 1.0, ptr(t["bias"]), sfq.F32, sfq.ACT_NONE, ptr(t["gate"]) if gated else None,
                      ptr(t["gate_index"]) if gated else None)

    def call():
        if int8:
            sfq.check(lib.sfq_gemm_int8(ptr(a8), ptr(w8), C.byref(ep), ptr(y), rows, n, k, sfq.stream_ptr()))
        else:
            sfq.check(lib.sfq_gemm_bf16(ptr(t["x"]), ptr(w), C.byref(ep), ptr(y), rows, n, k, sfq.stream_ptr()))
        out = y.clone()
        y.zero_()  # the gated form adds
        return [out]

    agrees(front, random_bytes(front, dtype), call)


def weight(fmt, n, k):
    rng = np.random.default_rng(n + k)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    if fmt == "nvfp4":
        data, scale, g = pack_nvfp4((0.02 * rng.standard_normal((n, k))).astype(np.float32))
        keep = dict(data=dev(data), block_scale=dev(scale))
        return sfq.new_weight(format=sfq.NVFP4, out_features=n, in_features=k, global_scale=g, **{a: ptr(b) for a, b in keep.items()}), keep
    if fmt in ("w4a8", "w6a8"):
        bits_, group = (4, 16) if fmt == "w4a8" else (6, 64)
        packed, s_rel, s_ch, book = synthetic_packed_int8(bits_, group, n, k, seed=3)
        keep = dict(data=dev(packed), block_scale=dev(s_rel), weight_scale=dev(s_ch))
        if book is not None:
            keep["w4_codebook"] = dev(book)
        return sfq.new_weight(format=sfq.W4A8 if fmt == "w4a8" else sfq.W6A8, out_features=n, in_features=k, packed_group_size=group, convrot=1,
                              convrot_group=256, **{a: ptr(b) for a, b in keep.items()}), keep
    if fmt == "i8":
        keep = dict(data=dev(rng.integers(-127, 128, (n, k), dtype=np.int8)), weight_scale=dev(rng.random(n).astype(np.float32) * 0.01))
        return sfq.new_weight(format=sfq.I8, out_features=n, in_features=k, per_channel_scale=1, convrot=1, convrot_group=256,
                              **{a: ptr(b) for a, b in keep.items()}), keep
    keep = dict(data=bf16((n, k), 4, 0.02))
    return sfq.new_weight(format=sfq.BF16, out_features=n, in_features=k, data=ptr(keep["data"])), keep


LINEARS = [("nvfp4", 77, 512, 5120, True), ("nvfp4", 300, 1024, 5120, True), ("nvfp4", 300, 1024, 5120, False), ("w4a8", 300, 1024, 5120, True),
           ("w4a8", 300, 2048, 5120, True),  # decoded on the side stream
           ("w6a8", 77, 512, 5120, True), ("i8", 333, 4096, 4096, True),  # the rotation beside the unpacker
           ("bf16", 100, 512, 5120, True)]


@pytest.mark.parametrize("fmt,rows,n,k,native", LINEARS)
def test_linear_layers(fmt, rows, n, k, native):
    front = Front(2 * rows * k)
    x = front.view(torch.bfloat16, rows, k)
    w, keep = weight(fmt, n, k)
    runner = sfq.LinearRunner()
    runner.set_native(native)
    agrees(front, random_bytes(front, "bf16"), lambda: [runner.forward(w, x)])


def test_a_chain_with_overlapped_and_plain_launches():
    """Rows around the size from which a launch is a plain one: both kinds follow each other in one Linear."""
    k, n = 5120, 512
    w, keep = weight("nvfp4", n, k)
    runner = sfq.LinearRunner()
    runner.set_native(True)
    for rows in (4900, 5000, 6500, 6600):  # the rotation in front and the quantizer, either side of 96 MB
        x = bf16((rows, k), rows)
        rotated = torch.zeros_like(x)
        sfq.check(lib.sfq_convrot(ptr(x), ptr(rotated), rows, k, 256, sfq.stream_ptr()))
        torch.cuda.synchronize()
        want = runner.forward(w, rotated).clone()
        for _ in range(5):
            rotated.zero_()
            torch.cuda.synchronize()
            sfq.check(lib.sfq_convrot(ptr(x), ptr(rotated), rows, k, 256, sfq.stream_ptr()))
            assert torch.equal(runner.forward(w, rotated), want)


@pytest.mark.parametrize("fmt,rows,n,k,native", LINEARS)
def test_captured_and_behind_another_stream(fmt, rows, n, k, native):
    """The front kernel on the same stream and on another one, eagerly and as a graph that is replayed with new inputs."""
    front = Front(2 * rows * k)
    x = front.view(torch.bfloat16, rows, k)
    w, keep = weight(fmt, n, k)
    side, main = torch.cuda.Stream(), torch.cuda.Stream()
    runner = sfq.LinearRunner(main)
    runner.set_native(native)
    source = front.x.clone()
    y = torch.empty((rows, n), dtype=torch.bfloat16, device="cuda")
    want = {}
    for factor in (1, -2):
        front.x.copy_(source).mul_(factor)
        front.launch()
        torch.cuda.synchronize()
        runner.forward(w, x, y)
        torch.cuda.synchronize()
        want[factor] = y.clone()

    def body(other):
        if other:
            side.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(side):
                front.launch()
            sfq.check(lib.sfq_rmsnorm(ptr(front.x), C.byref(norm), ptr(scrap), 64, DIM, sfq.stream_ptr()))  # a kernel of this stream before the join
            torch.cuda.current_stream().wait_stream(side)
        else:
            front.launch()
        return runner.forward(w, x, y)

    ones = torch.ones(DIM, dtype=torch.bfloat16, device="cuda")
    norm = sfq.Norm(ptr(ones), None, None, None, 1e-5)
    scrap = torch.empty((64, DIM), dtype=torch.bfloat16, device="cuda")
    torch.cuda.synchronize()
    for other in (False, True):
        with torch.cuda.stream(main):
            for factor in (1, -2):
                front.x.copy_(source).mul_(factor)
                front.tail.zero_()
                main.synchronize()
                body(other)
                main.synchronize()
                assert torch.equal(y, want[factor])
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=main):
            body(other)
        for factor in (1, -2, 1):
            front.x.copy_(source).mul_(factor)
            front.tail.zero_()
            y.zero_()
            torch.cuda.synchronize()
            graph.replay()
            torch.cuda.synchronize()
            assert torch.equal(y, want[factor])
    assert sfq.device_status() == 0


def test_a_block_behind_the_kernel_that_writes_its_input():
    rows, heads, ffn = 300, 8, 2048
    hidden = heads * 128
    front = Front(2 * rows * hidden)
    x = front.view(torch.bfloat16, rows, hidden)

    def linear(n, k):
        data, scale, g = pack_nvfp4((0.02 * np.random.default_rng(n).standard_normal((n, k))).astype(np.float32))
        return Nvfp4Linear(torch.from_numpy(data).cuda(), torch.from_numpy(scale).cuda(), g, n, k)

    ones = torch.ones(hidden, dtype=torch.bfloat16, device="cuda")
    w = BlockWeights(linear(3 * hidden, hidden), linear(hidden, hidden), linear(ffn, hidden), linear(hidden, ffn), ones, ones, bf16((128,), 1), bf16((128,), 2))
    mod = {name: bf16((3, hidden), i, 0.1).float() for i, name in enumerate(("scale_msa", "shift_msa", "gate_msa", "scale_mlp", "shift_mlp", "gate_mlp"))}
    index = torch.arange(rows, device="cuda", dtype=torch.int32) % 3
    angle = torch.arange(rows, device="cuda").unsqueeze(1) * torch.logspace(0, -4, 48, device="cuda").repeat(2)
    block = Nvfp4Block(rows, hidden, heads, ffn)
    agrees(front, random_bytes(front, "bf16"), lambda: [block.forward(x, w, mod, index, rope=(torch.cos(angle), torch.sin(angle)))])
