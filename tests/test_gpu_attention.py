"""Full self-attention (head_dim 128) against the dense fp64 softmax of the reference's test fixture, on the
reference's own shapes, seeds and bound (tests/test_nn_kernels_attention_synthetic.cu:4-160)."""
import ctypes as C
import zlib

import numpy as np
import pytest
import torch

import oracle
import slopfab_b200 as sfq
from helpers import bf16_tensor, bits

pytestmark = pytest.mark.gpu
D = 128


def attention(q, k, v, heads, kv_heads, out=None, scale=0.0, ld_q=None, ld_kv=None):
    """q: bf16 [seq_q, >= heads*128] tensors (views allowed); returns out [seq_q, heads*128]."""
    seq_q, seq_kv = q.shape[0], k.shape[0]
    out = torch.empty((seq_q, heads * D), dtype=torch.bfloat16, device="cuda") if out is None else out
    n = C.c_size_t()
    sfq.check(sfq.lib.sfq_attention_workspace_bytes(seq_kv, kv_heads, D, C.byref(n)))
    ws = torch.empty(n.value, dtype=torch.uint8, device="cuda")
    sfq.check(sfq.lib.sfq_attention_forward(q.data_ptr(), ld_q or q.stride(0), k.data_ptr(), v.data_ptr(), ld_kv or k.stride(0),
                                            out.data_ptr(), out.stride(0), seq_q, seq_kv, heads, kv_heads, D, scale, ws.data_ptr(), n.value,
                                            sfq.stream_ptr()))
    return out


def data(seq, heads, seed, scale):
    return oracle.from_bf16(oracle.to_bf16(oracle.make_data(seq * heads * D, seed, scale))).reshape(seq, heads * D)


def close(want, got):
    err = np.abs(got - want)
    bound = 1e-3 + 1e-2 * np.abs(want)
    assert (err <= bound).all(), (float(err.max()), int(np.argmax(err - bound)))


def run_case(q, k, v, heads, kv_heads):
    want = oracle.attention(q, k, v, heads, kv_heads, D, 1.0 / np.sqrt(D))
    out = attention(bf16_tensor(oracle.to_bf16(q)), bf16_tensor(oracle.to_bf16(k)), bf16_tensor(oracle.to_bf16(v)), heads, kv_heads)
    close(want, oracle.from_bf16(bits(out)))
    assert sfq.device_status() == 0
    return out


def test_reference_blocked_case():
    run_case(data(512, 4, 161, 0.3), data(512, 4, 162, 0.3), data(512, 4, 163, 1.0), 4, 4)


@pytest.mark.parametrize("seq", [17, 61, 127, 199])
def test_ragged_tail(seq):
    run_case(data(seq, 3, 401 + seq, 0.3), data(seq, 3, 402 + seq, 0.3), data(seq, 3, 403 + seq, 1.0), 3, 3)


@pytest.mark.parametrize("seq", [1, 127, 128, 259, 2051])
def test_compact_query_chunks_equal_the_full_call(seq):
    q, k, v = data(seq, 2, 9701, 0.3), data(seq, 2, 9702, 0.3), data(seq, 2, 9703, 1.0)
    full = run_case(q, k, v, 2, 2)
    dq, dk, dv = (bf16_tensor(oracle.to_bf16(t)) for t in (q, k, v))
    for chunk in (64, 257):
        parts = [attention(dq[s:s + chunk], dk, dv, 2, 2) for s in range(0, seq, chunk)]
        assert torch.equal(torch.cat(parts), full)  # a query row never depends on which chunk carried it


def test_grouped_heads_and_fused_projection_views():
    seq, heads, kv_heads = 300, 8, 2
    q, k, v = data(seq, heads, 51, 0.3), data(seq, kv_heads, 52, 0.3), data(seq, kv_heads, 53, 1.0)
    run_case(q, k, v, heads, kv_heads)
    # q, k, v as the thirds of one [seq, 3 * heads * 128] buffer, as the fused QKV projection leaves them
    heads = 3
    q, k, v = data(seq, heads, 61, 0.3), data(seq, heads, 62, 0.3), data(seq, heads, 63, 1.0)
    fused = bf16_tensor(oracle.to_bf16(np.concatenate([q, k, v], axis=1)))
    w = heads * D
    out = attention(fused[:, :w], fused[:, w:2 * w], fused[:, 2 * w:], heads, heads)
    close(oracle.attention(q, k, v, heads, heads, D, 1.0 / np.sqrt(D)), oracle.from_bf16(bits(out)))


def test_running_maximum_that_keeps_growing():
    """Keys grow along the sequence so that every few tiles the maximum jumps by more than the rescale threshold: the
    accumulator rescale in tensor memory runs many times."""
    seq, heads = 1500, 2
    q = data(seq, heads, 71, 1.0)
    ramp = (0.2 + 3.0 * np.arange(seq) / seq).astype(np.float32)[:, None]
    sign = np.sign(q[0:1])
    sign[sign == 0] = 1
    k = oracle.from_bf16(oracle.to_bf16(sign * ramp))  # q[0] . k[j] = ramp[j] * sum |q[0]|: grows along the sequence
    v = data(seq, heads, 73, 1.0)
    want = oracle.attention(q, k, v, heads, heads, D, 1.0 / np.sqrt(D))
    out = attention(bf16_tensor(oracle.to_bf16(q)), bf16_tensor(oracle.to_bf16(k)), bf16_tensor(oracle.to_bf16(v)), heads, heads)
    close(want, oracle.from_bf16(bits(out)))
    scores = (q[0, :D] @ k[:, :D].T) / np.sqrt(D) * np.log2(np.e)
    assert scores.max() - scores[:128].max() > 16  # row 0 crosses the threshold at least twice
    assert sfq.device_status() == 0


@pytest.mark.parametrize("spike", [0, 33, 95, 96, 127, 128 + 31, 128 + 63, 128 + 64, 128 + 95, 128 + 96, 128 + 127, 256, 256 + 110, 399])
def test_one_key_that_outgrows_the_reference(spike):
    """One key raises some rows' scores by more than 2^15 in base-2 units of probability: past the first 128 keys, over which the first
    reference is taken, the reference maximum moves in that key's step and the accumulator is rescaled."""
    seq, heads = 400, 2
    q, k, v = data(seq, heads, 81, 1.0), data(seq, heads, 82, 0.3), data(seq, heads, 83, 1.0)
    k[spike] = oracle.from_bf16(oracle.to_bf16((4.0 * np.where(q[spike // 2] < 0, -1.0, 1.0)).astype(np.float32)))
    scores = (q[:, :D] @ k[:, :D].T) / np.sqrt(D) * np.log2(np.e)
    assert scores[spike // 2, spike] - np.delete(scores[spike // 2], spike).max() > 16
    run_case(q, k, v, heads, heads)


def run_not_finite(q, k, v, heads):
    """Every query head is the same one, over one key / value head; NaN exactly where the dense softmax has it, close elsewhere."""
    want = oracle.attention(q, k, v, 1, 1, D, 1.0 / np.sqrt(D))
    dq, dk, dv = (bf16_tensor(oracle.to_bf16(t)) for t in (q, k, v))
    got = oracle.from_bf16(bits(attention(dq.repeat(1, heads), dk, dv, heads, 1)))
    for h in (0, heads - 1):
        part = got[:, h * D:(h + 1) * D]
        nan = np.isnan(want)
        assert np.array_equal(nan, np.isnan(part)), (int(nan.sum()), int(np.isnan(part).sum()))
        close(want[~nan], part[~nan])
    assert sfq.device_status() == 0
    return want


@pytest.mark.parametrize("whole_blocks", [False, True])
@pytest.mark.parametrize("value", [np.nan, np.inf])
@pytest.mark.parametrize("key", [0, 1, 2, 3, 4, 5, 6, 7, 64, 66, 129, 130, 192, 299])
def test_one_key_that_is_not_finite(key, value, whole_blocks):
    """A score that is NaN or +inf makes its row NaN, wherever in a group of eight keys it stands; one that is -inf has no weight."""
    seq = 300
    q, k, v = data(seq, 1, 84, 1.0), data(seq, 1, 85, 0.3), data(seq, 1, 86, 1.0)
    k[key, 5] = value
    want = run_not_finite(q, k, v, heads_of_whole_blocks(seq) if whole_blocks else 2)
    assert np.isnan(want).any() and (np.isnan(value) or not np.isnan(want).all())


@pytest.mark.parametrize("whole_blocks", [False, True])
@pytest.mark.parametrize("first", [1, 64, 127, 128, 129, 130, 192, 257, 299, 300])
def test_keys_of_no_weight_at_the_start(first, whole_blocks):
    """Rows whose first scores are all -inf are the average of the other keys; a row without any finite score is NaN."""
    seq = 300
    q, k, v = data(seq, 1, 87, 1.0), data(seq, 1, 88, 0.3), data(seq, 1, 89, 1.0)
    q[:, 5] = np.where(np.arange(seq) % 3 == 0, 0.0, np.abs(q[:, 5]) + 0.25)  # 0 * -inf is NaN: every third row
    k[:first, 5] = -np.inf
    want = run_not_finite(q, k, v, heads_of_whole_blocks(seq) if whole_blocks else 2)
    assert np.isnan(want[0]).all() and np.isnan(want[1]).all() == (first == seq)


@pytest.mark.parametrize("aligned_v", [True, False])
@pytest.mark.parametrize("seq_q,seq_kv", [(1, 1), (130, 63), (300, 64), (256, 65), (129, 127), (300, 128), (130, 129), (40, 191), (300, 192), (257, 193)])
def test_edges_of_the_steps_of_64_keys(seq_q, seq_kv, aligned_v):
    """One step, a full or ragged first or second half of a key tile at the end, in CTAs of one query tile."""
    heads = 3
    q, k, v = data(seq_q, heads, 31, 0.3), data(seq_kv, heads, 32, 0.3), data(seq_kv, heads, 33, 1.0)
    dq, dk, dv = (bf16_tensor(oracle.to_bf16(t)) for t in (q, k, v))
    if not aligned_v:
        shifted = torch.empty(seq_kv * heads * D + 8, dtype=torch.bfloat16, device="cuda")[1:1 + seq_kv * heads * D].view(seq_kv, heads * D)
        shifted.copy_(dv)
        dv = shifted
    close(oracle.attention(q, k, v, heads, heads, D, 1.0 / np.sqrt(D)), oracle.from_bf16(bits(attention(dq, dk, dv, heads, heads))))
    assert sfq.device_status() == 0


@pytest.mark.parametrize("aligned_v", [True, False])
@pytest.mark.parametrize("seq_kv", [1, 63, 64, 65, 127, 128, 129, 191, 192, 193, 256])
@pytest.mark.parametrize("seq_q", [256, 300])
def test_edges_of_the_steps_with_two_query_tiles(seq_q, seq_kv, aligned_v):
    """The same ends of the keys in CTAs whose second query tile has rows (the launches above run one query tile per CTA, or one
    whose second tile is empty): every query head is the same one, over one key / value head."""
    heads = heads_of_whole_blocks(seq_q)
    q, k, v = data(seq_q, 1, 34, 0.3), data(seq_kv, 1, 35, 0.3), data(seq_kv, 1, 36, 1.0)
    dq, dk, dv = (bf16_tensor(oracle.to_bf16(t)) for t in (q, k, v))
    if not aligned_v:
        shifted = torch.empty(seq_kv * D + 8, dtype=torch.bfloat16, device="cuda")[1:1 + seq_kv * D].view(seq_kv, D)
        shifted.copy_(dv)
        dv = shifted
    out = attention(dq.repeat(1, heads), dk, dv, heads, 1)
    close(oracle.attention(q, k, v, 1, 1, D, 1.0 / np.sqrt(D)), oracle.from_bf16(bits(out[:, :D].contiguous())))
    assert torch.equal(out, out[:, :D].repeat(1, heads))
    assert sfq.device_status() == 0


@pytest.mark.parametrize("spikes", [(63,), (64,), (128 + 63, 128 + 64), (128 + 64, 256), (129, 200, 384)])
def test_reference_that_moves_at_the_edge_of_a_step(spikes):
    """Spikes at the edges of steps, inside the first 128 keys (where they raise the first reference) and behind them."""
    seq, heads = 385, 2
    q, k, v = data(seq, heads, 81, 1.0), data(seq, heads, 82, 0.3), data(seq, heads, 83, 1.0)
    for i, s in enumerate(spikes):
        k[s] = oracle.from_bf16(oracle.to_bf16(((4.0 + 2 * i) * np.where(q[s // 2] < 0, -1.0, 1.0)).astype(np.float32)))
    run_case(q, k, v, heads, heads)


def moves_of_the_reference(scores):
    """What the kernel's rule does with a row's scores (log2 units): the steps of 64 keys whose sum exceeds 2^15 against the reference,
    as (step, what exceeded it: the step itself or only the sum carried over from the tile's first half, whether the reference moved)."""
    reference, carried, found = scores[:128].max(), 0.0, []
    for step in range(-(-len(scores) // 64)):
        part = scores[64 * step:64 * step + 64]
        carried = carried if step % 2 else 0.0
        alone = np.exp2(part - reference).sum()
        total = carried + alone
        if total > 32768:
            higher = max(reference, part.max())
            found.append((step, "step" if alone > 32768 else "carried", bool(higher > reference)))
            reference = higher
            total = np.exp2(part - reference).sum()
        carried = total
    return found


@pytest.mark.parametrize("aligned_v", [True, False])
@pytest.mark.parametrize("whole_blocks", [False, True])
def test_each_way_a_reference_can_move(whole_blocks, aligned_v):
    """Rows that outgrow their reference in successive steps, in the first or second half of a key tile alone, in the last step, through the
    sum of a tile's halves alone (with a higher maximum and without one), several of them in one warp; rows beside them keep their bits."""
    seq_q, seq_kv = 300, 449
    plans = {  # of a row: {key: score in log2 units}, 0 elsewhere, and the moves it is made for
        "successive": ({128 + 10: 30, 192 + 63: 60, 256: 90, 320 + 5: 120, 448: 150},
                       [(2, "step", True), (3, "step", True), (4, "step", True), (5, "step", True), (7, "step", True)]),
        "first half": ({256 + 40: 33}, [(4, "step", True)]),
        "second half": ({192 + 1: 33}, [(3, "step", True)]),
        "carried": ({j: np.log2(20000 / 64) for j in range(128, 256)}, [(3, "carried", True)]),
        "carried, no higher": ({j: np.log2(32736 / 64) for j in range(128, 192)}, [(3, "carried", False)]),
        "within the limit": ({j: np.log2(20000 / 64) for j in range(256, 320)}, []),
    }
    rows = {5: "successive", 6: "carried", 7: "within the limit", 40: "first half", 70: "carried, no higher", 71: "second half",
            133: "successive", 134: "carried, no higher", 200: "carried", 260: "carried", 261: "first half", 290: "within the limit"}
    q, k, v = data(seq_q, 1, 91, 1.0), data(seq_kv, 1, 92, 0.3), data(seq_kv, 1, 93, 1.0)
    q[:, :12], k[:, :12] = 0.0, 0.0  # two channels per plan, in which a row of the plan is (8, 1) and everything else 0
    for row in rows:
        q[row] = 0.0
    for i, (name, (scores, _)) in enumerate(plans.items()):
        for row in (r for r in rows if rows[r] == name):
            q[row, 2 * i:2 * i + 2] = 8.0, 1.0
        for key, score in scores.items():
            dot = np.float32(score * np.sqrt(D) / np.log2(np.e))
            k[key, 2 * i] = oracle.from_bf16(oracle.to_bf16(np.array([dot / 8], np.float32)))[0]
            k[key, 2 * i + 1] = oracle.from_bf16(oracle.to_bf16(np.array([dot - 8 * k[key, 2 * i]], np.float32)))[0]
    scores = q.astype(np.float64) @ k.T.astype(np.float64) / np.sqrt(D) * np.log2(np.e)
    for row in range(seq_q):
        assert moves_of_the_reference(scores[row]) == (plans[rows[row]][1] if row in rows else []), row
    heads = heads_of_whole_blocks(seq_q) if whole_blocks else 2
    dk, dv = bf16_tensor(oracle.to_bf16(k)), bf16_tensor(oracle.to_bf16(v))
    if not aligned_v:
        shifted = torch.empty(seq_kv * D + 8, dtype=torch.bfloat16, device="cuda")[1:1 + seq_kv * D].view(seq_kv, D)
        shifted.copy_(dv)
        dv = shifted
    out = attention(bf16_tensor(oracle.to_bf16(q)).repeat(1, heads), dk, dv, heads, 1)
    close(oracle.attention(q, k, v, 1, 1, D, 1.0 / np.sqrt(D)), oracle.from_bf16(bits(out[:, :D].contiguous())))
    assert torch.equal(out, out[:, :D].repeat(1, heads))
    still = q.copy()
    moving = [row for row in rows if plans[rows[row]][1]]
    still[moving] = 0.0
    alone = attention(bf16_tensor(oracle.to_bf16(still)).repeat(1, heads), dk, dv, heads, 1)
    others = [row for row in range(seq_q) if row not in moving]
    assert torch.equal(out[others], alone[others])  # a row's bits do not depend on its neighbours
    assert sfq.device_status() == 0


def test_launches_repeat_bit_for_bit():
    """The next scores are written over the columns the product before them reads its probabilities from, with nothing between the two
    but the order in which they were issued: a product that were overtaken would show in some launch of many."""
    seq, heads = 2048, 40
    g = torch.Generator("cuda").manual_seed(17)
    q, k, v = (torch.randn((seq, heads * D), device="cuda", generator=g).to(torch.bfloat16) for _ in range(3))
    first = attention(q, k, v, heads, heads)
    same = torch.ones((), dtype=torch.bool, device="cuda")
    for _ in range(300):
        same &= (attention(q, k, v, heads, heads) == first).all()
    assert bool(same)
    assert sfq.device_status() == 0


def test_values_that_do_not_start_on_sixteen_bytes():
    """q, k and out need 16-byte rows, v never did: such a v is copied to the workspace first."""
    seq, heads = 259, 2
    q, k, v = data(seq, heads, 91, 0.3), data(seq, heads, 92, 0.3), data(seq, heads, 93, 1.0)
    dq, dk, dv = (bf16_tensor(oracle.to_bf16(t)) for t in (q, k, v))
    shifted = torch.empty(seq * heads * D + 8, dtype=torch.bfloat16, device="cuda")[3:3 + seq * heads * D].view(seq, heads * D)
    shifted.copy_(dv)
    assert torch.equal(attention(dq, dk, shifted, heads, heads), attention(dq, dk, dv, heads, heads))
    assert sfq.device_status() == 0


@pytest.mark.parametrize("seq,heads", [(130, 150), (256, 160), (385, 80), (513, 50)])
def test_last_wave_as_single_query_tiles(seq, heads):
    """Whole blocks of 256 queries and blocks run as two CTAs side by side in one launch (the last wave of 148 SMs): each head,
    whichever form carried it, equals the same head computed alone."""
    g = torch.Generator("cuda").manual_seed(seq)
    q, k, v = (torch.randn((seq, heads * D), device="cuda", generator=g).to(torch.bfloat16) for _ in range(3))
    out = attention(q, k, v, heads, heads)
    for h in (0, heads // 2, heads - 1):
        one = attention(*(t[:, h * D:(h + 1) * D].contiguous() for t in (q, k, v)), 1, 1)
        assert torch.equal(out[:, h * D:(h + 1) * D], one)
    assert sfq.device_status() == 0


def heads_of_whole_blocks(seq):
    """A head count whose launch keeps every block of 256 queries in one CTA of two query tiles: the last wave is more than half full."""
    sms, blocks = torch.cuda.get_device_properties(0).multi_processor_count, -(-seq // 256)
    heads = next(h for h in range(1, 4 * sms) if 2 * (blocks * h % sms) > sms)
    assert blocks * heads < 16 * sms
    return heads


@pytest.mark.parametrize("seq", [257, 385, 513, 1000])
@pytest.mark.parametrize("aligned_v", [True, False])
def test_whole_blocks_of_two_query_tiles(seq, aligned_v):
    """Two query tiles per CTA throughout, V as it lies and transposed: against torch, and each head bit for bit the same head alone
    (which runs as single query tiles)."""
    heads = heads_of_whole_blocks(seq)
    g = torch.Generator("cuda").manual_seed(seq)
    q, k, v = (torch.randn((seq, heads * D), device="cuda", generator=g).to(torch.bfloat16) for _ in range(3))
    if not aligned_v:
        shifted = torch.empty(seq * heads * D + 8, dtype=torch.bfloat16, device="cuda")[3:3 + seq * heads * D].view(seq, heads * D)
        shifted.copy_(v)
        v = shifted
    out = attention(q, k, v, heads, heads)
    sh = lambda t: t.view(seq, heads, D).transpose(0, 1).float()  # noqa: E731
    want = torch.nn.functional.scaled_dot_product_attention(sh(q), sh(k), sh(v)).transpose(0, 1).reshape(seq, heads * D)
    assert bool(((out.float() - want).abs() <= 1e-3 + 1e-2 * want.abs()).all())
    for h in (0, heads // 2, heads - 1):
        one = attention(*(t[:, h * D:(h + 1) * D].contiguous() for t in (q, k, v)), 1, 1)
        assert torch.equal(out[:, h * D:(h + 1) * D], one)
    assert sfq.device_status() == 0


@pytest.mark.parametrize("aligned_v", [True, False])
@pytest.mark.parametrize("spike", [0, 95, 96, 128 + 95, 128 + 127, 256 + 110, 399, "ramp"])
def test_reference_that_moves_in_whole_blocks(spike, aligned_v):
    """The maxima of the tests above through CTAs of two query tiles: every query head is the same one, over one key / value head."""
    seq = 400
    heads = heads_of_whole_blocks(seq)
    q, k, v = data(seq, 1, 81, 1.0), data(seq, 1, 82, 0.3), data(seq, 1, 83, 1.0)
    if spike == "ramp":
        k = oracle.from_bf16(oracle.to_bf16(np.where(q[0:1] < 0, -1.0, 1.0) * (0.2 + 3.0 * np.arange(seq) / seq).astype(np.float32)[:, None]))
    else:
        k[spike] = oracle.from_bf16(oracle.to_bf16((4.0 * np.where(q[spike // 2] < 0, -1.0, 1.0)).astype(np.float32)))
    want = oracle.attention(q, k, v, 1, 1, D, 1.0 / np.sqrt(D))
    dq, dk, dv = (bf16_tensor(oracle.to_bf16(t)) for t in (q, k, v))
    if not aligned_v:
        shifted = torch.empty(seq * D + 8, dtype=torch.bfloat16, device="cuda")[5:5 + seq * D].view(seq, D)
        shifted.copy_(dv)
        dv = shifted
    out = attention(dq.repeat(1, heads), dk, dv, heads, 1)
    close(want, oracle.from_bf16(bits(out[:, :D].contiguous())))
    assert torch.equal(out, out[:, :D].repeat(1, heads))
    assert sfq.device_status() == 0


@pytest.mark.parametrize("seq,heads,scale,crc", [(1500, 2, 1.0, 0xBF518A00), (2051, 4, 0.3, 0x633D8771), (513, 40, 1.0, 0x323EB421)])
def test_bits_of_seeded_calls(seq, heads, scale, crc):
    """How a key tile's probabilities are handed to the second product is a matter of speed alone: their sum is one chain over the
    tile's keys, and a call's bits are those of the kernel that handed them over in one part (its checksums). A sum per part
    shows in a few of a million elements. No row of these calls outgrows its first reference; one that does has bits that depend on the
    keys over which its new reference is taken."""
    q, k, v = (bf16_tensor(oracle.to_bf16(data(seq, heads, 300 + i + seq, scale))) for i in range(3))
    assert zlib.crc32(bits(attention(q, k, v, heads, heads)).tobytes()) == crc


def test_against_torch_on_a_longer_sequence():
    torch.manual_seed(5)
    seq, heads = 4096 + 77, 4
    q, k, v = (torch.randn(seq, heads * D, device="cuda").mul_(s).to(torch.bfloat16) for s in (1.0, 1.0, 1.0))
    out = attention(q, k, v, heads, heads)
    sh = lambda t: t.view(seq, heads, D).transpose(0, 1).float()  # noqa: E731
    want = torch.nn.functional.scaled_dot_product_attention(sh(q), sh(k), sh(v)).transpose(0, 1).reshape(seq, heads * D)
    err = (out.float() - want).abs()
    assert bool((err <= 1e-3 + 1e-2 * want.abs()).all()), float(err.max())
    assert sfq.device_status() == 0


def test_refusals():
    t = torch.zeros((128, 128), dtype=torch.bfloat16, device="cuda")
    with pytest.raises(sfq.SfqError, match="head_dim"):
        sfq.check(sfq.lib.sfq_attention_forward(t.data_ptr(), 64, t.data_ptr(), t.data_ptr(), 64, t.data_ptr(), 64, 128, 128, 1, 1, 64, 0.0,
                                                t.data_ptr(), 1 << 20, None))
    o = torch.zeros_like(t)
    with pytest.raises(sfq.SfqError, match="workspace"):
        sfq.check(sfq.lib.sfq_attention_forward(t.data_ptr(), 128, t.data_ptr(), t.data_ptr(), 128, o.data_ptr(), 128, 128, 128, 1, 1, 128, 0.0,
                                                t.data_ptr(), 16, None))
    with pytest.raises(sfq.SfqError, match="alias"):
        sfq.check(sfq.lib.sfq_attention_forward(t.data_ptr(), 128, t.data_ptr(), t.data_ptr(), 128, t.data_ptr(), 128, 128, 128, 1, 1, 128, 0.0,
                                                o.data_ptr(), 1 << 16, None))
