"""Steps of few tokens: the greedy choice over a cluster, decode attention in the order of the lengths, experts read once for their pairs."""
import numpy as np
import pytest
import torch

from qwen_triton_b200.engine.step import ORDERED_FROM, _DecodePlan, longest_first
from qwen_triton_b200.ops import kernels
from qwen_triton_b200.ops.kernels import GemmOut
from test_gpu_kernels import DEV, PAGE, rand

pytestmark = pytest.mark.gpu
BF16 = torch.bfloat16


@pytest.mark.parametrize("rows, vocab", [(1, 151936), (3, 151937), (40, 32768), (64, 16384), (2, 4099)])
def test_greedy_choice_over_parts_of_a_row(rows, vocab):
    logits = rand(rows, vocab, seed=1)
    places = [(7 * i * i + 13) % (vocab - 1) for i in range(rows)]
    for i, at in enumerate(places):
        logits[i, at], logits[i, vocab - 1] = 50.0, 50.0                     # a tie with another part's last id: the lower one
    logits[0, :] = -float("inf")
    if rows > 1:
        logits[1, : vocab // 2] = float("nan")                               # never chosen
        logits[1, vocab - 1] = 60.0
    out = torch.empty(rows, dtype=torch.int32, device=DEV)
    kernels.argmax(logits, out)
    assert out.tolist() == [0] + ([vocab - 1] if rows > 1 else []) + places[2:]


@pytest.mark.parametrize("window", [None, 70])
def test_decode_attention_does_not_depend_on_the_order_of_the_lengths(window):
    """More blocks than are resident at once are handed out longest first; eight sequences at a time are not."""
    seqs, nq, nkv, d = 41, 16, 8, 128
    lengths = torch.tensor([1 + (i * 7919) % 193 for i in range(seqs)], dtype=torch.int32, device=DEV)
    width = -(-193 // PAGE)
    k, v = rand(seqs * width, nkv, PAGE, d, seed=2, dtype=BF16), rand(seqs * width, nkv, PAGE, d, seed=3, dtype=BF16)
    table = torch.arange(seqs * width, dtype=torch.int32, device=DEV).view(seqs, width)
    q = rand(seqs, nq, d, seed=4, dtype=BF16)
    whole, parts = torch.full_like(q, float("nan")), torch.full_like(q, float("nan"))
    kernels.attention_decode(q, k, v, whole, table, lengths, nkv, PAGE, 0, window, d ** -0.5, 1, None, None, warps=3)
    for i in range(0, seqs, 8):
        some = slice(i, min(i + 8, seqs))
        kernels.attention_decode(q[some], k, v, parts[some], table[some].contiguous(), lengths[some], nkv, PAGE, 0, window, d ** -0.5, 1, None, None, warps=3)
    assert torch.equal(whole, parts)


@pytest.mark.parametrize("seqs, mask, splits", [(41, {}, 1), (41, {"window": 70}, 1), (41, {"window": 70, "keep_first": 40}, 1), (41, {"chunk": 64}, 1), (41, {}, 3),
                                                (130, {}, 1), (3, {}, 2)])
def test_decode_attention_in_a_given_order(seqs, mask, splits):
    """The same results whatever order the sequences are handed out in: one block a sequence and head, several that merge in a cluster, more
    sequences than a block's threads, fewer blocks than are resident (the order is not read)."""
    nq, nkv, d = 16, 8, 128
    lengths = [1 + (i * 7919) % 193 for i in range(seqs)]
    seq_len = torch.tensor(lengths, dtype=torch.int32, device=DEV)
    width = -(-193 // PAGE)
    k, v = rand(seqs * width, nkv, PAGE, d, seed=2, dtype=BF16), rand(seqs * width, nkv, PAGE, d, seed=3, dtype=BF16)
    table = torch.arange(seqs * width, dtype=torch.int32, device=DEV).view(seqs, width)
    q = rand(seqs, nq, d, seed=4, dtype=BF16)
    order = np.empty((seqs, 2), dtype=np.int32)
    longest_first(np.array(lengths, dtype=np.int32), order)
    results = []
    for given in (None, order, order[::-1].copy()):
        out = torch.full_like(q, float("nan"))
        kernels.attention_decode(q, k, v, out, table, seq_len, nkv, PAGE, 0, mask.get("window"), d ** -0.5, splits, rand(seqs * nq * splits * d, seed=5),
                                 rand(seqs * nq * splits * 2, seed=6), impl="ws", warps=3, chunk=mask.get("chunk"), keep_first=mask.get("keep_first", 0),
                                 order=None if given is None else torch.from_numpy(given).to(DEV))
        results.append(out)
    assert torch.isfinite(results[0]).all()
    assert torch.equal(results[0], results[1]) and torch.equal(results[0], results[2])


@pytest.mark.parametrize("n, widths", [(1, (16,)), (16, (16, 3)), (ORDERED_FROM, (16, 3)), (48, (5,)), (128, (16,))])
def test_the_order_lies_behind_the_tables_of_many_sequences(n, widths):
    plan = _DecodePlan(torch.zeros(8192, dtype=torch.int32, device=DEV), n, widths)
    assert (plan.order is None) is (n < ORDERED_FROM)
    if plan.order is not None:
        assert plan.order.shape == (n, 2) and plan.order.data_ptr() % 8 == 0
        assert plan.order.data_ptr() >= plan.tables[len(widths) - 1].data_ptr() + 4 * n * widths[-1]


@pytest.mark.parametrize("experts, top, width, ff, tokens, skew", [(8, 1, 1024, 2048, 8, False), (4, 2, 2048, 1040, 15, False), (3, 1, 2064, 1024, 32, True),
                                                                   (2, 2, 1040, 2032, 1, False), (16, 2, 2048, 1024, 16, True)])
@pytest.mark.parametrize("gated", [True, False])
@pytest.mark.parametrize("weights", ["output", "input", "none"])
def test_experts_read_once_for_all_of_their_pairs(experts, top, width, ff, tokens, skew, gated, weights):
    """Groups of one pair to four groups of eight of one expert; features and columns that end inside a block."""
    x, up, down = rand(tokens, width, seed=1, dtype=BF16), rand(experts, (2 if gated else 1) * ff, width, seed=2, scale=0.03, dtype=BF16), \
        rand(experts, width, ff, seed=3, scale=0.03, dtype=BF16)
    table = torch.stack([torch.arange(top) if skew else torch.randperm(experts, generator=torch.Generator().manual_seed(t))[:top] for t in range(tokens)]).int().to(DEV)
    pair = 0.5 + rand(tokens, top, seed=5).abs()
    base, scale = rand(2, tokens, width, seed=6), rand(tokens, seed=7)
    mid, out = torch.empty(tokens * top, ff, dtype=BF16, device=DEV), torch.full((tokens, width), float("nan"), device=DEV)
    kernels.experts_by_pair(x, None, table, up, down, mid, out, "silu", pair_weight=0.7, pair_weights=pair if weights == "output" else None, gated=gated,
                            in_weights=pair if weights == "input" else None, base=GemmOut(base), row_scale=scale)
    want = scale[:, None].double() * base.double().sum(0)
    for t in range(tokens):
        for k in range(top):
            e, share = int(table[t, k]), float(pair[t, k])
            h = up[e].double() @ x[t].double() * (share if weights == "input" else 1.0)
            act = torch.nn.functional.silu(h[:ff]) * h[ff:] if gated else torch.nn.functional.silu(h)
            want[t] += (down[e].double() @ act.to(BF16).double()) * (share if weights == "output" else 0.7)
    # the activations are rounded to bfloat16 (2^-9 of each; here some round the other way than the 64-bit ones), the rest are float sums
    assert float((out.double() - want).norm()) <= 2.0 ** -9 * float(want.norm())
