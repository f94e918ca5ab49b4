"""Which products of few tokens run where (host decisions, no device)."""
import numpy as np
import pytest
import torch

from qwen_triton_b200.engine.step import StepContext, longest_first
from qwen_triton_b200.ops import kernels
from qwen_triton_b200.ops.kernels import GemmOut, ScaledRows
from qwen_triton_b200.parts import linear
from test_linear_plans import _Runtime


def _linear(out_features, in_features, role="attn_out", dtype=torch.bfloat16):
    made = linear.Linear("x", out_features, in_features, _Runtime(dtype, 64), role=role)
    made.weight = torch.zeros(out_features, in_features, dtype=dtype)
    return made


@pytest.mark.parametrize("rows, role, plan", [(1, "gate", (32, 8)), (8, "qkv", (32, 8)), (9, "gate", (32, 16)), (16, "attn_out", (16, 16)), (17, "attn_out", None), (1, "", (16, 16))])
def test_few_tokens_on_a_small_weight(rows, role, plan):
    x = torch.zeros(rows, 1024, dtype=torch.bfloat16)
    assert _linear(4096, 1024, role).few_plan(x) == plan
    assert _linear(4096, 1024, role).few_plan(ScaledRows(x, torch.zeros(8, rows), 1024, 1e-6)) == plan


def test_what_keeps_the_ring():
    x = torch.zeros(4, 4096, dtype=torch.bfloat16)
    assert _linear(4096, 4096).few_plan(x) is None                               # 16 M elements: bound by its bytes
    assert _linear(2048, 4096).few_plan(x) == (16, 16)                           # 8 M
    assert _linear(512, 1000).few_plan(torch.zeros(4, 1000, dtype=torch.bfloat16)) is None     # rows off 32-byte boundaries
    shifted = torch.zeros(4 * 1024 + 8, dtype=torch.bfloat16)[8:].view(4, 1024)
    assert _linear(512, 1024).few_plan(shifted) is None or shifted.data_ptr() % 32 == 0


@pytest.mark.parametrize("setting, role, few", [("1", "", True), ("1", "qkv", True), ("0", "", False), ("0", "attn_out", False), ("qkv,gate", "qkv", True),
                                                ("qkv,gate", "mlp_out", False), ("qkv,gate", "", False)])
def test_plain_products_follow_the_switch_of_the_fused_ones(monkeypatch, setting, role, few):
    monkeypatch.setenv("QT_B200_FUSED", setting)
    x = torch.zeros(4, 1024, dtype=torch.bfloat16)
    assert (_linear(4096, 1024, role).plain_few_plan(x) is not None) is few
    monkeypatch.setattr(linear, "_FUSED_ROWS", 3)
    assert _linear(4096, 1024, role).plain_few_plan(x) is None


def test_the_product_itself_asks_the_switch(monkeypatch):
    made, taken = _linear(512, 1024, ""), []
    made.runtime.workspace.view = lambda name, *shape: torch.empty(shape)
    monkeypatch.setattr(kernels, "gemm_fused_store", lambda *args, **kwargs: taken.append("few"))
    monkeypatch.setattr(kernels, "gemm", lambda *args, **kwargs: taken.append("plain"))
    x = torch.zeros(4, 1024, dtype=torch.bfloat16)
    for setting in ("1", "0"):
        monkeypatch.setenv("QT_B200_FUSED", setting)
        made(x)
    assert taken == ["few", "plain"]


@pytest.mark.parametrize("out_features, role, few", [(4736, "", True), (4737, "", False), (8192, "mlp_out", False), (8192, "gate", True), (6144, "qkv", True)])
def test_a_second_wave_of_blocks_keeps_the_ring(out_features, role, few):
    assert (_linear(out_features, 512, role).few_plan(torch.zeros(4, 512, dtype=torch.bfloat16)) is not None) is few


def test_the_sums_of_squares_follow_the_kernel():
    few, many = torch.zeros(8, 2048, dtype=torch.bfloat16), torch.zeros(17, 2048, dtype=torch.bfloat16)
    made = _linear(1024, 2048)
    assert made.norm_tiles(few, 1024) == 64 and made.norm_tiles(many, 1024) == 8
    assert _linear(1000, 2048).norm_tiles(few, 1000) == 63


@pytest.mark.parametrize("rows, on", [(1, False), (32, False), (33, True), (549, True)])
def test_float_products_on_the_tensor_cores(rows, on):
    a, w = torch.zeros(rows, 64), torch.zeros(128, 64)
    assert kernels.gemm_f32_on_tc(a, w, GemmOut(torch.zeros(1, rows, 128))) is on


@pytest.mark.parametrize("lengths, places", [([5, 5, 5], [0, 1, 2]), ([1, 700, 3, 700, 2], [1, 3, 2, 4, 0]), ([9, 1], [0, 1])])
def test_the_longest_sequences_come_first(lengths, places):
    into = np.full((len(lengths), 2), -1, dtype=np.int32)
    longest_first(np.array(lengths, dtype=np.int32), into)
    assert into[:, 0].tolist() == places and into[:, 1].tolist() == [lengths[i] for i in places]


def test_the_step_metadata_has_room_for_the_order():
    for n in (2, 3, 48, 256):
        # a one-token pass of n of the 2 n tokens a pass may have: ids, sequences, positions, starts, pasts, lengths, slots, wanted rows, tables, order
        assert 8 * n + 1 + n * (16 + 32) + 1 + 2 * n <= StepContext.meta_size(2 * n, n, [16, 32])
