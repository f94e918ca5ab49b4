"""The split plans of ``Linear`` (host decisions, no device): every plan is one the kernels accept."""
import itertools

import pytest
import torch

from qwen_triton_b200.ops import kernels
from qwen_triton_b200.parts import linear


class _Workspace:
    def __init__(self):
        self.declared = {}

    def declare(self, name, numel, dtype):
        self.declared[name] = (numel, dtype)


class _Runtime:
    def __init__(self, dtype, max_step_tokens):
        self.dtype, self.max_step_tokens, self.workspace, self.device = dtype, max_step_tokens, _Workspace(), "cpu"
        self.sm_count = 148


SHAPES = [(6144, 4096), (4096, 12288), (24576, 4096), (151936, 4096), (1024, 2048), (130, 72), (5003, 1000), (200, 8), (51200, 5120)]


@pytest.mark.parametrize("out_features, in_features", SHAPES)
def test_every_split_count_leaves_no_split_without_k_blocks(out_features, in_features):
    for rows, per_sm in linear._SPLIT_PLANS:
        splits = linear.pick_splits(out_features, in_features, per_sm * 148, rows)
        assert 1 <= splits <= 16 and kernels.tc_normalise_splits(in_features, splits) == splits
        fused = linear.pick_splits(out_features, in_features, per_sm * 148, rows, kernels.FUSED_MAX_SPLITS, 1.0)
        assert 1 <= fused <= kernels.FUSED_MAX_SPLITS and kernels.tc_normalise_splits(in_features, fused) == fused
    for rows in (257, 300, 512, 1000, 2048, 4096):
        splits = linear.pick_pair_splits(out_features, in_features, rows, 74)
        assert 1 <= splits <= 4 and kernels.tc_normalise_splits(in_features, splits) == splits
        blocks = -(-in_features // 64)
        assert (splits - 1) * -(-blocks // splits) < blocks


def test_a_weight_whose_tiles_fill_the_machine_is_not_cut_into_a_second_wave():
    """192 tiles of the 8B shape's gate/up weight: three ranges up to 16 rows (576 blocks of 592 resident), none beyond
    (two blocks per SM: 384 blocks would be a second wave); the fused form (three blocks per SM for this product)
    keeps two ranges there and gives the 32B shape's 400 tiles none."""
    assert [linear.pick_splits(24576, 4096, per_sm * 148, rows, sms=148) for rows, per_sm in linear._SPLIT_PLANS] == [3, 1, 1, 1]
    assert linear.pick_splits(24576, 4096, 3 * 148, 16, kernels.FUSED_MAX_SPLITS, 1.0, sms=148) == 2
    assert linear.pick_splits(51200, 5120, 3 * 148, 16, kernels.FUSED_MAX_SPLITS, 1.0, sms=148) == 1
    # a weight with fewer tiles than SMs is cut as before
    assert linear.pick_splits(6144, 4096, 2 * 148, 64, sms=148) == linear.pick_splits(6144, 4096, 2 * 148, 64) == 6


def test_a_product_with_many_tiles_is_not_split():
    assert linear.pick_splits(151936, 4096, 296, 64) == 1
    assert linear.pick_pair_splits(24576, 4096, 2048, 74) == 1
    assert linear.pick_pair_splits(4096, 4096, 512, 74) > 1          # 32 tiles on 74 pairs


@pytest.mark.parametrize("max_rows", [40, 256, 300, 4096])
def test_plans_are_sorted_and_the_partial_buffer_holds_every_plan(max_rows):
    runtime = _Runtime(torch.bfloat16, max_rows)
    layer = linear.Linear("x", 4096, 12288, runtime)
    most = [rows for rows, _ in layer.split_plans]
    assert most == sorted(set(most))
    words = max((rows * splits for rows, splits in layer.split_plans if splits > 1), default=0)
    assert runtime.workspace.declared["x.partial"][0] == words * 4096
    for rows, splits in layer.split_plans:
        assert kernels.tc_normalise_splits(12288, splits) == splits
    # float32 models and rows that TMA cannot address take no split plan at all
    assert linear.Linear("y", 4096, 12288, _Runtime(torch.float32, max_rows)).split_plans == []
    assert linear.Linear("z", 4096, 12284, _Runtime(torch.bfloat16, max_rows)).split_plans == []


def test_the_fused_ring_is_as_deep_as_keeps_every_block_resident():
    """8B shapes: four stages for q/k/v and o (384 and 256 blocks of the 444 that three to an SM give), five for down
    (256 of 296); the 32B shape's q/k/v has 480 blocks and keeps the default three stages, its down takes four."""
    runtime = _Runtime(torch.bfloat16, 64)
    def stages(out_features, in_features, role):
        return linear.Linear(f"t.{role}.{out_features}", out_features, in_features, runtime, role=role)._fused_stages(8)
    assert [stages(6144, 4096, "qkv"), stages(4096, 4096, "attn_out"), stages(24576, 4096, "gate"), stages(4096, 12288, "mlp_out")] == [4, 4, 4, 5]
    assert [stages(10240, 5120, "qkv"), stages(5120, 8192, "attn_out"), stages(5120, 25600, "mlp_out")] == [0, 4, 4]
    assert stages(4096, 4096, "") == 0


# (heads, key channels, value columns, portions, token by token, in chunks): measured, microseconds with cold caches
_RECURRENCES = [
    (16, 128, 128, [64], 36.6, 58.2), (16, 128, 128, [100], 46.9, 58.7), (16, 128, 128, [128], 51.2, 56.5), (16, 128, 128, [200], 69.7, 63.8),
    (16, 128, 128, [1024], 284.4, 94.1), (16, 128, 128, [64] * 2, 44.8, 59.4), (16, 128, 128, [90] * 5, 102.4, 84.3), (16, 128, 128, [64] * 32, 232.3, 142.9),
    (16, 128, 128, [64] + [3] * 31, 49.6, 103.1), (16, 128, 128, [128] + [3] * 31, 66.5, 108.4), (16, 128, 128, [64] + [20] * 31, 103.1, 117.7),
    (32, 128, 128, [64], 41.4, 56.3), (32, 128, 128, [100], 57.7, 72.7), (32, 128, 128, [200], 96.9, 77.6), (32, 128, 128, [300] + [3] * 31, 151.5, 212.8),
    (8, 128, 128, [150], 50.8, 56.1), (8, 128, 128, [200], 61.9, 55.9), (8, 128, 128, [300] + [3] * 31, 116.8, 88.6), (8, 128, 128, [128] + [3] * 31, 61.7, 84.4),
    (16, 256, 128, [64], 62.3, 70.8), (16, 256, 128, [100], 84.1, 71.3), (16, 96, 128, [100], 42.8, 52.4), (16, 96, 128, [400], 119.9, 69.9)]


@pytest.mark.parametrize("heads, dim, vdim, lengths, walk, chunks", _RECURRENCES)
def test_recurrences_take_the_faster_form(heads, dim, vdim, lengths, walk, chunks):
    """A short prompt, or many short portions beside a long one, keeps the walk; no choice costs more than a tenth."""
    from types import SimpleNamespace
    step = SimpleNamespace(max_q_len=max(lengths), n_seqs=len(lengths))
    taken = chunks if kernels.decay_chunks_pay(step, sum(lengths), heads, dim, vdim, 4096, 148) else walk
    assert taken <= 1.1 * min(walk, chunks)


def test_recurrences_walk_where_chunks_are_less_exact_or_do_not_fit():
    from types import SimpleNamespace
    step = SimpleNamespace(max_q_len=1000, n_seqs=1)
    assert not kernels.decay_chunks_pay(step, 1000, 8, 64, 128, 4096, 148)          # up to 64 key channels
    assert kernels.decay_chunks_pay(SimpleNamespace(max_q_len=1024, n_seqs=1), 1024, 8, 64, 128, 4096, 148)
    assert not kernels.decay_chunks_pay(SimpleNamespace(max_q_len=2000, n_seqs=100), 2099, 16, 128, 128, 2100, 148)      # more sequences than the scratch has ends for


# (heads, d, rot, dv, rank, longest, sequences, tokens, over latent rows, over keys and values per head): measured, microseconds
_LATENT_PROMPTS = [
    (16, 128, 64, 128, 512, 64, 1, 64, 59.2, 58.7), (16, 128, 64, 128, 512, 400, 1, 400, 121.6, 97.5), (16, 128, 64, 128, 512, 1000, 1, 1000, 199.4, 117.2),
    (16, 128, 64, 128, 512, 2048, 1, 2048, 518.5, 165.8), (16, 128, 64, 128, 512, 64, 8, 512, 91.0, 93.4), (16, 128, 64, 128, 512, 64, 32, 2048, 213.5, 166.5),
    (16, 128, 64, 128, 512, 128, 16, 2048, 223.8, 142.6), (16, 128, 64, 128, 512, 64, 32, 157, 62.7, 99.1), (16, 128, 64, 128, 512, 64, 32, 591, 106.5, 121.7),
    (16, 128, 64, 128, 512, 64, 32, 1056, 131.7, 133.9), (128, 128, 64, 128, 512, 64, 1, 64, 89.2, 88.2), (128, 128, 64, 128, 512, 400, 1, 400, 448.4, 255.1),
    (128, 128, 64, 128, 512, 1000, 1, 1000, 1260.7, 435.4), (128, 128, 64, 128, 512, 64, 8, 512, 407.3, 323.0), (128, 128, 64, 128, 512, 64, 32, 157, 161.6, 485.3),
    (128, 128, 64, 128, 512, 64, 32, 591, 482.6, 660.3), (8, 64, 32, 64, 256, 64, 1, 64, 32.0, 41.2), (8, 64, 32, 64, 256, 400, 1, 400, 80.4, 71.1),
    (8, 64, 32, 64, 256, 1000, 1, 1000, 113.4, 79.9), (8, 64, 32, 64, 256, 2048, 1, 2048, 174.1, 94.1), (8, 64, 32, 64, 256, 64, 8, 512, 61.2, 65.2),
    (8, 64, 32, 64, 256, 64, 32, 2048, 78.9, 73.5), (8, 64, 32, 64, 256, 128, 16, 2048, 84.6, 72.3), (8, 64, 32, 64, 256, 64, 32, 157, 42.4, 46.9),
    (8, 64, 32, 64, 256, 64, 32, 591, 61.7, 63.8), (8, 64, 32, 64, 256, 64, 32, 1056, 65.3, 64.8), (16, 64, 32, 64, 64, 64, 1, 64, 28.9, 41.8),
    (16, 64, 32, 64, 64, 400, 1, 400, 69.1, 73.2), (16, 64, 32, 64, 64, 1000, 1, 1000, 89.2, 80.4), (16, 64, 32, 64, 64, 2048, 1, 2048, 193.5, 105.2),
    (16, 64, 32, 64, 64, 64, 8, 512, 58.0, 66.6), (16, 64, 32, 64, 64, 64, 32, 2048, 89.3, 96.2), (16, 64, 32, 64, 64, 128, 16, 2048, 93.2, 82.2),
    (16, 64, 32, 64, 64, 64, 32, 157, 39.1, 62.9), (16, 64, 32, 64, 64, 64, 32, 591, 64.1, 82.8), (16, 64, 32, 64, 64, 64, 32, 1056, 66.4, 85.8),
    (16, 128, 64, 128, 64, 64, 1, 64, 30.9, 47.3), (16, 128, 64, 128, 64, 400, 1, 400, 75.6, 88.8), (16, 128, 64, 128, 64, 1000, 1, 1000, 107.2, 104.3),
    (16, 128, 64, 128, 64, 2048, 1, 2048, 227.3, 143.2), (16, 128, 64, 128, 64, 64, 8, 512, 64.0, 83.0), (16, 128, 64, 128, 64, 64, 32, 2048, 114.5, 141.9),
    (16, 128, 64, 128, 64, 128, 16, 2048, 118.4, 119.6), (16, 128, 64, 128, 64, 64, 32, 157, 41.6, 83.6), (16, 128, 64, 128, 64, 64, 32, 591, 71.0, 108.8),
    (16, 128, 64, 128, 64, 64, 32, 1056, 81.9, 118.3)]


@pytest.mark.parametrize("heads, d, rot, dv, rank, longest, n_seqs, tokens, rows, own", _LATENT_PROMPTS)
def test_latent_prompts_take_the_faster_form(heads, d, rot, dv, rank, longest, n_seqs, tokens, rows, own):
    """Small latents, short prompts and short portions beside a long one keep the latent rows; no choice costs more than a fifth."""
    from qwen_triton_b200.parts.latent_attention import own_keys_pay
    taken = own if own_keys_pay(heads, d, rot, dv, rank, None, longest, n_seqs, tokens) else rows
    assert taken <= 1.2 * min(rows, own)


@pytest.mark.parametrize("heads, tokens", [(16, 4096), (128, 4096), (16, 256)])
def test_latent_prompts_need_little_memory_of_their_own(heads, tokens):
    """Queries, keys and values per head lie where the form over latent rows has its queries and results (a step takes one of the two): a fifth
    more than that form alone at most."""
    from qwen_triton_b200.config.spec import PartSpec
    from qwen_triton_b200.parts.base import Runtime, Workspace
    from qwen_triton_b200.parts.latent_attention import LatentAttention
    params = {"hidden_size": 2048, "num_heads": heads, "head_dim": 128, "rot_dim": 64, "v_head_dim": 128, "q_rank": 768, "kv_rank": 512, "scale": 0.07,
              "position": PartSpec("rope", {"theta": 1e4, "rotary_dim": 64, "head_dim": 64, "pairing": "half"})}
    sizes = []
    for page in (64, 128):                  # pages of 64: the form exists
        runtime = Runtime(device=torch.device("cpu"), dtype=torch.bfloat16, max_step_tokens=tokens, max_positions=tokens, workspace=Workspace(torch.device("cpu")),
                          page_tokens=page, sm_count=148)
        assert LatentAttention(params, "m", runtime).expands == (page == 64)
        sizes.append(sum(numel * dtype.itemsize for name, (numel, dtype) in runtime.workspace._need.items() if name.startswith("latent.")))
    assert sizes[0] <= 1.2 * sizes[1], sizes


# (head size, longest context, window, kept keys, mma.sync, tcgen05): 16 heads, measured, microseconds
@pytest.mark.parametrize("d, context, window, keep_first, mma, tc", [
    (128, 64, 100, 16, 8.3, 7.3), (128, 2048, 100, 16, 48.0, 25.6), (128, 16, None, 0, 8.3, 6.4), (64, 2048, None, 0, 86.7, 46.1), (64, 400, None, 0, 17.4, 14.5),
    (64, 128, None, 0, 8.4, 10.6), (64, 64, None, 0, 6.3, 6.9), (64, 516, None, 0, 21.5, 15.7), (64, 600, 512, 16, 24.8, 20.9), (64, 400, 512, 16, 15.5, 13.2),
    (64, 200, 512, 16, 10.2, 10.9), (64, 600, 384, 16, 22.2, 23.0), (64, 600, 256, 16, 18.8, 22.7), (64, 600, 128, 16, 15.2, 20.7), (64, 1000, 100, 16, 17.0, 22.9)])
def test_kept_keys_and_linear_penalties_take_the_faster_kernel(d, context, window, keep_first, mma, tc):
    taken = tc if kernels._kept_on_tcgen05(d, context, window, keep_first) else mma
    assert taken <= 1.05 * min(mma, tc)
