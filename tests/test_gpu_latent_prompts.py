"""Prompts over keys and values of every head's own through the engine, on models whose latent layers have the sizes for it: a windowed group
with its ring of pages and a gate per head (Misudra), a layer that reads another's latent and a gate per element (Bisodra), no query
latent, neighbouring pairs and no gate (Bizurax); each against the plain implementation, with the form that ran counted."""
import functools
import tempfile

import pytest
import torch

import plain_bisodra
import plain_bizurax
import plain_misudra
from qwen_triton_b200 import Engine, StepEntry, config_from_dict, write_random_model
from qwen_triton_b200.ops import kernels
from qwen_triton_b200.parts import latent_attention
from qwen_triton_b200.weights import Checkpoint
from test_gpu_vunepel import close

pytestmark = pytest.mark.gpu
_KEEP = []
_LATENT = {"heads": 2, "dim": 32, "rot_dim": 32, "vdim": 64, "kv_rank": 64, "scale": 0.2, "rot": {"base": 100.0, "dims": 32}}
_DENSE = {"kind": "dense", "ff": 48}
MODELS = {
    "misudra": (plain_misudra, 2, {
        "architecture": "Misudra", "vocab": 61, "width": 64, "norm": {"eps": 1e-5}, "loop": {"start": 0, "stop": 1, "times": 1}, "layers": [
            {"type": "latent_attention", "mlp": _DENSE, "mixer": {**_LATENT, "q_rank": 24, "mask": {"size": 100}}},
            {"type": "gla", "mlp": None, "mixer": {"heads": 2, "dim": 16, "vdim": 16, "tau": 4.0, "ranks": {"decay": 4}}},
            {"type": "latent_attention", "mlp": _DENSE, "mixer": {**_LATENT, "heads": 3, "dim": 128, "rot_dim": 48, "q_rank": 40, "vdim": 128, "kv_rank": 128, "mask": {"size": 65},
                                                                   "rot": {"base": 100.0, "dims": 16}}}]}),
    "bisodra": (plain_bisodra, 2, {
        "architecture": "Bisodra", "vocab": 61, "width": 64, "norm": {"eps": 1e-5}, "embedding": {"scale": 1.0}, "logit_scale": 1.0, "layers": [
            {"type": "latent_attention", "mlp": _DENSE, "mixer": {**_LATENT, "q_rank": 24}},
            {"type": "attention", "mlp": None, "mixer": {"heads": 2, "kv_heads": 1, "dim": 16, "vdim": 16, "scale": 0.25, "conv": 2, "mask": {"size": 40, "keep_first": 3}}},
            {"type": "latent_attention", "mlp": _DENSE, "mixer": {**_LATENT, "heads": 5, "dim": 64, "q_rank": 16, "kv_from": 0}}]}),
    "bizurax": (plain_bizurax, 1, {
        "architecture": "Bizurax", "vocab": 61, "width": 64, "norm": {"eps": 1e-5}, "streams": 2, "residual_mult": 0.5, "layers": [
            {"type": "latent_attention", "mlp": _DENSE, "mixer": _LATENT},
            {"type": "retention", "mlp": _DENSE, "mixer": {"heads": 2, "dim": 16, "vdim": 16, "decay": [0.9, 0.99], "rot": {"base": 100.0, "dims": 16}}}]}),
}


@functools.lru_cache(maxsize=None)
def model(name):
    holder = tempfile.TemporaryDirectory(prefix=f"qt_latent_{name}_")
    _KEEP.append(holder)
    config = config_from_dict(MODELS[name][2])
    folder = write_random_model(holder.name, config, seed=5, dtype=torch.bfloat16)
    checkpoint = Checkpoint(folder)
    return folder, config.to_hf_dict(), {n: checkpoint.read(n).float() for n in checkpoint.names()}


@pytest.mark.parametrize("name", list(MODELS))
def test_steps_of_prompts_alone_and_beside_other_sequences(name, monkeypatch):
    """New prompts alone take the form, cut at the engine's portions where there is a window (the longest as long as a portion); prompts beside a
    sequence that has a past, later portions, and more sequences than its scratch has runs for, do not; all give the same logits."""
    monkeypatch.setattr(latent_attention, "own_keys_pay", lambda *sizes: True)
    calls, launch = [], kernels.attention_prefill_rows
    monkeypatch.setattr(kernels, "attention_prefill_rows", lambda *args, **kwargs: (calls.append(1), launch(*args, **kwargs)))
    plain, latent_layers, raw = MODELS[name]
    folder, hf, weights = model(name)
    engine = Engine.from_pretrained(folder, dtype="bf16", max_tokens=4096, max_step_tokens=256, chunk_tokens=128)
    generator = torch.Generator().manual_seed(3)

    def tokens(n):
        return torch.randint(0, raw["vocab"], (n,), generator=generator).tolist()

    def step(rows, slots, done):
        """The given sequences' tokens from ``done`` on, every logit against the plain implementation; how often the form ran."""
        calls.clear()
        got = engine.step([StepEntry(slot, row[d:], list(range(len(row) - d))) for slot, row, d in zip(slots, rows, done)])
        engine.check_kernels()
        want = torch.cat([plain.forward(hf, weights, row)[d:] for row, d in zip(rows, done)])
        close(got, want, "bf16", f"{name}: {[len(r) - d for r, d in zip(rows, done)]} tokens", model_rows=True)
        return len(calls)

    rows = [tokens(n) for n in (130, 64, 7)]
    slots = [engine.new_sequence() for _ in rows]
    assert step(rows, slots, [0] * 3) == latent_layers          # two passes where a portion ends at 128 tokens, the second with a past
    further = [row + tokens(1) for row in rows] + [tokens(70)]
    slots.append(engine.new_sequence())
    assert step(further, slots, [len(row) for row in rows] + [0]) == 0 and not engine._ctx.from_start
    more = [tokens(128), tokens(100)]
    assert step(more, [engine.new_sequence() for _ in more], [0, 0]) == latent_layers and engine._ctx.from_start
    many = [tokens(64)] + [tokens(8) for _ in range(20)]
    others = [engine.new_sequence() for _ in many]
    assert step(many, others, [0] * len(many)) == 0 and engine._ctx.from_start
    assert step([row + tokens(1) for row in many], others, [len(row) for row in many]) == 0
