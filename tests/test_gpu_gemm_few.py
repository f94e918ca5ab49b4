"""The product for few tokens (csrc/gemm_few.cu): every epilogue against a plain float statement, at the edges of its ranges: one
token, a full and a begun second tile of eight, widths that end inside a block of rows, K of one element group to many turns."""
import pytest
import torch

import plain_qwen3 as plain
from qwen_triton_b200.ops import kernels
from test_gpu_gemm_fused import product, scaled_rows
from test_gpu_kernels import DEV, PAGE, close, paged, rand

pytestmark = pytest.mark.gpu
BF16 = torch.bfloat16
FORMS = [(16, 8), (32, 8), (32, 16), (16, 16)]


@pytest.mark.parametrize("rows, n, k", [(1, 503, 96), (8, 4096, 1024), (16, 130, 512), (9, 33, 2064), (3, 15, 16), (5, 128, 4112), (1, 1024, 3072)])
@pytest.mark.parametrize("few", FORMS)
@pytest.mark.parametrize("out_dtype", [torch.float32, BF16])
def test_store(rows, n, k, few, out_dtype):
    x, w = rand(rows, k, seed=1, dtype=BF16), rand(n, k, seed=2, scale=0.05, dtype=BF16)
    bias = rand(n, seed=9)
    out = torch.full((rows, n), float("nan"), dtype=out_dtype, device=DEV)
    kernels.gemm_fused_store(x, w, out, bias=bias, few=few)
    close(out, product(x, w) + bias.cpu(), BF16, "plain product")
    handed, factor = scaled_rows(rows, k, seed=3)
    kernels.gemm_fused_store(handed, w, out, few=few)
    close(out, product(handed.tensor, w) * factor, BF16, "with the deferred norm factor")


@pytest.mark.parametrize("rows, n, k", [(1, 1024, 2048), (8, 4096, 12288), (16, 136, 512), (11, 20, 160), (4, 96, 48)])
@pytest.mark.parametrize("few", FORMS)
def test_residual_add_and_norm_preparation(rows, n, k, few):
    x, w = rand(rows, k, seed=4, dtype=BF16), rand(n, k, seed=5, scale=0.05, dtype=BF16)
    stream = rand(rows, n, seed=6)
    expected = stream.cpu() + product(x, w)
    residual = stream.clone()
    assert kernels.gemm_fused_residual(x, w, residual, few=few) is None
    torch.testing.assert_close(residual.cpu(), expected, atol=2e-3, rtol=2e-3)          # float sums of bfloat16 products
    residual = stream.clone()
    g = 1.0 + rand(n, seed=7, scale=0.2)
    xw = torch.full((rows, n), float("nan"), dtype=BF16, device=DEV)
    sq = torch.full((-(-n // few[0]), rows), float("nan"), device=DEV)
    handed = kernels.gemm_fused_residual(x, w, residual, g, 3e-6, xw, sq, few=few)
    torch.testing.assert_close(residual.cpu(), expected, atol=2e-3, rtol=2e-3)
    close(handed.tensor, residual.cpu() * g.cpu(), BF16, "weighted stream")
    torch.testing.assert_close(handed.sq.sum(0).cpu(), residual.pow(2).sum(-1).cpu(), atol=1e-3, rtol=1e-4)


@pytest.mark.parametrize("rows, inter, k", [(1, 48, 80), (8, 3072, 1024), (16, 560, 512), (13, 16, 4096)])
@pytest.mark.parametrize("warps", [8, 16])
def test_gate(rows, inter, k, warps):
    gate, up = rand(inter, k, seed=9, scale=0.1, dtype=BF16), rand(inter, k, seed=10, scale=0.1, dtype=BF16)
    w = kernels.interleave_gate_up(gate, up, kernels.SWIGLU_GROUP)
    handed, factor = scaled_rows(rows, k, seed=11)
    out = torch.full((rows, inter), float("nan"), dtype=BF16, device=DEV)
    kernels.gemm_fused_swiglu(handed, w, out, few=(32, warps))
    g, u = product(handed.tensor, gate) * factor, product(handed.tensor, up) * factor
    close(out, g * torch.sigmoid(g) * u, BF16, "silu(gate) * up")


@pytest.mark.parametrize("nq, nkv, d, rotary, ring, own_kv, rows", [(8, 2, 16, 16, 128, True, 3), (5, 1, 128, 128, 0, True, 1), (3, 3, 64, 32, 0, True, 16),
                                                                    (6, 2, 32, 24, 0, True, 9), (7, 1, 64, 64, 0, False, 6), (16, 8, 128, 128, 0, True, 8)])
@pytest.mark.parametrize("interleaved", [False, True])
@pytest.mark.parametrize("warps", [8, 16])
def test_qkv_equals_the_product_for_more_tokens(nq, nkv, d, rotary, ring, own_kv, rows, interleaved, warps):
    """The same epilogue behind the same product by csrc/gemm_fused.cu, which test_gpu_gemm_fused.py holds to a plain statement."""
    k, eps, past = 512, 1e-5, [(130 + 37 * i) % 300 for i in range(rows)]
    n = (nq + (2 * nkv if own_kv else 0)) * d
    w = rand(n, k, seed=12, scale=0.08, dtype=BF16)
    handed, _ = scaled_rows(rows, k, seed=13)
    qw, kw = 1.0 + rand(d, seed=14, scale=0.2), 1.0 + rand(d, seed=15, scale=0.2)
    cos, sin = plain.rope_tables(torch.arange(400), rotary, 50000.0, torch.float32)
    cos_sin = torch.cat((cos, sin), dim=-1).contiguous().to(DEV)
    seq, pos = torch.arange(rows, dtype=torch.int32, device=DEV), torch.tensor(past, dtype=torch.int32, device=DEV)
    zeros = [torch.zeros(p + 1, nkv, d) for p in past]
    results = []
    for few in (None, (32, warps)):
        k_cache, v_cache, table = paged(zeros, zeros, [p + 1 for p in past], BF16, ring_tokens=ring, seed=16, garbage=False)
        q_out = torch.full((rows, nq, d), float("nan"), dtype=BF16, device=DEV)
        kernels.gemm_fused_qkv(handed, w, q_out, k_cache, v_cache, seq, pos, table, qw, kw, eps, cos_sin, nq, nkv, d, PAGE, ring,
                               write_kv=own_kv, interleaved=interleaved, few=few)
        results.append((q_out.float().cpu(), k_cache.float().cpu(), v_cache.float().cpu()))
    for want, got, name in zip(*results, ("q", "k", "v")):
        close(got, want, BF16, name)


def test_what_it_refuses():
    x, w, out = rand(4, 64, seed=1, dtype=BF16), rand(256, 64, seed=2, dtype=BF16), torch.empty(4, 256, device=DEV)
    with pytest.raises(kernels.KernelError, match="up to 16 tokens"):
        kernels.gemm_fused_store(rand(17, 64, seed=1, dtype=BF16), w, torch.empty(17, 256, device=DEV), few=(32, 8))
    with pytest.raises(kernels.KernelError, match="32-byte"):
        kernels.gemm_fused_store(rand(4, 72, seed=1, dtype=BF16), rand(256, 72, seed=2, dtype=BF16), out, few=(32, 8))
    with pytest.raises(kernels.KernelError, match="rows for epilogue"):
        kernels.gemm_fused_swiglu(x, w, torch.empty(4, 128, dtype=BF16, device=DEV), few=(16, 8))
    assert not kernels.few_supported(torch.empty(5 * 64 + 8, dtype=BF16, device=DEV)[8:].view(5, 64), w)
    assert not kernels.few_supported(rand(4, 72, seed=1, dtype=BF16), rand(256, 72, seed=2, dtype=BF16))
