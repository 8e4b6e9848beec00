"""Weight-streaming products by the number of batch rows: groups of 8, 16 and 32 rows at their borders, both K forms, plain and SwiGLU and
arg-max, launched plainly and early.  Bound: fp32 sums of exact products in another order (K 2^-24 of the sum of magnitudes, far below)
and one rounding to bf16: half an ulp, 2^-9 of the value, taken as 2^-8 of the largest."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _case(m, n, k):
    gen = torch.Generator().manual_seed(m * 7 + n + k)
    x = torch.randn(m, k, generator=gen).to(torch.bfloat16).to(DEV)
    return x, (torch.randn(n, k, generator=gen) * 0.05).to(torch.bfloat16).to(DEV)


@pytest.mark.parametrize("m", [1, 2, 7, 8, 9, 15, 16, 17, 24, 32])
@pytest.mark.parametrize("n,k", [(8, 128), (136, 1024), (9480, 1280), (24, 1536), (1024, 3584), (2400, 4096)])
def test_rows(m, n, k):
    from b200attn import ops
    x, w = _case(m, n, k)
    ref = x.double() @ w.double().t()
    for flags in (0, ops.OVERLAP_START):
        y = ops.skinny_gemm(x, w, overlap=flags)
        assert (y.double() - ref).abs().max().item() <= 2.0 ** -8 * ref.abs().max().item()


@pytest.mark.parametrize("m", [1, 8, 9, 16, 17])
def test_rows_swiglu_and_argmax(m):
    from b200attn import ops
    x, w = _case(m, 2 * 360, 1024)
    y = ops.skinny_gemm(x, w, swiglu=True, overlap=ops.OVERLAP_START)
    assert torch.equal(y, ops.swiglu_fused(ops.skinny_gemm(x, w), 360))
    x, w = _case(m, 20008, 640)
    ids = ops.lm_head_argmax(x, w, ops.argmax_workspace(DEV), overlap=ops.OVERLAP_START)
    logits = x.double() @ w.double().t()
    best = logits.gather(1, ids.view(-1, 1)).squeeze(1)
    assert bool((logits.max(1).values - best <= 1e-4).all())       # fp32 sums: ties up to their rounding


@pytest.mark.parametrize("m", [2, 9, 20])
@pytest.mark.parametrize("k", [256, 2048])
def test_rows_over_one_another(m, k):
    """Rows that share their memory, and one row of any stride: X goes through a tensor map of its strides."""
    from b200attn import ops
    x, w = _case(1, 72, k)
    wide = torch.empty(m, 3 * k, dtype=torch.bfloat16, device=DEV).copy_(x.repeat(1, 3))
    want = ops.skinny_gemm(x.repeat(m, 1), w)
    for rows in (x.expand(m, k), wide[:, k: 2 * k], torch.as_strided(wide, (m, k), (8 * 3 * k // 8, 1), 2 * k)):
        assert torch.equal(ops.skinny_gemm(rows, w), want)
    assert torch.equal(ops.skinny_gemm(torch.as_strided(wide, (1, k), (16, 1), k), w), want[:1])
