"""Products around a residual add and RMSNorm without a launch between them: skinny_gemm_join, then skinny_gemm_normed (plain, SwiGLU) or
lm_head_argmax, against skinny_gemm and 64 bits."""
import pytest
import torch

pytestmark = pytest.mark.gpu
EPS = 1e-6


def _rows(m, n, k, seed, scale=1.0):
    g = torch.Generator().manual_seed(seed)
    make = lambda *shape: torch.randn(shape, generator=g).to("cuda", torch.bfloat16)   # noqa: E731
    return make(m, k), make(n, k) * k ** -0.5, make(m, n) * scale, make(n) * 0.1


@pytest.mark.parametrize("n,k", [(128, 1536), (1024, 2048), (1024, 3584), (1280, 4096)])
@pytest.mark.parametrize("m", [1, 8, 9, 16, 17, 32])
def test_join_and_normed(m, n, k):
    from b200attn import ops

    x, w, residual, gain = _rows(m, n, k, 100 * m + k)
    if m > 1:
        residual[1] *= 1e4                                   # far from unit size: the factor of its row is far from one
    plain = ops.skinny_gemm(x, w)
    want = plain + residual
    total, scaled, squares = ops.skinny_gemm_join(x, w, residual, gain)
    assert torch.equal(total, want)                          # the same roundings: product, then sum
    assert torch.equal(scaled, (total.float() * (1 + gain.float())).bfloat16())
    s64 = total.double()
    exact = s64.square().view(m, n // 16, 16).sum(-1)
    assert ((squares.double() - exact).abs() <= 16 * 2.0 ** -24 * exact).all()

    up = torch.randn((2 * 80, n), generator=torch.Generator().manual_seed(k)).to("cuda", torch.bfloat16) * n ** -0.5
    rms = torch.rsqrt(s64.square().mean(-1, keepdim=True) + EPS)
    y64 = (scaled.double() @ up.double().T) * rms
    bound = ((scaled.double().abs() @ up.double().abs().T) * rms) * (n * 2.0 ** -24)   # fp32 sums of n products
    y = ops.skinny_gemm_normed(scaled, squares, up, EPS)
    assert ((y.double() - y64).abs() <= bound + 2.0 ** -8 * y64.abs()).all()
    # silu(g) u of the rounded halves: each off by at most 2^-8 of itself and the bound, silu's slope is below 1.1
    act = ops.skinny_gemm_normed(scaled, squares, up, EPS, swiglu=True)
    a, b = y64[:, :80], y64[:, 80:]
    da, db = bound[:, :80] + 2.0 ** -8 * a.abs(), bound[:, 80:] + 2.0 ** -8 * b.abs()
    act64 = torch.nn.functional.silu(a) * b
    assert ((act.double() - act64).abs() <= 1.1 * da * b.abs() + torch.nn.functional.silu(a).abs() * db + 1.1 * da * db + 2.0 ** -8 * act64.abs() + 1e-6).all()

    table = torch.randn((4096, n), generator=torch.Generator().manual_seed(n)).to("cuda", torch.bfloat16)
    ids = ops.lm_head_argmax(scaled, table, ops.argmax_workspace())
    logits = (scaled.double() @ table.double().T) * rms
    slack = 2 * (scaled.double().abs() @ table.double().abs().T).amax(-1) * rms[:, 0] * (n * 2.0 ** -24)
    assert (logits.gather(1, ids[:, None])[:, 0] >= logits.amax(-1) - slack).all()


def test_rows_keep_to_themselves():
    """Zero rows come out as zeros; a NaN or an overflowing row changes no other."""
    from b200attn import ops

    x, w, residual, gain = _rows(20, 1024, 2048, 7)
    up = torch.randn((64, 1024), generator=torch.Generator().manual_seed(1)).to("cuda", torch.bfloat16)
    total, scaled, squares = ops.skinny_gemm_join(x, w, residual, gain)
    clean = ops.skinny_gemm_normed(scaled, squares, up, EPS)
    x[3], residual[3] = 0, 0
    residual[5, 17] = float("nan")
    residual[6] = 2.0 ** 100                                 # its squares overflow: normed rows of zeros, as the norm by itself has them
    total, scaled, squares = ops.skinny_gemm_join(x, w, residual, gain)
    y = ops.skinny_gemm_normed(scaled, squares, up, EPS)
    assert (y[3] == 0).all() and y[5].isnan().all() and (y[6] == 0).all()
    others = [r for r in range(20) if r not in (3, 5, 6)]
    assert torch.equal(y[others], clean[others])


def test_shapes_refused():
    from b200attn import ops

    for m, n, k in ((33, 1024, 2048), (8, 1024, 1280), (8, 1024, 4352), (8, 2048, 2048), (8, 1032, 2048), (8, 1024, 2176)):
        assert not ops.skinny_gemm_joins(m, n, k)


@pytest.mark.parametrize("m,streams,parts,k", [(1, 2, 0, 2048), (8, 1, 1, 1536), (9, 4, 2, 3584), (32, 2, 1, 4096), (17, 3, 0, 1536)])
def test_hyper_join(m, streams, parts, k, n=1024):
    """Against the product and hyper_connect in two launches: the streams are the same bits, the rows times 1 / rms the same values."""
    from b200attn import hybrid_ops as hops
    from b200attn import ops

    true_n = n - 40
    x, w, _, gain = _rows(m, n, 2 * k, m + k)
    x, w = x[:, k:].contiguous(), w[:, :k]                    # a column range
    g = torch.Generator().manual_seed(k)
    state = torch.randn((m, streams, n), generator=g).to("cuda")
    weights = torch.rand(streams * streams + 2 * streams + 1, generator=g).to("cuda")
    state[:, :, true_n:], w[true_n:] = 0, 0                   # padding columns
    earlier = torch.randn((parts, m, n), generator=g).to("cuda", torch.bfloat16) if parts else None
    gains = gain.float() + 1 if parts else None
    y = torch.empty((m, n), dtype=torch.bfloat16, device="cuda")
    ops.skinny_gemm_part(x, w, y)
    if parts:
        earlier[:, :, true_n:] = 0
        y = torch.cat((earlier, y[None]))
    want_state, have_state = state.clone(), state.clone()
    want = hops.hyper_connect(want_state, weights, true_n, EPS, torch.bfloat16, y=y, gains=gains)
    rows = hops.hyper_join(x, w, have_state, weights, gains, earlier)
    assert torch.equal(have_state, want_state)
    rms = torch.rsqrt(rows.squares.double().sum(-1, keepdim=True) / true_n + EPS)
    # either is rounded to bf16 once
    assert ((rows.scaled.double() * rms - want.double()).abs() <= 2.0 ** -7 * want.double().abs() + 1e-30).all()
    up = torch.randn((64, n), generator=g).to("cuda", torch.bfloat16) * n ** -0.5
    y64 = (rows.scaled.double() @ up.double().T) * rms
    bound = ((rows.scaled.double().abs() @ up.double().abs().T) * rms) * (n * 2.0 ** -24)
    got = ops.skinny_gemm_normed(*rows, up, EPS, width=true_n)
    assert ((got.double() - y64).abs() <= bound + 2.0 ** -8 * y64.abs()).all()
