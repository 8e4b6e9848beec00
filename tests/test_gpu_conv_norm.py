"""Convolution, q/k norms and gates of a prompt in one pass against the two operators it stands for: odd numbers of heads, runs of
eight tokens cut by the end and by sequence borders, sequences of one token."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("heads", [1, 3, 16])
@pytest.mark.parametrize("lengths", [[1], [7, 1, 2, 30], [8, 3, 1, 1, 19, 500]])
def test_conv_norm_gates(heads, lengths):
    from b200attn import engine, ops
    gen, total, kd = torch.Generator().manual_seed(heads), sum(lengths), heads * 128
    x = torch.randn(total, 4 * kd + 8 * heads, generator=gen).bfloat16().to(DEV)
    weight = torch.randn(3 * kd, 4, generator=gen).bfloat16().to(DEV)
    a_log, dt_bias = torch.rand(heads, generator=gen).to(DEV), torch.randn(heads, generator=gen).bfloat16().to(DEV)
    start = torch.tensor([sum(lengths[:i]) for i, n in enumerate(lengths) for _ in range(n)], dtype=torch.int32, device=DEV)
    if len(lengths) > 1:                     # what a neighbour holds never counts
        x[lengths[0]: lengths[0] + 1] = float("nan")
    qkv, a, b = x[:, : 3 * kd], x[:, 4 * kd: 4 * kd + heads], x[:, 4 * kd + heads: 4 * kd + 2 * heads]
    got = ops.gdn_conv_norm_gates(qkv, weight, start, a, b, a_log, dt_bias)
    q, k, v = engine._conv4_prefill(qkv, weight, start).view(total, 3, heads, 128).unbind(1)
    q_n, k_n, beta, g = engine._qk_norm_gates(q, k, a, b, a_log, dt_bias)
    for name, have, want in zip(("q", "k", "v", "beta", "g"), got, (q_n, k_n, v, beta, g)):
        assert have.shape == want.shape
        # the same operations; the norm's sum may run in another order: half an ulp of bf16 either way
        assert torch.allclose(have.float(), want.float(), rtol=2.0 ** -7 if name in "qk" else 0.0, atol=0.0, equal_nan=True), name


def test_conv_norm_gates_refuses_ragged_rows():
    from b200attn import ops
    x = torch.randn(5, 4 * 128 + 2, device=DEV).bfloat16()
    start = torch.zeros(5, dtype=torch.int32, device=DEV)
    weight, dt_bias = torch.zeros(384, 4, dtype=torch.bfloat16, device=DEV), torch.zeros(1, dtype=torch.bfloat16, device=DEV)
    assert ops.gdn_conv_norm_gates(x[:, :384], weight, start, x[:, 512:513], x[:, 513:], torch.zeros(1, device=DEV), dt_bias) is None


@pytest.mark.parametrize("heads", [1, 3, 16])
@pytest.mark.parametrize("lengths", [[1], [7, 1, 2, 30], [8, 3, 4, 0, 5, 500]])
def test_conv_norm_gates_leaves_the_state(heads, lengths):
    """The last four inputs of every sequence, zeros in front of short ones, in the same launch; the other results stay the same bits."""
    from b200attn import engine, ops
    gen, total, kd = torch.Generator().manual_seed(heads), sum(lengths), heads * 128
    x = torch.randn(total, 3 * kd + 8 * heads, generator=gen).bfloat16().to(DEV)
    weight, gates = torch.randn(3 * kd, 4, generator=gen).bfloat16().to(DEV), torch.randn(2, total, heads, generator=gen).bfloat16().to(DEV)
    a_log, dt_bias = torch.rand(heads, generator=gen).to(DEV), torch.randn(heads, generator=gen).bfloat16().to(DEV)
    start = torch.tensor([sum(lengths[:i]) for i, n in enumerate(lengths) for _ in range(n)], dtype=torch.int32, device=DEV)
    cu = torch.tensor([sum(lengths[:i]) for i in range(len(lengths) + 1)], dtype=torch.int32, device=DEV)
    args = (x[:, : 3 * kd], weight, start, gates[0], gates[1], a_log, dt_bias)
    have, want = (torch.full((len(lengths), 4, 3 * kd), 7.0, dtype=torch.bfloat16, device=DEV) for _ in range(2))
    got = ops.gdn_conv_norm_gates(*args, cu, have)
    engine._conv_state_pack(want, args[0], cu)
    assert torch.equal(have, want)
    assert all(torch.equal(g, w) for g, w in zip(got, ops.gdn_conv_norm_gates(*args)))
