"""The CTA-pair prefill attention where its tiles, pairs and items can go wrong: sequences around 8 (output tile), 32 (CTA), 64 (pair)
and 128 (key tile) tokens, more sequences than one read of their lengths covers, more items than a pair's ring holds, row maxima
that grow from tile to tile, and rows behind a sequence that must not be touched.

Bounds: bf16 keeps eight bits, so that a rounding moves a value by at most 2^-8 of itself.  An output element is off by at most 2^-8 sum p |v|
(rounding of the weights p) + 2^-8 |out| (its own) and what fp32 sums make of the scores: 2^-12 sum p |v| for products of unit size, where the
256 terms of a score sum up to some 10 in magnitude.  All elements together stay within 2^-8 max|v|, the gated form, which rounds once, and the
chain, which rounds twice more, within 2^-7 max|v| of one another.
"""
import pytest
import torch

from helpers import bf16_randn, cdiv, rope_inv_freq
from oracle import reference_ops as O

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _qkv(lengths, seed, kv_heads=2):
    gen, total = torch.Generator().manual_seed(seed), sum(lengths)
    cu = torch.tensor([0, *torch.tensor(lengths).cumsum(0).tolist()], dtype=torch.int32)
    return [bf16_randn(total, n, 256, gen=gen) for n in (4 * kv_heads, kv_heads, kv_heads)] + [cu, gen]


def _bounds(q, k, v, cu, scores=2 ** -12):
    """The exact output, and what rounding may move each element by."""
    exact, spread = O.varlen_causal_exact(q, k, v, cu).float(), O.varlen_causal_exact(q, k, v.abs(), cu).float()
    return exact, 1.01 * ((2 ** -8 + scores) * spread + 2 ** -8 * exact.abs()) + 1e-6


def _check(out, q, k, v, cu, scores=2 ** -12):
    import b200attn
    torch.cuda.synchronize()
    assert b200attn.load().b200_wait_timed_out() == 0
    exact, bound = _bounds(q, k, v, cu, scores)
    off = (out.float().cpu() - exact).abs()
    assert (off <= bound).all()
    assert off.max().item() <= 2 ** -8 * v.float().abs().max().item() + 1e-3


RAGGED = [int(x) for x in torch.randint(1, 200, (130,), generator=torch.Generator().manual_seed(9))]


@pytest.mark.parametrize("lengths", [[1], [8, 7, 9], [31, 32, 33, 40], [63, 64, 65, 72], [96, 97, 127, 128, 129], [191, 192, 193, 256, 257],
                                     RAGGED, [5] * 33, [640, 1, 320]])
@pytest.mark.parametrize("kv_heads", [2, 1])
def test_pairs_vs_oracle(lengths, kv_heads):
    from b200attn import ops
    q, k, v, cu, _ = _qkv(lengths, 11 + len(lengths), kv_heads)
    out = ops.gqa_attention_varlen_causal(q.to(DEV), k.to(DEV), v.to(DEV), cu.to(DEV), max(lengths))
    _check(out, q, k, v, cu)


def test_row_maxima_that_grow():
    """Every later key tile outweighs the ones before it by far more than the 2^8 a reference maximum may lag: O is rescaled, by both
    parities, and the sums of even and odd tiles stand against different references."""
    from b200attn import ops
    q, k, v, cu, _ = _qkv([700, 300], 5)
    q = q.abs()
    k = (k.abs() * (1 + 2 * (torch.arange(1000) // 128)).view(-1, 1, 1)).to(torch.bfloat16)
    out = ops.gqa_attention_varlen_causal(q.to(DEV), k.to(DEV), v.to(DEV), cu.to(DEV), 700)
    _check(out, q, k, v, cu, scores=2 ** -9)                                # terms up to eleven times as large


@pytest.mark.parametrize("lengths", [[3], [64, 33, 8, 129], RAGGED[:70]])
def test_gated_form_vs_chain(lengths):
    from b200attn import ops
    q, k, v, cu, gen = _qkv(lengths, 21)
    gate = bf16_randn(sum(lengths), 2048, gen=gen).to(DEV)
    q, k, v, cu = (t.to(DEV) for t in (q, k, v, cu))
    batch, pps = len(lengths), cdiv(max(lengths), 16)
    table = torch.randperm(batch * pps, generator=gen).view(batch, pps).to(torch.int32).to(DEV)
    ids = torch.cat([torch.arange(n) for n in lengths]).to(torch.int32).unsqueeze(0).to(DEV)
    inv = rope_inv_freq().to(DEV)
    caches = ops.allocate_paged_kv_cache(batch * pps, 2, 256, device=DEV)
    fused = ops.fused_prefill_attention(q, k, v, gate, *caches, table, cu, ids, inv, 64, max(lengths))
    qr, kr = (ops.partial_rope(t.unsqueeze(0).permute(0, 2, 1, 3), ids, inv, 64)[0].permute(1, 0, 2).contiguous() for t in (q, k))
    ctx = ops.gqa_attention_varlen_causal(qr, kr, v, cu, max(lengths)).permute(1, 0, 2).unsqueeze(0)
    chain = ops.attention_gate_pack(ctx, gate.view(1, -1, 8, 256).permute(0, 2, 1, 3))
    assert (fused.float() - chain.float()).abs().max().item() <= 2 ** -7 * v.float().abs().max().item()


def test_rows_behind_a_sequence_stay():
    """Sequences that end before the packed rows do: the output rows behind them are left alone (no tile of eight tokens is stored over
    a sequence's end)."""
    from b200attn import _lib, ops
    q, k, v, cu, _ = _qkv([13, 70], 31)
    q, k, v, cu = (t.to(DEV) for t in (q, k, v, cu))
    for ends in ([0, 13, 83], [0, 5, 60]):
        cu = torch.tensor(ends, dtype=torch.int32, device=DEV)
        out = torch.full_like(q, 7.0)
        _lib.call("b200_gqa_varlen_causal", q.data_ptr(), q.stride(0), q.stride(1), k.data_ptr(), k.stride(0), k.stride(1), v.data_ptr(), v.stride(0),
                  v.stride(1), out.data_ptr(), out.stride(0), out.stride(1), cu.data_ptr(), 2, 83, 70, 8, 2, 256, torch.cuda.current_stream().cuda_stream)
        _check(out[: ends[-1]], *(t[: ends[-1]].cpu() for t in (q, k, v)), cu.cpu())
        assert bool((out[ends[-1]:] == 7.0).all())


@pytest.mark.parametrize("lengths,longest", [([1 + n % 40 for n in range(190)] + [700] + [7] * 230, 5000), ([0] * 200 + [90] + [0] * 191 + [64, 65] + [0] * 33, 4096),
                                             ([33] * 192 + [129], 129)])
def test_items_of_many_sequences(lengths, longest):
    """More sequences than the items are dealt out of at a time, most of them short or empty, and a longest length far above any."""
    from b200attn import ops
    q, k, v, cu, _ = _qkv(lengths, 41, 1)
    out = ops.gqa_attention_varlen_causal(q.to(DEV), k.to(DEV), v.to(DEV), cu.to(DEV), longest)
    _check(out, q, k, v, cu)


@pytest.mark.parametrize("lengths", [[1000 - 17 * n for n in range(50)], [257] * 130, [2048] * 20])
def test_groups_beyond_the_l2(lengths):
    """Batches whose items are dealt in groups of sequences against their halves: an item is computed alike in whatever order it comes."""
    from b200attn import ops
    g, half = torch.Generator(device=DEV).manual_seed(3), len(lengths) // 2
    x = torch.randn((sum(lengths), 12, 256), generator=g, device=DEV, dtype=torch.bfloat16)

    def attend(lengths, x):
        cu = torch.tensor([0, *torch.tensor(lengths).cumsum(0).tolist()], dtype=torch.int32, device=DEV)
        return ops.gqa_attention_varlen_causal(x[:, :8], x[:, 8:10], x[:, 10:], cu, max(lengths))

    cut = sum(lengths[:half])
    out = attend(lengths, x)
    assert torch.equal(out[:cut], attend(lengths[:half], x[:cut])) and torch.equal(out[cut:], attend(lengths[half:], x[cut:]))
    assert bool(out.isfinite().all())


# Beside four long sequences, which make a call more than one wave of CTAs, the lengths above meet the pairs' tiles; by themselves they are
# the one-CTA kernel's.
@pytest.mark.parametrize("lengths", [[1], [8, 7, 9], [31, 32, 33, 40], [63, 64, 65, 72], [96, 97, 127, 128, 129], [191, 192, 193, 256, 257]])
@pytest.mark.parametrize("kv_heads", [2, 1])
def test_edges_on_pairs(lengths, kv_heads):
    from b200attn import ops
    lengths = [1100, 1300] + lengths + [1200, 1170]
    q, k, v, cu, _ = _qkv(lengths, 51 + len(lengths), kv_heads)
    out = ops.gqa_attention_varlen_causal(q.to(DEV), k.to(DEV), v.to(DEV), cu.to(DEV), max(lengths))
    _check(out, q, k, v, cu)


@pytest.mark.parametrize("lengths", [[1], [32] * 74, [32] * 75, [31, 33], [128] * 16, [129] * 14, [2048], [2960], [2961], [4096], [4145], [1000, 1, 300], [512, 3, 64, 200, 77, 1, 1, 400]])
@pytest.mark.parametrize("longest", [0, 333])
def test_short_calls(lengths, longest):
    """Calls on both sides of the line to the one-CTA kernel: one CTA and one wave of them, one tile and many, longest lengths that say too much."""
    from b200attn import ops
    q, k, v, cu, _ = _qkv(lengths, 61 + len(lengths))
    out = ops.gqa_attention_varlen_causal(q.to(DEV), k.to(DEV), v.to(DEV), cu.to(DEV), max(lengths) + longest)
    _check(out, q, k, v, cu)


@pytest.mark.parametrize("lengths", [[700, 300], [1200, 1100, 900, 700, 650, 600]])
def test_bounds_catch_a_lost_tile(lengths):
    """On the CPU: an output without one of the 128-token key tiles, or with a tile counted twice, is outside the bounds in every long row."""
    q, k, v, cu, _ = _qkv(lengths, 71)
    exact, bound = _bounds(q, k, v, cu)
    n, (q, k, v) = lengths[0], (t[: lengths[0]].float() for t in (q, k, v))
    p = torch.exp((q[n - 1].view(2, 4, 256) @ k.permute(1, 2, 0)) / 16)     # weights of the last row, [kv head, head, token]
    for tile in range(n // 128):
        for factor in (0.0, 2.0):
            w = p.clone()
            w[:, :, tile * 128: tile * 128 + 128] *= factor
            out = ((w / w.sum(-1, keepdim=True)) @ v.permute(1, 0, 2)).view(8, 256)
            assert ((out - exact[n - 1]).abs() > bound[n - 1]).any(1).all()


@pytest.mark.parametrize("lengths", [[40, 9], [300, 45], [1100] * 5])
def test_gates_far_from_zero(lengths):
    """Gates of -12 to 12 against the exact sigmoid.  o/2 tanh(g/2) + o/2 with the hardware's tanh, off by 2^-11 of itself, is off by 2^-12 |o| at
    most, however small the sigmoid: an absolute error, of what the gate lets through where it is open."""
    from b200attn import ops
    q, k, v, cu, gen = _qkv(lengths, 81)
    total, batch, pps = sum(lengths), len(lengths), cdiv(max(lengths), 16)
    gate = ((torch.rand(total, 2048, generator=gen) * 24 - 12)).to(torch.bfloat16)
    table = torch.randperm(batch * pps, generator=gen).view(batch, pps).to(torch.int32).to(DEV)
    ids = torch.zeros(1, total, dtype=torch.int32, device=DEV)              # no rotation
    caches = ops.allocate_paged_kv_cache(batch * pps, 2, 256, device=DEV)
    out = ops.fused_prefill_attention(q.to(DEV), k.to(DEV), v.to(DEV), gate.to(DEV), *caches, table, cu.to(DEV), ids, rope_inv_freq().to(DEV), 64,
                                      max(lengths)).float().cpu().view(total, 8, 256)
    exact, bound = _bounds(q, k, v, cu)
    factor = torch.sigmoid(gate.double()).float().view(total, 8, 256)
    assert ((out - exact * factor).abs() <= bound * factor + 2 ** -12 * 1.01 * (exact.abs() + bound) + 1e-6).all()
