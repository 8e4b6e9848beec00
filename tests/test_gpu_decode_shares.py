"""Decode attention at the borders of what its prologue and merges tell apart: up to and beyond 32 sequences (lengths in the lanes of every
warp, or in shared memory), clusters of 16, 8, 4 and 2 CTAs, and segments shorter than a cluster has CTAs, or a CTA warps, so that
states without a page are merged.  bf16 keeps eight bits: a rounding moves a value by at most 2^-8 of itself."""
import pytest
import torch

from b200attn.synthetic import make_paged_case, rope_inv_freq
from oracle import reference_ops as O

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("lengths", [[1], [16, 17], [2000], [5, 900, 33], [300] * 9, [40, 700] * 8, list(range(1, 32)), [64] * 32, [33, 1, 500] * 11,
                                     [17] * 70])
@pytest.mark.parametrize("partition", [0, 1, 3])
def test_shares(lengths, partition):
    from b200attn import load, ops
    if partition == 3 and 2 * len(lengths) > 64:
        pytest.skip("clusters take up to 64 segments")
    c, inv = make_paged_case(lengths, seed=len(lengths)), rope_inv_freq()
    d = {k: (v.to(DEV) if isinstance(v, torch.Tensor) else v) for k, v in c.items()}
    kc, vc = d["k_cache"].clone(), d["v_cache"].clone()
    out = ops.fused_decode_attention(d["q"], d["k_new"], d["v_new"], d["gate"], kc, vc, d["block_table"], d["pos"], inv.to(DEV), 64,
                                     ops.fused_decode_workspace(DEV), partition=partition)
    torch.cuda.synchronize()
    assert load().b200_wait_timed_out() == 0
    kr, vr = c["k_cache"].clone(), c["v_cache"].clone()
    ref = O.fused_decode_attention(c["q"], c["k_new"], c["v_new"], c["gate"], kr, vr, c["block_table"], c["pos"], inv, 64, exact=True)
    assert torch.equal(vc.cpu(), vr)
    # some way below what roundings (p, context, output) could add up to; what it lets through is the next test's
    assert (out.float().cpu() - ref.float()).abs().max().item() <= 2 ** -7 * max(c["v_cache"].float().abs().max(), c["v_new"].float().abs().max()).item()


def _exact(c, kr, vr):
    """Exact gated output, and what rounding may move each element by: p (2^-8 of each weight), context and output (2^-8 each), fp32 scores and
    sigmoid (2^-12)."""
    lengths = (c["pos"] + 1).tolist()
    ctx, spread = (O.paged_decode_exact(c["q"], kr, values, c["block_table"], lengths) for values in (vr, vr.abs()))
    factor = torch.sigmoid(c["gate"].float()).view(ctx.shape)
    bound = 1.01 * factor * ((2 ** -8 + 2 ** -12) * spread + 2 * 2 ** -8 * ctx.abs()) + 1e-6
    return ctx, factor, bound


@pytest.mark.parametrize("lengths", [[2000], [500, 700, 900], [2000, 40, 1300, 9], [300] * 9, [33, 1, 500] * 11, [1926, 700] * 20])
@pytest.mark.parametrize("partition", [0, 1, 3])
def test_every_element(lengths, partition):
    """Element by element, which an output without one of the pages does not pass (checked here on the oracle).  Frequencies of zero: both
    sides rotate by nothing."""
    from b200attn import load, ops
    if partition == 3 and 2 * len(lengths) > 64:
        pytest.skip("clusters take up to 64 segments")
    c, inv = make_paged_case(lengths, seed=7 + len(lengths)), torch.zeros(32)
    d = {k: (v.to(DEV) if isinstance(v, torch.Tensor) else v) for k, v in c.items()}
    kc, vc = d["k_cache"].clone(), d["v_cache"].clone()
    out = ops.fused_decode_attention(d["q"], d["k_new"], d["v_new"], d["gate"], kc, vc, d["block_table"], d["pos"], inv.to(DEV), 64,
                                     ops.fused_decode_workspace(DEV), partition=partition)
    torch.cuda.synchronize()
    assert load().b200_wait_timed_out() == 0
    kr, vr = c["k_cache"].clone(), c["v_cache"].clone()
    O.paged_kv_append(kr, vr, c["k_new"], c["v_new"], c["block_table"], c["pos"])
    ctx, factor, bound = _exact(c, kr, vr)
    off = (out.float().cpu().view(ctx.shape) - ctx * factor).abs()
    assert (off <= bound).all()
    if partition == 0:
        n, row = int(c["pos"][0]) + 1, c["block_table"][0]
        k, v = (torch.cat([t[int(page)] for page in row[: -(-n // 16)]], dim=1)[:, :n].float() for t in (kr, vr))   # [kv head, token, 256]
        p = torch.exp((c["q"][0].float().view(2, 4, 256) @ k.transpose(1, 2)) / 16)
        for first in range(0, n // 16 * 16, 16):
            w = p.clone()
            w[:, :, first: first + 16] = 0
            lost = ((w / w.sum(-1, keepdim=True)) @ v).view(8, 256) * factor[0]
            assert ((lost - ctx[0] * factor[0]).abs() > bound[0]).any()
