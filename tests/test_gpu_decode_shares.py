"""Decode attention at the borders of what its prologue and merges tell apart: up to and beyond 32 sequences (lengths in the lanes of every
warp, or in shared memory), clusters of 16, 8, 4 and 2 CTAs, and segments shorter than a cluster has CTAs, or a CTA warps, so that
states without a page are merged.  Bound: p is rounded to bf16 (2^-9 of each weight) and the output twice (before and after the gate): at
most 2^-7 of the largest |v|."""
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
    assert (out.float().cpu() - ref.float()).abs().max().item() <= 2 ** -7 * max(c["v_cache"].float().abs().max(), c["v_new"].float().abs().max()).item()
