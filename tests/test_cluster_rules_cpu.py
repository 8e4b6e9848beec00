"""Rules between the CTAs of a cluster that no run can show without a race, read from the sources."""
import re

import pytest

from test_launch_rules_cpu import CSRC, body


def test_rotated_q_is_released_at_cluster_scope():
    """Q rotated in the odd CTA's shared memory is read by a product that the even CTA issues: the arrival that hands it over orders the
    stores for the other CTA.  The plain arrival is left to what tcgen05 fences order: tensor memory, behind a fence of its own."""
    text = body("prefill_umma", "prefill_pair_kernel")
    assert re.search(r"fence_proxy_async\(\);\s*__syncwarp\(\);\s*if \(lane == 0\) mbar_arrive\(rank == 0 \? &lead_q : &bar_rot\);", text)
    assert re.search(r"ready_q = cluster_map\(smem_u32\(&lead_q\), 0\);[^}]*ok = warp_wait_bounded\(&bar_rot, i & 1, ok\);\s*"
                     r"if \(ok && lane == 0\) mbar_arrive_cluster\(ready_q\);", text)
    assert "lead_q, FUSED ? PU_OUT_WARPS + 1 : 1" in text and "bar_rot, PU_OUT_WARPS)" in text      # the even CTA's warps and the odd one's 12
    plain = [m.start() for m in re.finditer(r"mbar_arrive_cluster_plain\(", text)]
    assert len(plain) == 2
    for at in plain:
        assert re.search(r"tc_fence_before_sync\(\);\s*__syncwarp\(\);\s*if \(lane == 0\) $", text[:at])
    helper = (CSRC / "common.cuh").read_text()
    assert "mbarrier.arrive.release.cluster.shared::cluster.b64" in helper[helper.index("void mbar_arrive_cluster("):][:160]


@pytest.mark.parametrize("name,function", [("decode_fused", "fused_decode_kernel"), ("skinny_gemm", "skinny_gemm_pairk_kernel"),
                                           ("prefill_umma", "prefill_pair_kernel")])
def test_no_remote_access_before_the_peer_runs(name, function):
    """A cluster barrier lies between a kernel's start and its first access to a peer's shared memory."""
    text = body(name, function)
    remote = r"st_cluster_f32x4\(|st\.shared::cluster|mbar_arrive_cluster(?:_plain)?\(|(?:umma_\w+|tma_load_\dd)_pair\("
    first = re.search(remote, text).start()
    before = text[:first]
    assert "cluster_sync();" in before or 0 < before.find("cluster_started();") < before.find("cluster_all_started();")


def test_every_cluster_kernel_is_looked_at():
    """Kernels that reach into a peer's shared memory are those of the test above."""
    users = {f.stem for f in CSRC.glob("*.cu") if re.search(r"cluster_map\(|st_cluster", re.sub(r"//[^\n]*", "", f.read_text()))}
    assert users == {"decode_fused", "skinny_gemm", "prefill_umma"}


def test_one_cta_prefill_waits_name_one_phase():
    """A wait by parity tells two phases apart.  Behind its last P a thread cannot say whether one PV product is still to come or two: the last
    one has a barrier of its own, and no other wait in the softmax warps follows an arrival that lets a second phase pass."""
    text = body("prefill_short", "prefill_short_kernel")
    assert "umma_commit_leader(jj + 1 < n_tiles ? &bar_pv : &bar_o, leader)" in text
    epilogue = text[text.rindex("mbar_arrive(&bar_p[s])"):]
    assert "bar_pv" not in epilogue and "warp_wait_bounded(&bar_o, 0, ok)" in epilogue
    rescale = text[text.index("if (__any_sync("): text.index("mbar_arrive(&bar_p[s])")]
    assert "warp_wait_bounded(&bar_pv, (j - 1) & 1)" in rescale      # in front of the own P(j), without which PV(j) cannot pass
