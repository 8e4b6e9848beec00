"""Rules of early launches and bounded waits that no run can show without a race or a lost copy, read from the sources."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "qwen3_5-triton-inference-engine_b200" / "csrc"
EARLY = {"linear_rnn_walk": "outer_walk_kernel", "ssd_walk": "ssd_walk_kernel"}     # file -> what is launched early


def body(name: str, function: str) -> str:
    """Text of a function (its own braces matched), without comments."""
    text = re.sub(r"//[^\n]*", "", (CSRC / f"{name}.cu").read_text())
    at = text.index("{", re.search(rf"(?<!launch_pdl\()\b{function}\([^;{{]*\{{", text).end() - 1)
    depth = 0
    for i in range(at, len(text)):
        depth += (text[i] == "{") - (text[i] == "}")
        if depth == 0:
            return text[at: i + 1]
    raise AssertionError(function)


@pytest.mark.parametrize("name", EARLY)
def test_every_cta_orders_the_grid(name):
    """A kernel that starts while its predecessor runs orders what follows only if no CTA leaves before it has waited."""
    text = body(name, EARLY[name])
    assert "pdl_wait()" in text
    assert "return" not in text[: text.index("pdl_wait()")]


def test_early_mixer_reads_plain_pointers():
    """Loads through `const __restrict__` may be moved above the wait for the kernel in front; its calls without flags are launched
    early too, so that anything it reads may be that kernel's output."""
    text = re.sub(r"//[^\n]*", "", (CSRC / "gdn_recurrent.cu").read_text())
    at = text.index("gdn_decode_fused_kernel(const")
    assert "__restrict__" not in text[at: text.index("{", at)]


@pytest.mark.parametrize("name", ["gdn_chunk_walk", "linear_rnn_walk", "ssd_walk"])
def test_warps_give_up_whole(name):
    """A wait that runs out must not leave some lanes of a warp to matrix instructions, or some threads to a barrier, that the others
    have left: what a wait says decides nothing before the warp has voted.  Single threads wait for copies that nobody waits for any
    more, and go nowhere afterwards."""
    text = re.sub(r"//[^\n]*", "", (CSRC / f"{name}.cu").read_text())
    if name == "gdn_chunk_walk":
        text = text.replace(body(name, "copy_chunks"), "")       # below
    assert not re.findall(r"if \([^\n]*(?:mbar_wait_bounded|team_wait)\(", text)
    assert "warp_wait_bounded(" in text


def test_copy_warps_give_up_together():
    """The copy threads of a Gated-DeltaNet walk, which do nothing as warps while they copy, meet between items: none leaves before it
    has said so there."""
    text = body("gdn_chunk_walk", "copy_chunks")
    assert "return" not in text
    assert text.index("__syncwarp()") < text.index("named_barrier_all(") < text.index("item = *handover")
    assert "if (ok) asm volatile(\"cp.async.mbarrier.arrive" in text       # ... and a stage it did not fill stays incomplete


def test_team_lanes_stay():
    """Lanes whose wait among the warps of a team ran out stay until the vote that opens a chunk, and store nothing."""
    text = body("gdn_chunk_walk", "gdn_walk_team_kernel")
    assert text.index("warp_wait_bounded(&full[stage], full_parity, ok)") < text.index("team_wait(")
    assert len(re.findall(r"ok = ok && team_wait\(", text)) == text.count("team_wait(")
    assert text.count("return;") == 2                   # the copy warps, and the end of the items


def test_idle_decode_ctas_leave_no_copy_behind():
    """A CTA without work has asked for the tables of norm weights and frequencies: it waits for these copies into its shared memory
    before it leaves."""
    text = body("decode_fused", "fused_decode_kernel")
    asked = text.index("cp_async16(")
    text = text[asked: text.index("auto issue_next")]
    assert text.count("return;") == len(re.findall(r"cp_async_wait_all\(\);\s*pdl_wait\(\);\s*return;", text)) == 3
