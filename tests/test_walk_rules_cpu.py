"""Rules of the chunk walks that no run can show without a race or a lost copy, read from their sources."""
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
