"""Warps that issue tensor-core products walk their loops as a whole (uniform_warp_id).  Lanes that poll a
barrier for themselves can get different answers once another warp has raised the abort flag, and a lane that
left its loop alone would be waited for at a warp barrier for good.  So these warps vote on every poll.  That
cannot be provoked without hanging a GPU, so the source is read."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "scpaper-2021_b200", "csrc")
HEAD = "// ---------------- "


def _issuing_sections():
    out = []
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu")) + glob.glob(os.path.join(CSRC, "*.cuh"))):
        with open(path) as f:
            text = f.read()
        if "= uniform_warp_id()" in text:
            start = text.index(HEAD + "MMA issuer")
            section = text[start:text.index(HEAD, start + len(HEAD))]
            out.append(pytest.param(re.sub(r"//[^\n]*", "", section), id=os.path.basename(path)))
    return out


@pytest.mark.parametrize("code", _issuing_sections())
def test_issuing_warps_take_every_answer_together(code):
    waits = re.findall(r"\bmbar_\w*wait\w*\(", code)
    assert waits and set(waits) == {"mbar_wait_bounded_warp("}


def test_the_warp_wait_votes_on_every_poll():
    with open(os.path.join(CSRC, "common.cuh")) as f:
        text = f.read()
    body = text[text.index("bool mbar_wait_bounded_warp("):]
    body = body[:body.index("\n}\n")]
    assert body.count("mbar_try_wait(") == 1 and "return false" in body
    assert "__all_sync(0xffffffffu, mbar_try_wait(" in body and "__any_sync(0xffffffffu, *abort_flag)" in body
