"""Rules that the CUDA sources keep and that no run on a healthy GPU can show."""

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "templar_b200" / "ops" / "csrc"


@pytest.mark.parametrize("src", sorted(p.name for p in CSRC.glob("*.cu")))
def test_drains_do_not_wait_on_the_shared_flag(src):
    """A wait whose result nobody looks at is a drain: it stands in front of a role's return so that no copy lands in shared
    memory that the CTA has given back.  With the CTA's own flag, which is up exactly when a role has given up, ``mbar_wait``
    returns at once, so a drain goes through ``Drain``."""
    text = re.sub(r"//[^\n]*", "", (CSRC / src).read_text())
    # a statement that starts with the call: after a brace, a semicolon or a loop head
    ignored = re.findall(r"(?:[;{}]|\bfor \([^{}]*\))\s*(mbar_wait\([^;]*);", text)
    assert not ignored, ignored


@pytest.mark.parametrize("src", sorted(p.name for p in CSRC.glob("*.cu") if "mbar_expect_tx(" in p.read_text()))
def test_every_kernel_that_asks_for_copies_drains_them(src):
    """Each kernel that arms a barrier for bulk copies waits for them before its CTA retires."""
    text = re.sub(r"//[^\n]*", "", (CSRC / src).read_text())
    kernels = re.split(r"__global__", text)[1:]
    arming = [k for k in kernels if "mbar_expect_tx(" in k.split("<<<")[0]]
    assert arming
    for k in arming:
        assert "Drain drain" in k, k[:200]
