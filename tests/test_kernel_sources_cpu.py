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


def _kernels(src):
    """(name, parameter list, body) of every kernel of a source file."""
    text = re.sub(r"//[^\n]*", "", (CSRC / src).read_text())
    for m in re.finditer(r"__global__[^;{]*?(\w+)\s*\(([^(){}]*)\)\s*\{", text):
        depth, i = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(text[i], 0)
            i += 1
        yield m.group(1), m.group(2), text[m.end():i]


@pytest.mark.parametrize("src", sorted(p.name for p in CSRC.glob("*.cu") if "grid_wait();" in p.read_text()))
def test_restrict_pointers_are_taken_anew_behind_the_grid_wait(src):
    """A kernel that may start while the one before it runs touches no memory before ``grid_wait``.  The compiler may move an
    access through a ``__restrict__`` pointer across the wait unless the pointer goes through ``behind_grid_wait`` there, those
    that are written and read as well as the constant ones."""
    waiting = [k for k in _kernels(src) if "grid_wait();" in k[2]]
    assert waiting
    for name, params, body in waiting:
        pointers = re.findall(r"__restrict__\s+(\w+)", params)
        before, behind = body.split("grid_wait();", 1)
        taken = set(re.findall(r"behind_grid_wait\((\w+)\)", behind))
        assert set(pointers) <= taken, (name, set(pointers) - taken)
        assert not any(re.search(rf"\b{p}\b", before) for p in pointers), name


def test_every_exit_of_a_loss_kernel_has_written_its_row():
    """The mean is taken over the rows' array whatever it holds, and the entry that must not allocate has no status word, so a
    kernel that writes rows of losses has neither a wait that can run out nor a ``return`` in front of the row's loss."""
    kernels = [k for k in _kernels("elementwise.cu") if re.search(r"\blosses\[\w+\] = ", k[2])]
    assert len(kernels) == 2
    for name, _, body in kernels:
        assert "mbar_wait" not in body, name
        for exit_at in re.finditer(r"\breturn;", body):
            assert re.search(r"\blosses\[row\] = ", body[:exit_at.start()]), name
