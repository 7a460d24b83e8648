"""Rules the kernel sources keep that no run can show to be broken: the loads
and the orderings below go wrong only with a compiler or a schedule that uses
the freedom they would leave."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "fbme-sbl_b200" / "fbme_b200" / "csrc"

# What may be read as constant for a kernel (__ldg): the tables and masks that
# are laid out before a replay, and operands of kernels launched the plain way.
CONSTANT = {
    "cg.cu": [r"fr \+"],  # cg_precond_kernel
    "cg_active.cu": [r"a\.d[12] \+", r"a\.bp \+"],
    "cnn.cu": [r"reinterpret_cast<const (uint4|float4)\*>\((x|gin|mask) \+"],  # wgrad_kernel
    "fft.cu": [r"(p|st\.p)\.tw \+", r"mask \+"],
    "polish.cu": [r"A\.p\.(gram2d|dir1|dir2) \+", r"row \+"],  # row: of gram2d
}


@pytest.mark.parametrize("path", sorted(CSRC.glob("*.cu*")), ids=lambda p: p.name)
def test_constant_loads_read_tables_only(path):
    """A kernel launched as a dependent starts before its predecessor ends, so
    what the chain writes is read by plain loads."""
    allowed = CONSTANT.get(path.name, [])
    code = re.sub(r"//.*", "", path.read_text())
    for m in re.finditer(r"__ldg\(", code):
        operand = code[m.end():m.end() + 80]
        assert any(re.match(a, operand) for a in allowed), operand.splitlines()[0]


def test_dependent_kernels_wait_for_their_predecessor():
    text = {p.name: p.read_text() for p in CSRC.glob("*.cu*")}
    code = "\n".join(text.values())
    names = set(re.findall(r"launch_dep\((\w+)", code)) - {"void", "kern", "scan"} | {"fft_fast_kernel", "cert_scan_kernel"}
    assert len(names) > 15
    for name in names:
        body = re.search(r"\b%s\([^;{]*\) \{(.*?)^\}" % name, code, re.S | re.M)
        assert body and "dep_sync();" in body.group(1), name


@pytest.mark.parametrize("name", ["polish.cu", "dense.cu"])
def test_posted_column_is_ordered_within_its_warp(name):
    """The warp that posts a column of a factorisation only arrives at the
    column's barrier, which orders nothing for its own later reads."""
    body = re.search(r"auto post = \[&\]\(int q, .*?\n  \};", (CSRC / name).read_text(), re.S).group(0)
    stores, arrive = body.rindex("S.rl[q] ="), re.search(r"\w+_arrive\(q\)", body).start()
    assert "__syncwarp();" in body[stores:arrive]
