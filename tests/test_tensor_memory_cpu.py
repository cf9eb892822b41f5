"""Rules by which launches share tensor memory, checked where a GPU run could only hang: in the sources and in the launch plans."""
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "turbopi_b200" / "csrc"


def _functions(text):
    """Bodies of the device functions, comments removed (a body starts at a line that ends in `{` in the first column's scope)."""
    text = re.sub(r"//[^\n]*", "", text)
    return re.findall(r"^[^\s#}][^\n;]*\([^;{}]*\)\s*\{\n(.*?)^\}", text, re.S | re.M)


@pytest.mark.parametrize("source", sorted(p.name for p in CSRC.glob("*.cu") if "tmem_alloc(" in p.read_text()))
def test_dependents_are_let_in_behind_the_allocation(source):
    """A kernel that lets the next launch in before its own allocation is complete can lose the columns to a CTA that keeps
    them until this kernel ends."""
    checked = 0
    for body in _functions((CSRC / source).read_text()):
        if "tmem_alloc(" not in body or "pdl_launch_dependents()" not in body:
            continue
        allocated = body.index("tmem_alloc(")
        barrier = body.index("__syncthreads()", allocated)
        assert body.index("pdl_launch_dependents()") > barrier, source
        checked += 1
    assert checked >= {"attention.cu": 2}.get(source, 1), source
