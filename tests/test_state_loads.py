"""How the solver's kernels read what other launches write.

The read-only load (__ldg, the compiler's __restrict__ on const pointers) is
for data that no launch writes while the kernel lives.  Sweeps and steps are
launched as programmatic dependents, so a block may be on the chip while an
earlier step still writes the state and the max-wave fields: kernels read
those with plain or L2 loads.  Read from the sources, comments left out."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cliffs-src_gb300", "csrc")
WRITTEN = re.compile(r"(srf|xu|yv|hmax|velmax)\w*\b")


def _code(name):
    with open(os.path.join(CSRC, name)) as f:
        return re.sub(r"//[^\n]*", "", f.read())


def _arguments(code, call):
    """The argument text of every call, brackets matched."""
    for m in re.finditer(re.escape(call) + r"\(", code):
        depth, at = 1, m.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(code[at], 0)
            at += 1
        yield code[m.end():at - 1]


@pytest.mark.parametrize("name", ["sweep.cuh", "step.cuh", "line.cuh", "ytile.cuh", "staged.cuh", "batch.cuh"])
def test_fields_that_launches_write_are_not_read_only(name):
    code = _code(name)
    bad = [a for a in _arguments(code, "__ldg") if WRITTEN.search(a)]
    assert not bad, bad
    assert not re.search(r"const float\s*\*\s*__restrict__\s+(srf|xu|yv|hmax|velmax)\b", code)


def test_state_loads_are_plain_or_from_l2():
    code = _code("sweep.cuh")
    for fn in ("ld_state", "ld_state4"):
        body = re.search(r"\b%s\(const float\* p\) \{(.*?)\}" % fn, code, re.S).group(1)
        assert "__ldg" not in body and "__ldcg" in body
