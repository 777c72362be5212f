"""Kernels that may start before the kernel ahead of them has ended read nothing through the read-only path.

A chained kernel (launch_chained) is resident while its predecessor still writes the populations, the adjoint
field or the window table.  Read-only loads (__ldg, ld.global.nc, const __restrict__ parameters) are
defined only for memory that nobody writes while the kernel lives, so none may reach such data.  Whether a
stale line is met depends on the hardware; the sources are what can be checked."""

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "particuology_hydraulic_penalty_b200" / "csrc"


def _source(path):
    text = path.read_text()
    return re.sub(r"//[^\n]*", "", re.sub(r"/\*.*?\*/", "", text, flags=re.S))


def _launches(text):
    """(kernel, whether it is always chained) of every launch_chained call."""
    found = []
    for m in re.finditer(r"launch_chained\(", text):
        depth, k = 1, m.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(text[k], 0)
            k += 1
        args = re.sub(r"<[^<>()]*>", "", re.sub(r"static_cast<[^<>]*>", "", text[m.end():k - 1]))
        parts, depth, cur = [], 0, ""
        for ch in args:
            depth += {"(": 1, ")": -1}.get(ch, 0)
            if ch == "," and depth == 0:
                parts.append(cur.strip())
                cur = ""
            else:
                cur += ch
        found.append((parts[0], parts[5] == "true"))
    return found


CHAINED = sorted((p.name, *x) for p in CSRC.glob("*.cu") for x in set(_launches(_source(p))))


def test_the_chained_kernels_are_found():
    names = {k for _, k, _ in CHAINED}
    assert {"k_step_exact", "k_step_fast", "k_step_pair", "k_bb_step", "k_reduce_windows", "k_adjoint_step",
            "k_adjoint_pair", "k_loads_final", "k_loads_final_multi"} <= names


@pytest.mark.parametrize("name", sorted({f for f, _, _ in CHAINED}) + sorted(p.name for p in CSRC.glob("*.cuh")))
def test_no_read_only_loads(name):
    text = _source(CSRC / name)
    assert not re.search(r"__ldg|\.nc\b", text)


@pytest.mark.parametrize("name,kernel,always", CHAINED)
def test_parameters_of_chained_kernels_are_not_restrict(name, kernel, always):
    """The window table of a step that is chained by PSC_STEP_CHAINED alone is not written by the kernel ahead."""
    text = _source(CSRC / name)
    m = re.search(r"\b" + kernel + r"\(([^)]*)\)\s*\{", text)
    params = m.group(1)
    if not always:
        params = params.replace("const psc_window* __restrict__ wins", "")
    assert "__restrict__" not in params
