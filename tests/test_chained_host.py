"""Kernels launched while their predecessor still runs (chain_begin): what an
earlier kernel of the stream wrote may not be read through the read-only data
path, neither by __ldg nor through a const __restrict__ argument.  Checked in
the sources: a wrong value would show on a GPU only by chance."""

import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "vlasolve_b200", "csrc")
FILES = ["vls_kernels.cu", "vls_rc.cu", "vls_adjoint.cu"]

# arguments that no kernel of a step or of a backward pass writes: the
# footpoint and chain tables, the inverse map, the grid's own tables
CONSTANT = {"idx", "fx", "fy", "fp2", "win_rows", "trip_kinds", "ch_start", "ch_len", "ch_at",
            "ch_cell", "t_idx", "t_x", "t_y", "chain_lo", "far_base", "far", "ent", "ebase",
            "ends", "geo", "R", "U", "J", "dR", "dU", "Ct1"}
# what a __ldg may name in a chained kernel: those, their fields and the local
# pointers into them
LDG = CONSTANT | {"mt", "g", "src", "ws", "p", "pn", "pp"}


def _functions(text):
    """(name, head, body) of every function definition of a source file."""
    text = re.sub(r"//[^\n]*", "", text)
    for m in re.finditer(r"\b(\w+)\s*\(", text):
        i, depth = m.end(), 1
        while i < len(text) and depth:
            depth += {"(": 1, ")": -1}.get(text[i], 0)
            i += 1
        k = re.match(r"\s*(const\s*)?\{", text[i:])
        if not k or m.group(1) in ("if", "for", "while", "switch", "__launch_bounds__"):
            continue
        b = i + k.end()
        e, depth = b, 1
        while e < len(text) and depth:
            depth += {"{": 1, "}": -1}.get(text[e], 0)
            e += 1
        head = text[max(0, text.rfind(";", 0, m.start()), text.rfind("}", 0, m.start())):m.start()]
        yield m.group(1), head, text[m.end():i], text[b:e]


@pytest.mark.parametrize("name", FILES)
def test_chained_kernels_read_written_data_by_plain_loads(name):
    with open(os.path.join(CSRC, name)) as fh:
        fns = list(_functions(fh.read()))
    chained = [f for f in fns if "__global__" in f[1] and "chain_begin();" in f[3]]
    assert chained
    for fn, _, args, body in chained:
        ro = re.findall(r"const\s+\w+\s*\*\s*__restrict__\s+(\w+)", args)
        assert set(ro) <= CONSTANT, (fn, sorted(set(ro) - CONSTANT))
        ldg = re.findall(r"__ldg\(\s*(?:reinterpret_cast<[^>]*>\()?(\w+)", body)
        assert set(ldg) <= LDG, (fn, sorted(set(ldg) - LDG))


def test_global_gather_uses_plain_loads():
    """eval2d reads C, which the r-solve before the drift wrote."""
    with open(os.path.join(CSRC, "vls_kernels.cu")) as fh:
        fns = [f for f in _functions(fh.read()) if f[0] in ("eval2d", "eval2d_f32x2")]
    assert len(fns) >= 2
    for _, _, args, body in fns:
        assert "__restrict__" not in args and "__ldg" not in body
