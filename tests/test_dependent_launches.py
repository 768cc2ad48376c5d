"""Kernels launched while their predecessor still runs (pdl_launch): each
waits for it, and reads what a kernel of the chain writes through pointers that
let the compiler assume nothing about the time before that wait.  A `const
__restrict__` parameter of such a kernel may be read with invariant loads,
which can be moved above the wait; so it may only be data that stays as it is
during a solve, and any other `__restrict__` parameter may only be stored to.
"""
from __future__ import annotations

import re
from pathlib import Path

import pytest

CUDA = Path(__file__).resolve().parent.parent / "nodals_b200" / "csrc" / "cuda"
HEADERS = "".join((CUDA / f).read_text() for f in ("kernels.cuh", "krylov.cuh", "split.cuh", "resident.cuh"))
SOLVER = (CUDA / "solver.cu").read_text()
# matrices, transfers, index arrays, geometry, smoother denominators (rewritten only behind an event wait, before a
# solve); setup data
CONSTANT = {
    "mom_gs_color": {"rows", "span", "ci"},
    "continuity": {"ref", "bco", "fixed_div"},
    "spmv": {"rp", "ci", "v"},
    "spmv_resid": {"rp", "ci", "v", "den"},
    "spmv_smooth": {"rp", "ci", "v", "den"},
    "level_window": {"win", "rp", "ci", "v", "den"},
    "jacobi_zero": {"d"},
    "loop_start": {"den0"},
    "xr_update": {"den0"},
    "prolong_add": {"pc", "pv"},
    "dense_rows": {"A"},
    "sell_spmv": {"v", "den"},
    "cast_jacobi": {"den0"},
    "restrict_stream": {"rr", "rc", "rv", "den0"},
    "restrict_rows": {"rr", "rc", "rv", "den0"},
    "fg_normalize": {"den0"},
    "split_vertex": {"rau"},
    "split_cell": {"den"},
}
# of the struct parameters: written by the kernel before this one
WRITTEN_MEMBERS = {"MomArgs": {"C", "pz"}, "PlainVector": {"x"}, "PlainVertices": {"w"}}


def _braces(text, start):
    depth = 0
    for k in range(start, len(text)):
        depth += {"{": 1, "}": -1}.get(text[k], 0)
        if depth == 0:
            return text[start:k + 1]
    raise AssertionError("unbalanced")


def _function(name):
    """Parameters and body of a function template of the headers."""
    m = [q for q in re.finditer(r"\b%s\(((?:[^(){};]|\([^()]*\))*)\)\s*\{" % name, HEADERS)]
    assert len(m) == 1, (name, len(m))
    body = _braces(HEADERS, m[0].end() - 1)
    params = [re.sub(r"\s+", " ", p).split("=")[0].strip() for p in m[0].group(1).split(",")]
    return params, re.sub(r"//[^\n]*", "", body)


def _launched():
    names = set(re.findall(r"pdl_launch\(k::(\w+)", SOLVER))
    names |= set(re.findall(r"auto\* kernel = k::(\w+)<[^;]*;(?:(?!\n  }).)*?pdl_launch\(kernel", SOLVER, flags=re.S))
    return sorted(names)


def test_launches_are_found():
    names = _launched()
    assert {"level_window", "split_cell", "spmv_smooth", "xr_update", "fg_dots"} <= set(names)
    assert len(re.findall(r"pdl_launch\((?!k::|kernel\b)", SOLVER)) == 0


@pytest.mark.parametrize("name", _launched())
def test_dependent_kernel(name):
    params, body = _function(name)
    assert "pdl_begin()" in body or ("pdl_trigger()" in body and ("pdl_wait()" in body or "group_row_dot" in body))
    for p in params:
        if "__restrict__" not in p:
            continue
        arg = p.split()[-1]
        if p.startswith("const "):
            assert arg in CONSTANT.get(name, set()), f"{name}: {p}"
            continue
        # only stored to: arg[...] = (or through a cast), tested against null, given to write_partials
        uses = re.sub(r"reinterpret_cast<\w+\*>\(%s\)\[[^;=]*\] = " % arg, "", body)
        uses = re.sub(r"(?<!\.)\b%s\[(?:[^][]|\[[^]]*\])*\] = " % arg, "", uses)
        uses = re.sub(r"if \(%s\)|if \(%s &&|= %s \?|write_partials<\w+>\(acc, %s\)" % ((arg,) * 4), "", uses)
        assert not re.search(r"(?<!\.)\b%s\b" % arg, uses), f"{name}: {p} is read"


def test_shared_helpers():
    for helper, arg in (("lane_batched_dot", "x"), ("group_row_dot", "x"), ("sell_row", "x"), ("stage_window", "x")):
        params, _ = _function(helper)
        p = [q for q in params if q.split()[-1] == arg]
        assert len(p) == 1 and "__restrict__" not in p[0], (helper, p)
    for struct, members in WRITTEN_MEMBERS.items():
        m = re.search(r"struct %s \{" % struct, HEADERS)
        body = _braces(HEADERS, m.end() - 1)
        for q in members:
            decl = re.findall(r"[^;{}]*\b%s;" % q, body)
            assert decl and all("__restrict__" not in d for d in decl), (struct, q)
