"""The convection table of the device assembly (exported as convTable) against
the exact integrals of barycentric monomials, as the device holds it: in FP64
within the rounding of the 125-point sums it comes from, in FP32 rounded once
(half a unit in the last place).  Formed in FP32 from the tensor rounded to
FP32 its differences would miss that.
"""
from __future__ import annotations

import math
from fractions import Fraction

import numpy as np

PAIRS = [(a, m) for a in range(8) for m in range(a, 8)]


def _unit(*idx):
    e = [0] * 4
    for i in idx:
        e[i] += 1
    return tuple(e)


PHI = [{_unit(i): Fraction(1)} for i in range(4)]
PHI += [{_unit(*[k for k in range(4) if k != i]): Fraction(27)} for i in range(4)]


def _mul(p, q):
    o = {}
    for a, x in p.items():
        for b, y in q.items():
            e = tuple(i + j for i, j in zip(a, b))
            o[e] = o.get(e, 0) + x * y
    return o


def _dlam(p, k):
    return {tuple(v - (q == k) for q, v in enumerate(e)): x * e[k] for e, x in p.items() if e[k]}


def _integral(p):
    return sum((x * Fraction(math.prod(math.factorial(i) for i in e), math.factorial(sum(e) + 3)) for e, x in p.items()),
               Fraction(0))


def _exact():
    out = []
    for a, m in PAIRS:
        am = _mul(PHI[a], PHI[m])
        for i in range(4):
            out += [_integral(_mul(am, _dlam(PHI[4 + i], k))) for k in range(4) if k != i]
            out.append(_integral(am))
    return out


def _errors(table, exact):
    return np.array([abs(float(Fraction(float(t)) - e)) for t, e in zip(table, exact)])


def test_conv_table(native, meshes):
    P = native.Problem(native.Mesh.from_tetmesh(meshes("pipe_tiny")), max_outer=10, amg_terminal=60)
    table, exact = P.array("convTable"), _exact()
    assert len(table) == len(exact) == 576
    scale = np.array([float(e) for e in exact])
    # 125 terms a sum, two sums a difference: 250 roundings of at most the record's scale
    assert np.all(_errors(table, exact) <= 250 * 2.0 ** -53 * np.abs(scale))
    half_ulp = 0.5 * np.spacing(np.abs(scale).astype(np.float32)).astype(np.float64)
    assert np.all(_errors(table.astype(np.float32), exact) <= half_ulp * (1 + 1e-6))
    # the same differences of the tensor rounded to FP32
    T = P.array("centT").reshape(8, 8, 8, 3).astype(np.float32)
    twice = []
    for a, m in PAIRS:
        for i in range(4):
            t = T[a, m, 4 + i]
            n0 = np.float32(0) if i == 0 else -t[i - 1]
            twice += [n0 if k == 0 else np.float32(t[k - 1] + n0) for k in range(4) if k != i] + [T[a, m, 1, 0]]
    assert np.any(_errors(twice, exact) > half_ulp * (1 + 1e-6))
