"""A cell without a free vertex, far larger than the cells around it: a long
tetrahedron on a wall or inlet face, its tip outside the pipe.  The FP16 operator scales
the vertices' vectors by the largest one of a free vertex; those of fixed
vertices, which no product needs, may be larger than that leaves room for
(here by factors of 12 and 18; the FP16 range ends at 2 to 4).  The FP16
V-cycle has to precondition as the FP32 one does: every solve meets p_rtol =
1e-6, so the fields agree to that, in as many iterations give or take two.
"""
from __future__ import annotations

import numpy as np
import pytest

from conftest import rel_l2

CFG = dict(re=20.0, alpha_u=0.7, alpha_p=0.3, p_rtol=1e-6, p_max=100, amg_terminal=16, max_outer=10,
           precision="mixed", p_krylov="pcg")


def _spiked(tag, length):
    from nodals_b200 import meshgen
    m = meshgen.pipe_mesh(nr=2, ntheta=8, nz=6, length=3.0, jitter=0.05, seed=7)
    k = int(np.flatnonzero(m.btag == tag)[len(m.btag) // 5 if tag == 0 else 3])
    a, b, c = m.bfaces[k]
    p = m.points[m.bfaces[k]]
    n = np.cross(p[1] - p[0], p[2] - p[0])
    n /= np.linalg.norm(n)
    out = p.mean(axis=0) * (1.0, 1.0, 0.0) if tag == 0 else np.array([0.0, 0.0, -1.0])  # wall, inlet at z = 0
    n *= np.sign(n @ out)
    tip = len(m.points)
    points = np.vstack([m.points, p.mean(axis=0) + length * n])
    t = np.array([a, b, c, tip])
    if np.linalg.det(points[t[1:]] - points[t[0]]) < 0.0:
        t[[0, 1]] = t[[1, 0]]
    faces = np.array([[a, b, tip], [b, c, tip], [c, a, tip]], dtype=np.int32)
    return meshgen.TetMesh(points, np.vstack([m.tets, t]).astype(np.int32),
                           np.vstack([np.delete(m.bfaces, k, axis=0), faces]),
                           np.concatenate([np.delete(m.btag, k), np.full(3, tag)]).astype(np.int32))


@pytest.mark.gpu
@pytest.mark.parametrize("resident", ["5000", "0"])
@pytest.mark.parametrize("tag,length", [(0, 5.0), (1, 20.0)], ids=["wall", "inlet"])
def test_large_fixed_cell(native, monkeypatch, tag, length, resident):
    mesh = native.Mesh.from_tetmesh(_spiked(tag, length))
    P = native.Problem(mesh, **CFG, amg_half=1)
    ref = P.array("cell.ref").reshape(-1, 8)[:, :4]
    B = np.abs(P.array("cell.bcoeff").reshape(-1, 8, 3)[:, :4])
    assert B[ref < 0].max() > 4.0 * B[ref >= 0].max()
    monkeypatch.setenv("NDS_RESIDENT", resident)
    A, F = native.Solver(P), native.Solver(native.Problem(mesh, **CFG))
    for _ in range(4):
        a, f = A.step(), F.step()
        assert a.p_rel <= 1e-6 and abs(a.p_its - f.p_its) <= 2, (a.p_its, f.p_its, a.p_rel)
    for x, y in zip(A.fields(), F.fields()):
        assert rel_l2(x, y) <= 1e-5
