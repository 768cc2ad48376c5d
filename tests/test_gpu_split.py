"""The pressure operator in split form (face couplings + vertex sums) against
B diag(rAU) B^T taken from the host setup's coefficients in FP64, at sizes
with every remainder of the launch shapes, straight and bent, and with the
wide index forms forced.

Tolerances, u = eps32 / 2.  Vertex step: coefficient, product, up to seven
additions in a row (four in a lane, three between lanes), rAU and the scaling
round once each, 11 u relative to |B|^T |x| per vertex.  Cell step: the
vertices enter as S_j (w_j - w_0) with the gradients S_1..S_3 of vertices 1
to 3, so vertex 0 weighs |S_1| + |S_2| + |S_3|; coefficient, difference and
nine additions round, 11 u; the faces' differences and sums fewer.  Together
|y - y64| <= 12 eps32 C diag(rAU) |B|^T |x| with C = |B| except for the row of
vertex 0.  The edge weights are formed in FP64 and rounded to FP32 after two
FP32 factors: 4 eps32 relative.
"""
from __future__ import annotations

import numpy as np
import pytest

EPS32 = 2.0 ** -23
MESHES = [(2, 8, 6, 0.0), (2, 8, 7, 0.0), (3, 16, 12, 0.0), (4, 24, 11, 35.0)]


def _problem(native, nr, ntheta, nz, bend):
    from nodals_b200 import meshgen
    m = meshgen.pipe_mesh(nr=nr, ntheta=ntheta, nz=nz, length=0.5 * nz, jitter=0.05, seed=nz, bend_deg=bend)
    return native.Problem(native.Mesh.from_tetmesh(m), max_outer=10, re=20.0, alpha_u=0.7, alpha_p=0.3, p_rtol=1e-6,
                          p_max=400, amg_terminal=60, precision="mixed", geom_from_inlet=int(bend > 0))


@pytest.mark.gpu
@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("nr,ntheta,nz,bend", MESHES)
def test_split_product_and_edges(native, monkeypatch, nr, ntheta, nz, bend, wide):
    import torch
    if wide:
        monkeypatch.setenv("NDS_SELL_COL32", "1")
    P = _problem(native, nr, ntheta, nz, bend)
    S = native.Solver(P)  # its operator is that of the setup's rAU
    nc, nv = S.nc, S.nv
    ref = P.array("cell.ref").reshape(nc, 8)
    B = P.array("cell.bcoeff").reshape(nc, 8, 3) * (ref >= 0)[:, :, None]
    g = np.maximum(ref, 0).reshape(-1)
    rau = P.array("initRau")

    def apply(coef, x):
        v = np.zeros((nv, 3))
        np.add.at(v, g, (coef * x[:, None, None]).reshape(-1, 3))
        return (coef.reshape(-1, 3) * (rau[:, None] * v)[g]).reshape(nc, -1).sum(axis=1)

    def bound(x):
        raw = np.abs(P.array("cell.bcoeff").reshape(nc, 8, 3))
        cell = np.abs(B)
        cell[:, 0] = raw[:, 1:4].sum(axis=1) * (ref[:, :1] >= 0)
        v = np.zeros((nv, 3))
        np.add.at(v, g, (np.abs(B) * np.abs(x)[:, None, None]).reshape(-1, 3))
        return 12 * EPS32 * (cell.reshape(-1, 3) * (rau[:, None] * v)[g]).reshape(nc, -1).sum(axis=1)

    rng = np.random.default_rng(nc)
    for x in (rng.standard_normal(nc), np.ones(nc), np.eye(1, nc, nc // 2)[0]):
        x = x.astype(np.float32).astype(np.float64)
        xd = torch.from_numpy(x.astype(np.float32)).cuda()
        y = torch.full_like(xd, float("nan"))
        torch.cuda.synchronize()
        native.solver_apply_operator(S, xd, y)
        err = np.abs(y.cpu().numpy().astype(np.float64) - apply(B, x))
        assert np.all(err <= bound(x)), float((err - bound(x)).max())
    # edge weights and scaling of the face graph
    nbr = torch.zeros(4 * nc, dtype=torch.int32, device="cuda")
    ew = torch.zeros(4 * nc, dtype=torch.float32, device="cuda")
    ds = torch.zeros(nc, dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    native.solver_stage_graph(S, nbr, ew, ds)
    nbr, ew, ds = nbr.cpu().numpy().reshape(nc, 4), ew.cpu().numpy().reshape(nc, 4), ds.cpu().numpy().astype(np.float64)
    diag = (B ** 2 * np.where(ref >= 0, rau[np.maximum(ref, 0)], 0.0)[:, :, None]).sum(axis=(1, 2))
    assert np.all(np.abs(ds - diag ** -0.5) <= 4 * EPS32 * diag ** -0.5)
    rows = {}
    for c in range(nc):
        for a in range(8):
            if ref[c, a] >= 0:
                rows.setdefault(ref[c, a], []).append((c, a))
    a_ij = {}
    for dof, inc in rows.items():
        for c, a in inc:
            for c2, b in inc:
                a_ij[c, c2] = a_ij.get((c, c2), 0.0) + rau[dof] * float(B[c, a] @ B[c2, b])
    for c in range(nc):
        for k in range(4):
            j = nbr[c, k]
            want = a_ij[c, j] * ds[c] * ds[j] if j >= 0 else 0.0
            # a_ij itself may cancel: the error scales with its largest terms, at most the geometric mean diagonal
            assert abs(ew[c, k] - want) <= 4 * EPS32 * max(abs(want), 1e-6)
