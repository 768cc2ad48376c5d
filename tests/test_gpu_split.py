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
vertex 0.  The state's FP64 and FP32 forms have the same steps in their own eps
(FP32: couplings from rounded factors, three roundings more on a part that
takes seven fewer).  The FP16 form is compared with the 64-bit product of the
same halves: vectors scaled and rounded in the records and the cells alike,
couplings scaled, saturated and rounded from the FP64 ones; what is left are the
FP32 sums of 12 products and 4 differences a cell, within the same bound with
C = |B|.  The edge weights are formed in FP64 and rounded to FP32 after two
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


LARGE = (12, 40, 59, 20.0)  # 34,000 free vertices: more than one pass of every persistent grid
KIND = {"fp64": dict(precision="fp64"), "fp32": dict(precision="fp32"), "mixed": dict(precision="mixed"),
        "half": dict(precision="mixed", amg_half=1)}


@pytest.mark.gpu
@pytest.mark.parametrize("kind,form", [("fp64", "state"), ("fp32", "state"), ("mixed", "state"), ("mixed", "vcycle"),
                                       ("half", "vcycle")])
@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("nr,ntheta,nz,bend", MESHES + [LARGE])
def test_split_forms(native, monkeypatch, nr, ntheta, nz, bend, wide, kind, form):
    import torch
    if wide:
        monkeypatch.setenv("NDS_SELL_COL32", "1")
    from nodals_b200 import meshgen
    m = meshgen.pipe_mesh(nr=nr, ntheta=ntheta, nz=nz, length=0.5 * nz, jitter=0.05, seed=nz, bend_deg=bend)
    P = native.Problem(native.Mesh.from_tetmesh(m), max_outer=10, re=20.0, alpha_u=0.7, alpha_p=0.3, p_rtol=1e-6,
                       p_max=400, amg_terminal=60, geom_from_inlet=int(bend > 0), **KIND[kind])
    S = native.Solver(P)
    nc, nv = S.nc, S.nv
    ref = P.array("cell.ref").reshape(nc, 8)
    free = ref >= 0
    raw = P.array("cell.bcoeff").reshape(nc, 8, 3)
    rau, g = P.array("initRau"), np.maximum(ref, 0)
    if (nr, ntheta, nz, bend) == LARGE:
        assert ref[:, :4].max() + 1 > 148 * 5 * 32
    rv = np.where(free, rau[g], 0.0)
    b2 = raw[:, :4, 0] ** 2 + raw[:, :4, 1] ** 2 + raw[:, :4, 2] ** 2  # of vertex i; its face's is kB2 of that
    kB2 = (27.0 / 20.0) * (27.0 / 20.0)
    tau = kB2 * b2 * rv[:, 4:]
    V = raw[:, :4] * free[:, :4, None]
    if kind == "half":
        scale = 2.0 ** (14 - np.floor(np.log2(np.abs(V).max())))
        V = (V * scale).astype(np.float32).astype(np.float16).astype(np.float64) / scale
        hs = 2.0 ** np.floor(np.log2(2048.0 / (b2 * rv[:, :4] + tau).sum(axis=1).astype(np.float32).max()))
        half = np.minimum(tau.astype(np.float32) * np.float32(hs), np.float32(65504.0)).astype(np.float16)
        tau = half.astype(np.float64) / hs
    # face neighbours: the other cell of each free face (itself on an outlet)
    order = np.argsort(ref[:, 4:].reshape(-1), kind="stable")
    f = ref[:, 4:].reshape(-1)[order]
    nbr = np.full(4 * nc, -1)
    same = np.flatnonzero((f[1:] == f[:-1]) & (f[1:] >= 0))
    nbr[order[same]], nbr[order[same + 1]] = order[same + 1] // 4, order[same] // 4
    nbr = nbr.reshape(nc, 4)
    real = np.longdouble

    def vertex_sums(coef, x):
        w = np.zeros((nv, 3), dtype=real)
        np.add.at(w, g[:, :4].reshape(-1), (coef.astype(real) * x[:, None, None]).reshape(-1, 3))
        return (rau[:, None] * w)[g[:, :4]]

    def exact(x):
        d = x[:, None] - np.where(nbr >= 0, x[nbr], 0.0)
        return (V.astype(real) * vertex_sums(V, x)).sum(axis=(1, 2)) + (tau.astype(real) * d).sum(axis=1)

    def bound(x, eps):
        C = np.abs(V)
        if kind != "half":
            C[:, 0] = np.abs(raw[:, 1:4]).sum(axis=1) * free[:, :1]  # a fixed vertex has w = 0
        d = np.abs(x)[:, None] + np.where(nbr >= 0, np.abs(x[nbr]), 0.0)
        return 12 * eps * ((C * vertex_sums(np.abs(V), np.abs(x))).sum(axis=(1, 2)) + (tau * d).sum(axis=1))

    double = kind == "fp64" or (kind, form) == ("mixed", "state")
    dt = np.float64 if double else np.float32
    rng = np.random.default_rng(nc)
    for x in (rng.standard_normal(nc), np.ones(nc), np.eye(1, nc, nc // 2)[0]):
        x = x.astype(dt)
        xd = torch.from_numpy(x).cuda()
        y = torch.full_like(xd, float("nan"))
        torch.cuda.synchronize()
        native.solver_apply_operator_form(S, form, xd, y)
        xr = x.astype(real)
        err, lim = np.abs(y.cpu().numpy().astype(real) - exact(xr)), bound(xr, np.finfo(dt).eps)
        assert np.all(err <= lim), float((err - lim).max())
