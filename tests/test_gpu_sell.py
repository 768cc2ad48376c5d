"""The pressure operator as assembled rows (SELL), which the L1-Jacobi and
Gauss-Seidel smoothers read, against B diag(rAU) B^T from the host setup's
coefficients in 64 bits: products in every precision, and the face graph's edge
weights.

Tolerances.  An entry is a sum in the state's precision of at most 12 products
of three factors each (vertices shared by two cells, times three components;
diagonal 24): 8 roundings after each other and their three factors, 12 eps of
the sum of its terms' sizes.  A row adds up to 100 entries in two or four
chains: 50 eps.  FP32 data: one rounding of the entry more.  FP16 data: 2^-11 of the entry, or 2^-25
in scaled units below the normal range; scale: the power of two that puts the
largest diagonal at 2^11.  Edge weights: as in the split form's test.
"""
from __future__ import annotations

import numpy as np
import pytest
import scipy.sparse as sp

KIND = {"fp64": (dict(precision="fp64"), "state", np.float64), "fp32": (dict(precision="fp32"), "state", np.float32),
        "amg_fp32": (dict(precision="amg_fp32"), "vcycle", np.float32),
        "mixed": (dict(precision="mixed"), "vcycle", np.float32), "mixed_state": (dict(precision="mixed"), "state", np.float64),
        "half": (dict(precision="mixed", amg_half=1), "vcycle", np.float32)}
MESHES = [(2, 8, 7), (3, 16, 12)]


def _solver(native, mesh, **kw):
    from nodals_b200 import meshgen
    nr, nt, nz = mesh
    m = meshgen.pipe_mesh(nr=nr, ntheta=nt, nz=nz, length=0.5 * nz, jitter=0.05, seed=nz)
    P = native.Problem(native.Mesh.from_tetmesh(m), max_outer=10, re=20.0, alpha_u=0.7, alpha_p=0.3, p_rtol=1e-6,
                       p_max=400, amg_terminal=60, amg_hierarchy="sa", amg_smoother="l1jacobi", **kw)
    S = native.Solver(P)
    nc, nv = S.nc, S.nv
    ref = P.array("cell.ref").reshape(nc, 8)
    B = P.array("cell.bcoeff").reshape(nc, 8, 3) * (ref >= 0)[:, :, None]
    rau = P.array("initRau")
    cells = np.repeat(np.arange(nc), 8)
    A = Aabs = 0.0
    for d in range(3):
        Bd = sp.csr_matrix((B[:, :, d].reshape(-1), (cells, np.maximum(ref, 0).reshape(-1))), shape=(nc, nv))
        A = A + Bd @ sp.diags(rau) @ Bd.T
        Aabs = Aabs + abs(Bd) @ sp.diags(rau) @ abs(Bd).T
    return S, A.tocsr(), Aabs.tocsr()


@pytest.mark.gpu
@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("mesh", MESHES, ids=["%d_%d_%d" % m for m in MESHES])
@pytest.mark.parametrize("kind", sorted(KIND))
def test_assembled_products(native, monkeypatch, kind, mesh, wide):
    import torch
    if wide:
        monkeypatch.setenv("NDS_SELL_COL32", "1")
    kw, form, dt = KIND[kind]
    S, A, Aabs = _solver(native, mesh, **kw)
    eps = float(np.finfo(dt).eps)
    rng = np.random.default_rng(S.nc)
    for x in (rng.standard_normal(S.nc), np.ones(S.nc), np.eye(1, S.nc, S.nc // 2)[0]):
        x = x.astype(dt)
        xd = torch.from_numpy(x).cuda()
        y = torch.full_like(xd, float("nan"))
        torch.cuda.synchronize()
        native.solver_apply_operator_form(S, form, xd, y)
        ax = np.abs(x.astype(np.float64))
        lim = 62 * eps * (Aabs @ ax)
        if kind == "half":
            hs = 2.0 ** np.floor(np.log2(2048.0 / A.diagonal().max()))
            lim += 2.0 ** -11 * (abs(A) @ ax) + 2.0 ** -25 / hs * ((A != 0) @ ax)
        err = np.abs(y.cpu().numpy().astype(np.float64) - A @ x.astype(np.float64))
        assert np.all(err <= lim), float((err - lim).max())


@pytest.mark.gpu
@pytest.mark.parametrize("mesh", MESHES, ids=["%d_%d_%d" % m for m in MESHES])
def test_assembled_edge_weights(native, mesh):
    import torch
    S, A, Aabs = _solver(native, mesh, precision="mixed", p_krylov="fgmres")
    nc = S.nc
    nbr = torch.zeros(4 * nc, dtype=torch.int32, device="cuda")
    ew = torch.zeros(4 * nc, dtype=torch.float32, device="cuda")
    ds = torch.zeros(nc, dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    native.solver_stage_graph(S, nbr, ew, ds)
    nbr, ew, ds = nbr.cpu().numpy().reshape(nc, 4), ew.cpu().numpy().reshape(nc, 4), ds.cpu().numpy().astype(np.float64)
    eps = 2.0 ** -23
    d = A.diagonal()
    assert np.all(np.abs(ds - d ** -0.5) <= 4 * eps * d ** -0.5)
    i = np.repeat(np.arange(nc), 4).reshape(nc, 4)
    want = np.where(nbr >= 0, np.asarray(A[i, np.maximum(nbr, 0)].todense()) * ds[i] * ds[np.maximum(nbr, 0)], 0.0)
    assert np.any(nbr < 0) and np.any(nbr >= 0)
    assert np.all(np.abs(ew - want) <= 4 * eps * np.maximum(np.abs(want), 1e-6))
