"""The streaming kernels of the FP64 AMG levels (x staged in shared memory) and
of the restriction, forced on small levels (NDS_STREAM_ROWS=1, with every level
explicit: NDS_DENSE_MB=0), against the kernels of a lane group per row: the
same sums in another order.  The forced levels of the small meshes have fewer
rows than blocks, rows longer than a round of loads and ragged ends; on 205,320
cells the first level's 12,419 rows give every block and warp several rows, so
that the next row's data is loaded ahead.  FP64: equal iteration counts and
iterates to 1e-9 relative; FP32 and FP16 levels (restriction only): every solve
meets its own target p_rtol = 1e-6, as do the fields, in as many iterations
give or take two.
"""
from __future__ import annotations

import pytest

from conftest import rel_l2

CFG = dict(re=20.0, alpha_u=0.7, alpha_p=0.3, p_rtol=1e-6, p_max=400, amg_terminal=16, max_outer=10,
           pressure_solver="pcg")
SA = dict(amg_hierarchy="sa", amg_smoother="cheb2")
CASES = {
    "fp64": (dict(SA), 1e-9, 1e-9),
    "fp64_jacobi": (dict(amg_hierarchy="cf", cf_interp="exti", cf_pmax=8, amg_smoother="jacobi", amg_jacobi_omega=0.5),
                    1e-9, 1e-9),
    "fp64_wide": (dict(SA), 1e-9, 1e-9),
    "half": (dict(SA, precision="mixed", amg_half=1), 1e-5, 1e-6),
    "fp32": (dict(SA, precision="amg_fp32"), 1e-5, 1e-6),
}


@pytest.mark.gpu
@pytest.mark.parametrize("case,mesh", [(c, m) for c in sorted(CASES) for m in ("pipe_tiny", "pipe_small", "large")
                                       if (c, m) != ("fp64_jacobi", "large")])
def test_streaming_levels_match(native, meshes, monkeypatch, case, mesh):
    kw, tol_cont, tol_field = CASES[case]
    monkeypatch.setenv("NDS_DENSE_MB", "0")
    monkeypatch.setenv("NDS_RESIDENT", "0")
    if case.endswith("wide"):
        monkeypatch.setenv("NDS_SELL_COL32", "1")
    if mesh == "large":
        from nodals_b200 import meshgen
        m = meshgen.pipe_mesh(nr=12, ntheta=40, nz=59, jitter=0.05, seed=59)
        kw = dict(kw, amg_terminal=1000)
    else:
        m = meshes(mesh)
    P = native.Problem(native.Mesh.from_tetmesh(m), **dict(CFG, **kw))
    if mesh == "large":  # more rows than the lane groups of 296 blocks and the warps of the restriction's grid
        assert P.array("amg.A0.row").size - 1 > max(296 * 32, 148 * 6 * 8)
    A = native.Solver(P)
    monkeypatch.setenv("NDS_STREAM_ROWS", "1")
    B = native.Solver(P)
    for _ in range(4):
        a, b = A.step(), B.step()
        assert abs(a.rel_cont - b.rel_cont) <= tol_cont * abs(b.rel_cont), (a.it, a.rel_cont, b.rel_cont)
        assert abs(a.p_its - b.p_its) <= (0 if tol_field == 1e-9 else 2), (a.it, a.p_its, b.p_its)
    for x, y in zip(A.fields(), B.fields()):
        assert rel_l2(x, y) <= tol_field
