"""PCG as one kernel of one cluster against the loop of kernels
(NDS_RESIDENT=0) on small meshes: the same method in another order of sums.
FP64: equal iteration counts, iterates to 1e-9 relative (rounding amplified by
the solves); FP32 state as the FP32 path against FP64; mixed and FP32 V-cycle:
every solve meets its own target p_rtol = 1e-6, as do the fields, in as many
iterations give or take two.  Sizes: parts of equal and unequal length, fewer
coarse rows than blocks, several cells per thread, and 7,680 cells, whose FP64
operators do not fit the shared memory; the smoother's degrees 1 (Jacobi), 2, 3
and 4.  The profiler (whose runs are bitwise equal) shows which form ran.
"""
from __future__ import annotations

import numpy as np
import pytest

from conftest import rel_l2

CFG = dict(re=20.0, alpha_u=0.7, alpha_p=0.3, p_rtol=1e-6, p_max=400, amg_terminal=60, max_outer=10,
           pressure_solver="pcg")
SA = dict(amg_hierarchy="sa", amg_smoother="cheb2")
CASES = {
    "fp64": (dict(SA), 1e-9, 1e-9),
    "fp64_terminal": (dict(SA, amg_terminal=1000), 1e-9, 1e-9),
    "degree3": (dict(SA, amg_cheb_degree=3), 1e-9, 1e-9),
    "degree4": (dict(SA, amg_cheb_degree=4), 1e-9, 1e-9),
    "jacobi": (dict(amg_hierarchy="cf", cf_interp="exti", cf_pmax=8, amg_smoother="jacobi", amg_jacobi_omega=0.5), 1e-9,
               1e-9),
    "fp32": (dict(SA, precision="fp32", p_rtol=1e-4), 1e-3, 1e-3),
    "amg_fp32": (dict(SA, precision="amg_fp32"), 1e-5, 1e-6),
    "mixed": (dict(SA, precision="mixed", p_guess=2), 1e-5, 1e-6),
    "mixed_half": (dict(SA, precision="mixed", amg_half=1), 1e-5, 1e-6),
    "mixed_half_wide": (dict(SA, precision="mixed", amg_half=1), 1e-5, 1e-6),
}
MESHES = [(2, 8, 6), (2, 8, 7), (3, 24, 7), (3, 16, 12), (4, 16, 16)]  # 720, 840, 4,536, 4,608, 7,680 cells
# more than the form's 512 coarse rows (the classical hierarchy keeps a quarter of the cells)
TOO_LARGE = {("jacobi", (3, 24, 7)), ("jacobi", (3, 16, 12)), ("jacobi", (4, 16, 16))}


@pytest.mark.gpu
@pytest.mark.parametrize("case,mesh", [(c, m) for c in sorted(CASES) for m in MESHES if (c, m) not in TOO_LARGE],
                         ids=lambda v: v if isinstance(v, str) else "%d_%d_%d" % v)
def test_resident_pcg_matches_the_loop(native, monkeypatch, case, mesh):
    from nodals_b200 import meshgen
    kw, tol_cont, tol_field = CASES[case]
    nr, nt, nz = mesh
    m = native.Mesh.from_tetmesh(meshgen.pipe_mesh(nr=nr, ntheta=nt, nz=nz, length=0.5 * nz, jitter=0.05, seed=nz))
    P = native.Problem(m, **dict(CFG, **kw))
    if case.endswith("wide"):
        monkeypatch.setenv("NDS_SELL_COL32", "1")
    monkeypatch.setenv("NDS_RESIDENT", "8000")  # also above the size rule
    A, A2 = native.Solver(P), native.Solver(P)
    monkeypatch.setenv("NDS_RESIDENT", "0")
    B = native.Solver(P)
    A2.profile(True)
    B.profile(True)
    for _ in range(4):
        a, a2, b = A.step(), A2.step(), B.step()
        assert (a.p_its, a.rel_cont, a.p_rel) == (a2.p_its, a2.rel_cont, a2.p_rel)  # reproducible
        assert abs(a.rel_cont - b.rel_cont) <= tol_cont * abs(b.rel_cont), (a.it, a.rel_cont, b.rel_cont)
        assert abs(a.p_its - b.p_its) <= (0 if tol_field == 1e-9 else 2), (a.it, a.p_its, b.p_its)
    assert A2.profile_read()["pcg_resident"][0] > 0 and B.profile_read()["pcg_resident"][0] == 0
    for x, y in zip(A.fields(), B.fields()):
        assert rel_l2(x, y) <= tol_field


@pytest.mark.gpu
@pytest.mark.parametrize("mesh", [(2, 8, 7), (3, 16, 12)], ids=["one_kernel", "loop"])
@pytest.mark.parametrize("case", ["fp64", "mixed_half"])
def test_graphs_off_runs_the_same_solves(native, monkeypatch, case, mesh):
    """NDS_NO_GRAPHS=1 and the profiler keep the form a solver takes by its
    size: bitwise-equal runs (840 cells: one kernel; 4,608: the loop)."""
    from nodals_b200 import meshgen
    nr, nt, nz = mesh
    m = native.Mesh.from_tetmesh(meshgen.pipe_mesh(nr=nr, ntheta=nt, nz=nz, length=0.5 * nz, jitter=0.05, seed=nz))
    P = native.Problem(m, **dict(CFG, **CASES[case][0]))
    A, C = native.Solver(P), native.Solver(P)
    C.profile(True)
    monkeypatch.setenv("NDS_NO_GRAPHS", "1")
    B = native.Solver(P)
    for _ in range(4):
        a, b, c = A.step(), B.step(), C.step()
        assert (a.p_its, a.rel_cont, a.p_rel) == (b.p_its, b.rel_cont, b.p_rel) == (c.p_its, c.rel_cont, c.p_rel)
    assert (C.profile_read()["pcg_resident"][0] > 0) == (mesh[0] == 2)
    for x, y, z in zip(A.fields(), B.fields(), C.fields()):
        assert np.array_equal(x, y) and np.array_equal(x, z)


@pytest.mark.gpu
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("mesh,rows,one_kernel", [((2, 16, 8), 500, True), ((3, 16, 6), 536, False),
                                                  ((3, 16, 10), 834, False)])
def test_coarse_rows_line(native, mesh, rows, one_kernel, precision):
    """The form is taken up to 512 coarse rows, above which the loop of
    kernels is faster."""
    from nodals_b200 import meshgen
    nr, nt, nz = mesh
    m = native.Mesh.from_tetmesh(meshgen.pipe_mesh(nr=nr, ntheta=nt, nz=nz, length=0.5 * nz, jitter=0.05, seed=0))
    P = native.Problem(m, **dict(CFG, **CASES["jacobi"][0], precision=precision, p_rtol=1e-4))
    assert abs(P.array("amg.A0.row").size - 1 - rows) <= 10
    S = native.Solver(P)
    S.profile(True)
    S.step()
    assert (S.profile_read()["pcg_resident"][0] > 0) == one_kernel
