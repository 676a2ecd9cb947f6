"""Solves on one thread-block cluster (forests whose vectors fit its shared
memory): against the grid solver, which an explicit grid selects, and the
oracle, at the sizes where the cluster's shares go wrong first: one block, fewer
blocks than CTAs, odd shares (a half-filled FP32 chunk), the largest that fit,
periodic edges, and corner rows longer than the shared-memory rows.
"""
import numpy as np
import pytest

import oracle
from cup2d_b200 import Mesh, Solver
from cup2d_b200 import _lib as L
from cup2d_b200.problems import sized_mesh, small_mesh

pytestmark = pytest.mark.gpu

MESHES = {
    "one_block": lambda: Mesh.uniform(1, 1, 1, 0, 1.0),
    "two_blocks": lambda: Mesh.uniform(2, 1, 1, 0, 2.0),
    "uniform_25": lambda: Mesh.uniform(5, 5, 1, 0, 1.0),
    "small": small_mesh,
    "periodic_x": lambda: Mesh.disks(4, 2, 4, 2.0, [(1.9, 0.5, 0.12)], 0.1, periodic_x=True),
    "periodic_xy": lambda: Mesh.disks(2, 2, 5, 1.0, [(0.03, 0.95, 0.1)], 0.06, periodic_x=True, periodic_y=True),
    "sized_900": lambda: sized_mesh(np.random.default_rng(8), 900),
    "sized_1600": lambda: sized_mesh(np.random.default_rng(21), 1600, 5),
}


def _solve(cuda, m, b, grid, **kw):
    import torch
    x = torch.zeros(m.ncells, dtype=torch.float64, device=cuda)
    with Solver(m, **kw) as s:
        s.set_grid(grid)
        st = s.solve_device(torch.from_numpy(b).to(cuda), x)
    return x.cpu().numpy(), st


def _rel(a, b):
    return np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-300)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("name", list(MESHES))
def test_cluster_against_grid(cuda, name, precision):
    m = MESHES[name]()
    b = m.rhs_fourier(7)
    # the same algorithm in another summation order and another association
    # of the solution update: 3 FP64 iterations agree to rounding
    kw = dict(tol_rel=0.0, max_iter=3, precision=precision, subtract_mean=False)
    if m.nblocks > 1:
        xc, sc = _solve(cuda, m, b, 0, **kw)
        xg, sg = _solve(cuda, m, b, 8, **kw)
        if precision == "fp64":
            assert sc["iterations"] == sg["iterations"] == 3
            assert _rel(xc, xg) < 1e-11
            assert abs(sc["err_final"] - sg["err_final"]) <= 1e-9 * sg["err_init"]
        assert sc["status"] == sg["status"] == L.NOT_CONVERGED
    # converged: the residual is bounded by the stop test; what a residual of
    # 1e-8 leaves open in the solution grows with the forest (kappa ~ 1e5..1e6 on
    # 900..1600 blocks: the grid solver's launch shapes differ by 8e-7 among
    # themselves there, half of it each from the solution), so the bar against
    # the tighter oracle solution is five times that
    kw = dict(tol_rel=1e-8, max_iter=5000, precision=precision)
    xc, sc = _solve(cuda, m, b, 0, **kw)
    assert sc["status"] == L.OK and np.isfinite(xc).all()
    A = oracle.Matrix(m)
    bz = b - b.mean()
    assert np.abs(bz - A.spmv(xc)).max() <= 2e-8 * np.abs(bz).max()
    xo, so = oracle.solve(m, b, tol_rel=1e-9, max_iter=20000)[:2]
    assert _rel(xc, xo) < 4e-6


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_cluster_caps_and_warm_start(cuda, precision):
    """No iteration at all, a warm start that already meets the tolerance,
    and the result of a capped solve (its reported residual is x's own)."""
    import torch
    m = small_mesh()
    b = m.rhs_fourier(3)
    x0 = np.random.default_rng(1).standard_normal(m.ncells)
    d = torch.from_numpy(x0).to(cuda)
    with Solver(m, tol_rel=1e-8, max_iter=0, subtract_mean=False, precision=precision) as s:
        st = s.solve_device(torch.from_numpy(b).to(cuda), d)
        assert st["iterations"] == 0 and np.array_equal(d.cpu().numpy(), x0)
    x, st = _solve(cuda, m, b, 0, tol_rel=1e-8, max_iter=5000, precision=precision)
    d = torch.from_numpy(x).to(cuda)
    tol = 4.0 * st["err_final"]
    with Solver(m, tol_rel=0.0, tol_abs=tol, max_iter=5000, precision=precision) as s:
        st2 = s.solve_device(torch.from_numpy(b).to(cuda), d)
    assert st2["status"] == L.OK and st2["iterations"] <= 1
    x, st = _solve(cuda, m, b, 0, tol_rel=0.0, max_iter=40, precision=precision, subtract_mean=False)
    res = np.abs((b - b.mean()) - oracle.Matrix(m).spmv(x)).max()
    assert abs(res - st["err_final"]) <= 1e-6 * st["err_init"] + 1e-3 * st["err_final"]


def test_cluster_repeats_bit_for_bit(cuda):
    m = MESHES["periodic_xy"]()
    b = m.rhs_fourier(5)
    for precision in ("fp64", "mixed"):
        a = _solve(cuda, m, b, 0, tol_rel=1e-8, max_iter=5000, precision=precision)
        c = _solve(cuda, m, b, 0, tol_rel=1e-8, max_iter=5000, precision=precision)
        assert np.array_equal(a[0], c[0]) and a[1]["iterations"] == c[1]["iterations"]


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_cluster_timeout(cuda, precision):
    """The cluster kernel's own deadline: a 1 ms limit on a solve of some
    hundred iterations (15 us each) to 1e-12.  The call reports it, and the
    handle then solves as a fresh one does, bit for bit."""
    import torch
    from cup2d_b200 import Cup2dError
    m = MESHES["sized_900"]()
    b = torch.from_numpy(m.rhs_fourier(4)).to(cuda)
    kw = dict(tol_rel=1e-8, max_iter=5000, precision=precision)
    with Solver(m, tol_rel=1e-12, max_iter=100000, timeout_ms=1, precision=precision) as s:
        for _ in range(2):
            x = torch.zeros_like(b)
            with pytest.raises(Cup2dError) as e:
                s.solve_device(b, x)
            assert e.value.status == L.TIMEOUT
        s.set_opts(**kw)
        x = torch.zeros_like(b)
        assert s.solve_device(b, x)["status"] == L.OK
    with Solver(m, **kw) as s:
        y = torch.zeros_like(b)
        assert s.solve_device(b, y)["status"] == L.OK
    assert torch.equal(x, y)
