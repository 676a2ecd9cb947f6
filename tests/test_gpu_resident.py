"""Solves on the grid whose shares of p and x fit shared memory wholly, in part
(all of p and some of x, some of p only) and hardly at all: against the cluster
kernel, which keeps its vectors another way, and the oracle's operator.  With 900
blocks a CTA of a grid of 1, 3, 8 and 16 owns 900, 300, 113 and 57 blocks, and a
chunk of 2 blocks of the FP32 form is half filled at the ends of odd shares.
"""
import numpy as np
import pytest

import oracle
from cup2d_b200 import Solver
from cup2d_b200 import _lib as L
from cup2d_b200.problems import sized_mesh

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("grid", [1, 3, 8, 16])
def test_resident_shares(cuda, grid, precision):
    import torch
    m = sized_mesh(np.random.default_rng(8), 900)
    b = m.rhs_fourier(7)
    x0 = np.random.default_rng(2).standard_normal(m.ncells)
    bd = torch.from_numpy(b).to(cuda)

    def solve(g, **kw):
        x = torch.from_numpy(x0).to(cuda)
        with Solver(m, precision=precision, **kw) as s:
            s.set_grid(g)
            st = s.solve_device(bd, x)
        return x.cpu().numpy(), st

    if precision == "fp64":
        # the same algorithm in another summation order: 3 FP64 iterations agree
        # to rounding (the bar of the cluster's own comparison)
        kw = dict(tol_rel=0.0, max_iter=3, subtract_mean=False)
        xg, sg = solve(grid, **kw)
        xc, sc = solve(0, **kw)
        assert sg["iterations"] == sc["iterations"] == 3
        assert np.linalg.norm(xg - xc) < 1e-11 * np.linalg.norm(xc)
    # a capped solve returns the iterate whose residual it reports, a converged
    # one meets its tolerance: both by the oracle's operator on the returned x
    A = oracle.Matrix(m)
    bz = b - b.mean()
    xg, sg = solve(grid, tol_rel=0.0, max_iter=150)
    err = np.abs(bz - A.spmv(xg)).max()
    assert abs(err - sg["err_final"]) <= 1e-6 * sg["err_init"]
    xg, sg = solve(grid, tol_rel=1e-8, max_iter=5000)
    assert sg["status"] == L.OK
    assert np.abs(bz - A.spmv(xg)).max() <= 2e-8 * sg["err_init"]
