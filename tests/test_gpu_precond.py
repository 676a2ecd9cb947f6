"""The block solve of the solve kernels (P^-1 by sine transforms), alone, against
the oracle's dense product in 64 bits: one block, odd counts (a half-filled
FP32 chunk), more chunks than warps in flight; inputs of one sign, smooth,
alternating, over six decades and of one cell."""
import numpy as np
import pytest

import oracle
from cup2d_b200 import Mesh, Solver

pytestmark = pytest.mark.gpu

# Relative 2-norm.  Four products with an orthonormal matrix, each rounding at
# 2^-22 of its operand's norm in FP32 (two-term TF32 splits, FP32 sums),
# independently: 2 x 2^-22 = 4.8e-7 in quadrature (a dense FP32 product with P^-1
# comes out at 5e-7 to 8e-7 on the constant, smooth and alternating inputs).  In
# FP64 8 x 2^-53 a product (sums of eight); the oracle's dense sums of 64 add 64 x 2^-53.
BAR32 = 2 * 2.0 ** -22
BAR64 = (4 * 8 + 64) * 2.0 ** -53


def _inputs(nb):
    rng = np.random.default_rng(nb)
    ix, iy = np.arange(64) % 8, np.arange(64) // 8
    r = rng.random((nb, 1))
    return {
        "random": rng.standard_normal((nb, 64)),
        "constant": r * np.ones(64),
        "smooth": np.sin(0.1 * ix + 6.0 * r) * np.cos(0.13 * iy),
        "checkerboard": r * (-1.0) ** (ix + iy),
        "six decades": rng.standard_normal((nb, 64)) * 10.0 ** (-6.0 * rng.random((nb, 64))),
        "one cell": np.eye(64)[rng.integers(0, 64, nb)],
    }


@pytest.mark.parametrize("shape", [(1, 1), (3, 1), (17, 1), (31, 29), (260, 257)])
def test_block_solve_matches_oracle(cuda, shape):
    import torch
    m = Mesh.uniform(*shape, 1, 0, 1.0)
    P = oracle.pinv()
    with Solver(m) as s:
        for name, v in _inputs(m.nblocks).items():
            p = torch.from_numpy(v.reshape(-1)).to(cuda)
            z = torch.full_like(p, float("nan"))
            s.precond(p, z)
            ref = oracle.precond(P, v.reshape(-1))
            assert np.linalg.norm(z.cpu().numpy() - ref) <= BAR64 * np.linalg.norm(ref), name
            p32 = p.float()
            z32 = torch.full_like(p32, float("nan"))
            s.precond(p32, z32)
            ref = oracle.precond(P, p32.double().cpu().numpy())
            assert np.linalg.norm(z32.double().cpu().numpy() - ref) <= BAR32 * np.linalg.norm(ref), name


def test_block_solve_places(cuda):
    """Buffers aligned to their type only, and z in place of p, as before."""
    import torch
    m = Mesh.uniform(5, 3, 1, 0, 1.0)
    g = torch.Generator(device="cuda").manual_seed(1)
    with Solver(m) as s:
        for dt in (torch.float64, torch.float32):
            p = torch.randn(m.ncells, generator=g, device=cuda, dtype=dt)
            z = torch.empty_like(p)
            s.precond(p, z)
            buf = torch.full((m.ncells + 2,), 7.0, device=cuda, dtype=dt)
            buf[1:-1] = p
            s.precond(buf[1:-1], buf[1:-1])
            assert torch.equal(buf[1:-1], z) and buf[0] == 7.0 and buf[-1] == 7.0
