"""The seven-point stencil kernels on the grids where their column layout,
their z chunks and their in-register wall extrapolation can go wrong: 3 and 4
cells a side (every sample beyond a wall), rows one longer than a tile, ragged
planes walked as consecutive columns, a long and a flat box.  Against the FP64
oracle.

Tolerances: one update is a sum of a few dozen terms, so FP64 results agree to
1e-12 of the field's scale; FP32 contexts round inputs (given FP32 here) only
in the result and in the correction terms, 2e-6 of the scale (32 eps32).  Ten
Sussman steps: tenfold."""
import numpy as np
import pytest

import fluid_simulator_backup_b200 as fs
from oracle import fs_oracle as O

pytestmark = pytest.mark.gpu

SIZES = [(3, 3, 3), (4, 3, 5), (33, 9, 4), (32, 8, 40), (65, 17, 7), (5, 70, 6), (7, 4, 131), (40, 33, 36)]
PRECISIONS = [(fs.FS_PRECISION_FP64, 1e-12), (fs.FS_PRECISION_FP32_REFINE, 2e-6)]


def fields(n, seed):
    nx, ny, nz = n
    rng = np.random.default_rng(seed)
    x, y, z = ((np.arange(m) + 0.5) / nx for m in n)
    r = np.sqrt((x[None, None, :] - 0.45) ** 2 + (y[None, :, None] - 0.4 * ny / nx) ** 2 +
                (z[:, None, None] - 0.6 * nz / nx) ** 2)
    phi = (r - 0.3 * min(n) / nx) * (1.0 + 0.1 * np.sin(3.0 * x)[None, None, :])
    out = [phi, rng.normal(size=(nz, ny, nx + 1)), rng.normal(size=(nz, ny + 1, nx)), rng.normal(size=(nz + 1, ny, nx))]
    return [a.astype(np.float32).astype(np.float64) for a in out]


def solver(n, precision, f, **kw):
    s = fs.Solver(n, 1.0 / n[0], precision=precision, viscosity=0, **kw)
    for k, a in zip(("phi", "u", "v", "w"), f):
        s.upload(k, a)
    return s


def err(a, b):
    return np.abs(a - b).max() / np.abs(b).max()


@pytest.mark.parametrize("precision,tol", PRECISIONS)
@pytest.mark.parametrize("n", SIZES)
def test_advections(n, precision, tol):
    f = fields(n, 2)
    dx = 1.0 / n[0]
    dt = 0.2 * dx
    with solver(n, precision, f) as s:
        s.advect_levelset(dt)
        assert err(s.download("phi"), O.weno5_levelset(*f, dx, dt, 1e-6)) < tol
        s.advect_velocity(dt)
        for k, ref in zip("uvw", O.weno5_velocity(*f[1:], dx, dt, 1e-6)):
            assert err(s.download(k), ref) < tol
    if precision == fs.FS_PRECISION_FP64:  # (in FP32 a tie of two ENO differences may fall the other way)
        with solver(n, precision, f, velocity_scheme=fs.FS_VELOCITY_ENO3) as s:
            s.advect_velocity(dt)
            for k, ref in zip("uvw", O.eno3_velocity(*f[1:], dx, dt)):
                assert err(s.download(k), ref) < tol


@pytest.mark.parametrize("iterations", [1, 10])
@pytest.mark.parametrize("precision,tol", PRECISIONS)
@pytest.mark.parametrize("n", SIZES)
def test_reinitialisation(n, precision, tol, iterations):
    f = fields(n, 3)
    dx = 1.0 / n[0]
    with solver(n, precision, f, reinit_iterations=iterations) as s:
        s.reinitialize()
        got = s.download("phi")
    assert err(got, O.reinitialization_block(f[0], dx, iterations, 5, 1e-6)) < 10 * tol
