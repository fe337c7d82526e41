"""The semi-implicit viscosity's system kernel where its two shortcuts can go
wrong: faces all of whose samples lie outside the smearing width (no Heaviside
evaluated), faces next to the walls (samples extrapolated), and boxes in which
every face is both.  One solve against the FP64 oracle.

Tolerance: both sides solve the same symmetric system to 1e-13 relative in
FP64; its condition number here is below 1e3 (viscous numbers of order 1,
densities 1 to 100), so 1e-9 of the scale.  FP32 contexts: 2e-5 (FP32 system,
vectors and storage at that condition number: 1e3 * eps32 / 3)."""
import numpy as np
import pytest

import fluid_simulator_backup_b200 as fs
from oracle import fs_oracle as O

pytestmark = pytest.mark.gpu


def level_set(n, kind):
    nx, ny, nz = n
    x, y, z = ((np.arange(m) + 0.5) / nx for m in n)
    X, Y, Z = x[None, None, :], y[None, :, None], z[:, None, None]
    if kind == "far":  # one phase everywhere
        return np.full((nz, ny, nx), 10.0 / nx)
    if kind == "corner":  # the interface cuts three walls
        return np.sqrt(X ** 2 + Y ** 2 + Z ** 2) - 0.55 * min(n) / nx
    return np.broadcast_to(Y - 0.5 * ny / nx + 0.1 * X / nx, (nz, ny, nx)).copy()


@pytest.mark.parametrize("precision,tol", [(fs.FS_PRECISION_FP64, 1e-9), (fs.FS_PRECISION_FP32_REFINE, 2e-5)])
@pytest.mark.parametrize("kind", ["far", "corner", "layer"])
@pytest.mark.parametrize("n", [(3, 3, 3), (4, 5, 3), (33, 6, 9), (12, 34, 7), (20, 18, 31)])
def test_matches_oracle(n, kind, precision, tol):
    nx, ny, nz = n
    rng = np.random.default_rng(1)
    f = [level_set(n, kind), *O.zero_walls(rng.normal(size=(nz, ny, nx + 1)), rng.normal(size=(nz, ny + 1, nx)),
                                           rng.normal(size=(nz + 1, ny, nx)))]
    f = [a.astype(np.float32).astype(np.float64) for a in f]
    P = dict(rho_neg=1.0, rho_pos=100.0, mu_neg=0.05, mu_pos=2.0)
    dx, dt = 1.0 / nx, 0.02 / nx
    with fs.Solver(n, dx, precision=precision, viscosity=1,
                   viscosity_tolerance=1e-13 if precision == fs.FS_PRECISION_FP64 else 1e-7, **P) as s:
        for k, a in zip(("phi", "u", "v", "w"), f):
            s.upload(k, a)
        s.viscosity(dt)
        got = [s.download(k) for k in "uvw"]
    ref = O.viscosity_semi_implicit(*f, dx, dt, *P.values(), 1e-13, 10000)[0]
    for a, b in zip(got, ref):
        assert np.abs(a - b).max() < tol * np.abs(b).max()
