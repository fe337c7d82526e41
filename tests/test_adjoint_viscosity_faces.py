"""The viscosity adjoint where its faces differ: constant coefficients on either
side of the interface band, the band itself, extrapolated samples beyond each
wall with the interface meeting it, and boxes of few and of ragged cells.

Central differences of the forward against the adjoint, as in the transpose
tests of test_adjoint.py: the truncation error is (h |d phi| / band)^2 < 1e-9 and
the rounding 1e-14 / h = 1e-9 of the fields, both far below the bound 1e-6 that
those tests use."""
import numpy as np
import pytest

import fluid_simulator_backup_b200 as fs

from test_adjoint import FIELDS_VEL, rand_like, rel, transpose_check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(3, 3, 3), (37, 9, 5), (34, 3, 17), (6, 21, 20)])
@pytest.mark.parametrize("tilt", [(1.0, 0.3, -0.2), (-0.2, 1.0, 0.4), (0.3, 0.2, -1.0)])
def test_transpose(n, tilt):
    nx, ny, nz = n
    dx = 1.0 / nx
    rng = np.random.default_rng(sum(n))
    x, y, z = ((np.arange(m) + 0.5) / m - 0.45 for m in n)
    phi = (tilt[0] * nx * x[None, None, :] + tilt[1] * ny * y[None, :, None] + tilt[2] * nz * z[:, None, None]) * dx
    phi = phi + 0.02 * dx * rng.standard_normal(phi.shape)
    X = {"phi": phi, "u": rng.standard_normal((nz, ny, nx + 1)), "v": rng.standard_normal((nz, ny + 1, nx)),
         "w": rng.standard_normal((nz + 1, ny, nx))}
    dX = rand_like(X, rng, ("phi", "u", "v", "w"))
    dX["phi"] *= 0.1 * dx
    for st in (X, dX):
        st["u"][:, :, [0, -1]] = 0.0
        st["v"][:, [0, -1], :] = 0.0
        st["w"][[0, -1], :, :] = 0.0
    Ybar = rand_like(X, rng, FIELDS_VEL)
    with fs.Solver(n, dx, precision=fs.FS_PRECISION_FP64, mu_neg=2e-2, mu_pos=5e-2, viscosity_tolerance=1e-14,
                   viscosity_max_iteration=100000) as s:
        lhs, rhs = transpose_check(s, lambda s: s.viscosity(0.5 * dx), lambda s: s.viscosity_adjoint(0.5 * dx), X, dX, Ybar,
                                   FIELDS_VEL, ("phi", "u", "v", "w"), 1e-5, (1.0, 1000.0), (0.3, 70.0))
    assert rel(lhs, rhs) < 1e-6, (lhs, rhs)
