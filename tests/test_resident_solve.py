"""The resident FP64 pressure solve (one cooperative kernel, a brick of the box
per SM) at the sizes where its bricks and variants change: bricks of one cell,
uneven bricks, each number of cells per thread, the iterate in global memory,
and a grid that no longer fits (the three-kernel iteration).

Small grids: against the oracle's projection.  All: the residual of the
downloaded pressure, evaluated in numpy with the oracle's operator, equals the
reported one and meets the tolerance; FP64 rounding of the residual is
eps64 * diag * |p| / |b| < 1e-11 here, so the bound 1e-8 is the solve's."""
import numpy as np
import pytest

import fluid_simulator_backup_b200 as fs
from oracle import fs_oracle as O

pytestmark = pytest.mark.gpu


def case(n, seed):
    nx, ny, nz = n
    rng = np.random.default_rng(seed)
    x, y, z = ((np.arange(m) + 0.5) / nx for m in n)
    phi = np.sqrt((x[None, None, :] - 0.5) ** 2 + (y[None, :, None] - 0.4 * ny / nx) ** 2 +
                  (z[:, None, None] - 0.5 * nz / nx) ** 2) - 0.3 * min(n) / nx
    u, v, w = O.zero_walls(0.3 * rng.normal(size=(nz, ny, nx + 1)), 0.3 * rng.normal(size=(nz, ny + 1, nx)),
                           0.3 * rng.normal(size=(nz + 1, ny, nx)))
    return phi, u, v, w


def run(n, fields, faithful, **kw):
    with fs.Solver(n, 1.0 / n[0], precision=fs.FS_PRECISION_FP64, rho_neg=1.0, rho_pos=1000.0, viscosity=0,
                   flags=fs.FS_FLAG_FAITHFUL_PROJECTION if faithful else 0, **dict(dict(max_iteration=40000), **kw)) as s:
        for k, a in zip(("phi", "u", "v", "w"), fields):
            s.upload(k, a)
        rep = s.project(1e-3, allow_not_converged=True)
        return rep, s.download("pressure"), [s.download(k) for k in "uvw"]


def residual(n, fields, p, faithful):
    phi, u, v, w = fields
    dx = 1.0 / n[0]
    op = O.poisson_operator(phi, dx, 1.0, 1000.0, deflate=faithful)
    b = -O.divergence(u, v, w, dx, 1e-3)
    b = b - b.mean()
    return np.linalg.norm(b - O.apply_poisson(op, p)) / np.linalg.norm(b)


@pytest.mark.parametrize("faithful", [False, True])
@pytest.mark.parametrize("n", [(3, 3, 3), (5, 4, 7), (17, 18, 19), (40, 6, 9), (7, 33, 12), (26, 25, 24)])
def test_small_against_oracle(n, faithful):
    f = case(n, 1)
    rep, p, vel = run(n, f, faithful, tolerance=1e-11)
    ru, rv, rw, rp, info = O.projection(*f, 1.0 / n[0], 1e-3, 1.0, 1000.0, 1e-11, 40000,
                                        mode="faithful" if faithful else "corrected", criterion="rel")
    assert rep["status"] == fs.FS_OK and rep["rel_residual"] <= 1e-11
    assert abs(rep["iterations"] - info["iterations"]) <= max(3, 0.02 * info["iterations"])
    if not faithful:
        p, rp = p - p.mean(), rp - rp.mean()
    assert np.abs(p - rp).max() < 1e-7 * np.abs(rp).max()
    for a, b in zip(vel, (ru, rv, rw)):
        assert np.abs(a - b).max() < 1e-7 * np.abs(b).max()


# bricks of up to 4, 8, 16, 24, 32 cells per thread, the iterate in global memory, and no fit
@pytest.mark.parametrize("n", [(50, 51, 49), (63, 66, 65), (80, 85, 82), (96, 96, 96), (104, 101, 103), (112, 110, 111),
                               (124, 120, 122)])
def test_every_variant_solves(n):
    f = case(n, 2)
    rep, p, vel = run(n, f, False, tolerance=1e-8)
    assert rep["status"] == fs.FS_OK
    true = residual(n, f, p, False)
    assert true <= 1.01e-8 and abs(true - rep["rel_residual"]) < 1e-10
    assert rep["div_l2"] <= 2e-8 * np.linalg.norm(O.divergence(*f[1:], 1.0 / n[0], 1.0))


def test_caps_and_criteria():
    n = (18, 17, 20)
    f = case(n, 3)
    rep, p, _ = run(n, f, False, tolerance=1e-10, max_iteration=7)
    assert rep["status"] == fs.FS_NOT_CONVERGED and rep["iterations"] == 7
    rep0, p0, _ = run(n, f, False, tolerance=1e-10, max_iteration=0)
    assert rep0["status"] == fs.FS_NOT_CONVERGED and rep0["iterations"] == 0 and not p0.any()
    assert residual(n, f, p, False) < 1.0
    rep, _, _ = run(n, f, True, tolerance=1e-5, stop=fs.FS_STOP_ABSOLUTE)
    assert rep["status"] == fs.FS_OK and rep["rz"] < 1e-10
    bad = [a.copy() for a in f]
    bad[1][3, 4, 5] = np.nan
    with pytest.raises(fs.FsError) as e:
        run(n, bad, False, tolerance=1e-8)
    assert e.value.status == fs.FS_NONFINITE
