"""The resident red-black iteration (FP32 vectors, FP64 iterate, one cooperative
kernel between two reliable updates) at the sizes where its bricks and variants
change: bricks of one pair of columns, uneven bricks and odd widths, each number
of slots per thread, a deflated first cell, and a grid that no longer fits.

Small grids: against the oracle's projection (faithful: with the deflation).
All: the residual of the downloaded pressure, evaluated in numpy with the
oracle's operator, meets the tolerance; the solver decides on an FP64 residual
whose rounding is eps64 * diag * |p| / |b| < 1e-11 here.  The bound on the pressure
is that of the FP64 solve's test: the same system, solved to the same true residual."""
import numpy as np
import pytest

import fluid_simulator_backup_b200 as fs
from oracle import fs_oracle as O

from test_resident_solve import case, residual

pytestmark = pytest.mark.gpu


def run(n, fields, faithful, **kw):
    kw = dict(dict(max_iteration=40000, tolerance=1e-8), **kw)
    with fs.Solver(n, 1.0 / n[0], precision=fs.FS_PRECISION_FP32_REFINE, rho_neg=1.0, rho_pos=1000.0, viscosity=0,
                   pressure_preconditioner=fs.FS_PRECOND_RED_BLACK,
                   flags=fs.FS_FLAG_FAITHFUL_PROJECTION if faithful else 0, **kw) as s:
        for k, a in zip(("phi", "u", "v", "w"), fields):
            s.upload(k, a)
        rep = s.project(1e-3, allow_not_converged=True)
        return rep, s.download("pressure"), [s.download(k) for k in ("phi", "u", "v", "w")]


def rounded(fields):
    return [a.astype(np.float32).astype(np.float64) for a in fields]


@pytest.mark.parametrize("faithful", [False, True])
@pytest.mark.parametrize("n", [(3, 3, 3), (5, 4, 7), (17, 18, 19), (40, 6, 9), (7, 33, 12), (26, 25, 24)])
def test_small_against_oracle(n, faithful):
    f = rounded(case(n, 1))
    rep, p, _ = run(n, f, faithful, tolerance=1e-11)
    rp = O.projection(*f, 1.0 / n[0], 1e-3, 1.0, 1000.0, 1e-11, 40000,
                      mode="faithful" if faithful else "corrected", criterion="rel")[3]
    assert rep["status"] == fs.FS_OK and rep["rel_residual"] <= 1e-11
    if not faithful:
        p, rp = p - p.mean(), rp - rp.mean()
    assert np.abs(p - rp).max() < 1e-7 * np.abs(rp).max()


@pytest.mark.parametrize("n", [(50, 51, 49), (63, 66, 65), (81, 85, 82), (96, 96, 96), (105, 101, 103), (118, 120, 115),
                               (140, 130, 134)])
def test_every_variant_solves(n):
    f = rounded(case(n, 2))
    rep, p, _ = run(n, f, False)
    assert rep["status"] == fs.FS_OK
    assert residual(n, f, p, False) <= 1.01e-8


def test_caps_and_errors():
    n = (18, 17, 20)
    f = rounded(case(n, 3))
    rep, p, _ = run(n, f, False, max_iteration=7)
    assert rep["status"] == fs.FS_NOT_CONVERGED and rep["iterations"] == 7
    # a level set without a sign in one cell: no solve
    bad = [a.copy() for a in f]
    bad[0][3, 4, 5] = np.nan
    try:
        rep, _, _ = run(n, bad, False, max_iteration=400)
    except fs.FsError as e:
        assert e.status == fs.FS_NONFINITE
    else:
        assert rep["status"] == fs.FS_NOT_CONVERGED
