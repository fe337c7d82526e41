"""The multigrid-preconditioned pressure solve, the default of FP32 + FP64
refinement contexts: against the FP64 oracle's projection and against the
red-black solve of the same system, at the extents where its hierarchy and
its packed rows can go wrong (3 cells a side; odd extents at several levels;
one axis much longer; the first level small enough, and just too large, for
the one-block levels)."""
import numpy as np
import pytest

import fluid_simulator_backup_b200 as fs
from oracle import fs_oracle as O

pytestmark = pytest.mark.gpu


def level_set(n, kind):
    nx, ny, nz = n
    x, y, z = ((np.arange(m) + 0.5) / nx for m in n)
    X, Y, Z = x[None, None, :], y[None, :, None], z[:, None, None]
    if kind == "layer":  # a flat interface a tenth of a cell above a plane of cell centres
        return np.broadcast_to(Y - (y[ny // 2] + 0.1 / nx), (nz, ny, nx)).copy()
    return np.sqrt((X - 0.5) ** 2 + (Y - 0.4 * ny / nx) ** 2 + (Z - 0.5 * nz / nx) ** 2) - 0.3 * min(n) / nx


def state(n, kind, seed):
    nx, ny, nz = n
    rng = np.random.default_rng(seed)
    u, v, w = O.zero_walls(0.3 * rng.normal(size=(nz, ny, nx + 1)), 0.3 * rng.normal(size=(nz, ny + 1, nx)),
                           0.3 * rng.normal(size=(nz + 1, ny, nx)))
    return level_set(n, kind), u, v, w, 50.0 * rng.normal(size=(nz, ny, nx))


def project(n, precond, fields, tolerance, **kw):
    kw = dict(dict(rho_neg=1.0, rho_pos=1000.0, max_iteration=40000), **kw)
    with fs.Solver(n, 1.0 / n[0], precision=fs.FS_PRECISION_FP32_REFINE, tolerance=tolerance,
                   pressure_preconditioner=precond, **kw) as s:
        for k, a in zip(("phi", "u", "v", "w", "pressure"), fields):
            s.upload(k, a)
        rep = s.project(1e-3)
        return rep, s.download("pressure"), [s.download(k) for k in "uvw"]


def scaled(a, b):
    return np.abs(a - b).max() / max(np.abs(b).max(), 1e-300)


@pytest.mark.parametrize("host_loop", [0, 1])
@pytest.mark.parametrize("kind", ["sphere", "layer"])
@pytest.mark.parametrize("n", [(3, 3, 3), (5, 4, 3), (17, 18, 19), (33, 35, 34), (37, 40, 39), (70, 9, 6), (6, 7, 66)])
def test_matches_oracle_and_red_black(n, kind, host_loop):
    """The solve meets 1e-9 in the FP64 residual; pressures agree to the
    tolerance of test_red_black.py, velocities to the rounding of their FP32
    storage (2^-24 relative, and the solve's share).  The red-black solve from
    the same guess gives the same pressure, its constant included: both
    conserve one weighted sum, up to the FP32 rounding of the directions."""
    fields = state(n, kind, 7)
    rep, p, vel = project(n, fs.FS_PRECOND_DEFAULT, fields, 1e-9, host_loop=host_loop)
    assert rep["rel_residual"] <= 1e-9
    assert rep["iterations"] <= 60
    ru, rv, rw, rp, _ = O.projection(*fields[:4], 1.0 / n[0], 1e-3, 1.0, 1000.0, 1e-12, 40000, mode="corrected",
                                     criterion="rel")
    assert scaled(p - p.mean(), rp - rp.mean()) < 2e-6
    for a, b in zip(vel, (ru, rv, rw)):
        assert scaled(a, b) < 2e-5
    rep2, p2, _ = project(n, fs.FS_PRECOND_RED_BLACK, fields, 1e-9)
    assert rep2["rel_residual"] <= 1e-9
    assert scaled(p, p2) < 2e-5


def test_iterations_do_not_grow_with_the_grid():
    its = []
    for m in (24, 48, 96):
        n = (m, m, m)
        rep, _, _ = project(n, fs.FS_PRECOND_DEFAULT, state(n, "sphere", 3), 1e-6)
        assert rep["rel_residual"] <= 1e-6
        its.append(rep["iterations"])
    assert max(its) <= 40, its


def test_unreachable_tolerance_and_cap():
    """A tolerance below what FP64 can reach ends at the cap with the best
    pressure kept (the red-black solve takes over from the cycle); a cap of
    one iteration is reported; both leave the context usable."""
    n = (20, 22, 21)
    fields = state(n, "sphere", 5)
    with fs.Solver(n, 1.0 / n[0], precision=fs.FS_PRECISION_FP32_REFINE, rho_neg=1.0, rho_pos=1000.0, tolerance=0.0,
                   max_iteration=200) as s:
        for k, a in zip(("phi", "u", "v", "w", "pressure"), fields):
            s.upload(k, a)
        rep = s.project(1e-3, allow_not_converged=True)
        assert rep["status"] == fs.FS_NOT_CONVERGED and rep["rel_residual"] < 1e-9
        s.set_params(tolerance=1e-8, max_iteration=1)
        for k, a in zip(("u", "v", "w", "pressure"), fields[1:]):
            s.upload(k, a)
        rep = s.project(1e-3, allow_not_converged=True)
        assert rep["status"] == fs.FS_NOT_CONVERGED and rep["iterations"] == 1
        s.set_params(max_iteration=1000)
        assert s.project(1e-3)["rel_residual"] <= 1e-8


def test_right_hand_side_without_a_value():
    """A velocity of NaN leaves nothing to solve: reported by the divergence, as
    by the red-black solve, not refused."""
    n = (20, 22, 21)
    fields = [a.copy() for a in state(n, "sphere", 5)]
    fields[1][3, 4, 5] = np.nan
    for precond in (fs.FS_PRECOND_RED_BLACK, fs.FS_PRECOND_DEFAULT):
        rep, _, _ = project(n, precond, fields, 1e-8)
        assert rep["status"] == fs.FS_OK and rep["iterations"] == 0 and np.isnan(rep["div_l2"])


@pytest.mark.parametrize("n", [(30, 34, 18), (26, 24, 70), (66, 18, 40), (33, 65, 31), (64, 64, 64), (80, 20, 79)])
def test_levels_split_over_a_cluster(n):
    """Small levels in slabs over the blocks of a cluster: fewer planes than
    blocks, uneven slabs, one and two slots a thread.  The same pressure as the
    red-black solve, in the few iterations of an intact cycle (at most 40, as
    above)."""
    fields = state(n, "sphere", 7)
    rep, p, _ = project(n, fs.FS_PRECOND_DEFAULT, fields, 1e-9)
    assert rep["rel_residual"] <= 1e-9 and rep["iterations"] <= 40
    p2 = project(n, fs.FS_PRECOND_RED_BLACK, fields, 1e-9)[1]
    assert scaled(p, p2) < 2e-5


@pytest.mark.parametrize("n", [(88, 90, 86), (93, 91, 95), (97, 99, 98)])
def test_slots_per_thread_on_either_side_of_the_rule(n):
    """Finest grids whose half sweeps take one and four slots a thread (444
    blocks of four lie between 92^3 and 96^3), with odd rows: the pressure of
    the red-black solve, as above."""
    fields = state(n, "sphere", 8)
    rep, p, _ = project(n, fs.FS_PRECOND_DEFAULT, fields, 1e-9)
    assert rep["rel_residual"] <= 1e-9 and rep["iterations"] <= 40
    assert scaled(p, project(n, fs.FS_PRECOND_RED_BLACK, fields, 1e-9)[1]) < 2e-5
