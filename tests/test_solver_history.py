"""What one solve leaves in a context's buffers must not reach the next: the
FP32 + FP64 refinement solvers (multigrid, red-black, Jacobi) share vectors, so
each is run after the others, and after input without a value, in one context
and compared with the same call in a fresh one.

The solvers sum in a fixed order, so equal means equal in every bit."""
import numpy as np
import pytest

import fluid_simulator_backup_b200 as fs
from oracle import fs_oracle as O

pytestmark = pytest.mark.gpu

NAMES = ("phi", "u", "v", "w", "pressure")
FP32 = dict(precision=fs.FS_PRECISION_FP32_REFINE, rho_neg=1.0, rho_pos=1000.0, tolerance=1e-9, max_iteration=2000,
            viscosity=0)


def state(n, seed):
    nx, ny, nz = n
    rng = np.random.default_rng(seed)
    x, y, z = ((np.arange(m) + 0.5) / nx for m in n)
    phi = np.sqrt((x[None, None, :] - 0.5) ** 2 + (y[None, :, None] - 0.4 * ny / nx) ** 2 +
                  (z[:, None, None] - 0.5 * nz / nx) ** 2) - 0.3 * min(n) / nx
    u, v, w = O.zero_walls(0.3 * rng.normal(size=(nz, ny, nx + 1)), 0.3 * rng.normal(size=(nz, ny + 1, nx)),
                           0.3 * rng.normal(size=(nz + 1, ny, nx)))
    return phi, u, v, w, np.zeros((nz, ny, nx))


def upload(s, fields):
    for k, a in zip(NAMES, fields):
        s.upload(k, a)


def project(s, fields, precond, **kw):
    s.set_params(pressure_preconditioner=precond, **kw)
    upload(s, fields)
    rep = s.project(1e-3, allow_not_converged=True)
    return rep["status"], rep["iterations"], s.download("pressure")


def without_a_value(fields, name):
    bad = [a.copy() for a in fields]
    bad[NAMES.index(name)][3, 4, 5] = np.nan
    return bad


def same(a, b):
    return a[:2] == b[:2] and np.array_equal(a[2], b[2])


@pytest.mark.parametrize("n,name", [((20, 22, 18), "u"), ((20, 22, 18), "phi"), ((21, 22, 20), "u"),
                                    ((21, 22, 20), "phi"), ((125, 126, 122), "u"), ((125, 126, 122), "phi")])
def test_after_a_field_without_a_value(n, name):
    """A NaN velocity is a right-hand side of NaN (FS_OK, nothing solved), a NaN
    level set is an error (FS_NONFINITE, or FS_NOT_CONVERGED where only the FP32
    couplings see it); then good fields solve as in a fresh context, with every
    solver.  The last box is too large for a resident solve."""
    good = state(n, 1)
    bad = without_a_value(good, name)
    for precond in (fs.FS_PRECOND_RED_BLACK, fs.FS_PRECOND_JACOBI_BF16, fs.FS_PRECOND_DEFAULT):
        with fs.Solver(n, 1.0 / n[0], **FP32) as s:
            fresh = project(s, good, precond)
        assert fresh[0] == fs.FS_OK and fresh[1] > 0
        with fs.Solver(n, 1.0 / n[0], **FP32) as s:
            upload(s, bad)
            if name == "phi":
                with pytest.raises(fs.FsError) as e:
                    s.project(1e-3)
                assert e.value.status in (fs.FS_NONFINITE, fs.FS_NOT_CONVERGED)
            else:
                assert s.project(1e-3)["iterations"] == 0
            assert same(project(s, good, precond), fresh), precond


def test_adjoint_after_a_field_without_a_value():
    """The step adjoint's transposed solves are red-black: bars after a
    projection with a NaN velocity, against a fresh context's.  FP64 atomics add
    in any order, so the two runs' solves end at different remainders of 1e-9;
    the system's condition (density ratio 1000 times about n^2) lets these reach
    1e-4 of a bar.  A solve that starts from NaN does not converge."""
    n = (14, 15, 12)
    good = state(n, 2)
    rng = np.random.default_rng(3)
    bars = {k: rng.normal(size=a.shape) for k, a in zip(("adj_phi", "adj_u", "adj_v", "adj_w"), good)}

    def adjoint(s):
        upload(s, good)
        for k, a in bars.items():
            s.upload(k, a)
        s.step_adjoint(1e-4)
        return {k: s.download(k) for k in bars}

    kw = dict(FP32, reinit_iterations=2)
    with fs.Solver(n, 1.0 / n[0], **kw) as s:
        fresh = adjoint(s)
    with fs.Solver(n, 1.0 / n[0], **kw) as s:
        upload(s, without_a_value(good, "u"))
        s.project(1e-3)
        after = adjoint(s)
    for k in bars:
        assert np.abs(after[k] - fresh[k]).max() <= 1e-4 * np.abs(fresh[k]).max(), k


@pytest.mark.parametrize("n", [(21, 22, 20), (3, 4, 5), (93, 91, 95), (97, 99, 98)])
def test_multigrid_after_red_black_with_odd_rows(n):
    """An odd row's last packed slot holds a cell of one colour only; the
    red-black solve's value there (large: velocities a thousand times the next
    solve's, stopped after three iterations) must not enter the multigrid
    solve's sums."""
    fields = state(n, 4)
    large = [fields[0]] + [1e3 * a for a in fields[1:4]] + [fields[4]]
    with fs.Solver(n, 1.0 / n[0], **FP32) as s:
        fresh = project(s, fields, fs.FS_PRECOND_DEFAULT)
        project(s, large, fs.FS_PRECOND_RED_BLACK, max_iteration=3)
        after = project(s, fields, fs.FS_PRECOND_DEFAULT, max_iteration=FP32["max_iteration"])
    assert fresh[0] == fs.FS_OK and same(after, fresh), (after[:2], fresh[:2])


def test_projection_after_step_adjoint_with_odd_rows():
    n = (15, 14, 13)
    fields = state(n, 5)
    rng = np.random.default_rng(6)
    with fs.Solver(n, 1.0 / n[0], **dict(FP32, reinit_iterations=2)) as s:
        fresh = project(s, fields, fs.FS_PRECOND_DEFAULT)
        upload(s, fields)
        for k, a in zip(("adj_phi", "adj_u", "adj_v", "adj_w"), fields):
            s.upload(k, 1e3 * rng.normal(size=a.shape))
        s.step_adjoint(1e-4)
        assert same(project(s, fields, fs.FS_PRECOND_DEFAULT), fresh)


@pytest.mark.parametrize("precision", [fs.FS_PRECISION_FP64, fs.FS_PRECISION_FP32_REFINE])
def test_resumed_step_repeats(precision, tmp_path):
    """A step after a checkpoint, in the context that wrote it (after a step, a
    step adjoint and a projection there) and in a fresh one that reads it: equal in
    every bit, in a box whose resident FP64 solve has more mixed cells than its
    list holds."""
    n = (97, 95, 96)
    fields = state(n, 7)
    kw = dict(FP32, precision=precision, tolerance=1e-7, viscosity=1, reinit_iterations=2, max_iteration=20000)
    path = str(tmp_path / "state")
    out = []
    with fs.Solver(n, 1.0 / n[0], **kw) as s:
        upload(s, fields)
        s.step(1e-4)
        s.step_adjoint(1e-4)
        s.write_state(path)
        s.project(1e-4)
        s.read_state(path)
        s.step(1e-4)
        out.append([s.download(k) for k in NAMES])
    with fs.Solver(n, 1.0 / n[0], **kw) as s:
        s.read_state(path)
        s.step(1e-4)
        out.append([s.download(k) for k in NAMES])
    for k, a, b in zip(NAMES, *out):
        assert np.array_equal(a, b), k
