"""A pressure that already meets the tolerance costs the multigrid solve the
operator's set-up and a true residual: no cycle."""
import numpy as np
import pytest

import fluid_simulator_backup_b200 as fs
from oracle import fs_oracle as O

pytestmark = pytest.mark.gpu

FP32 = dict(precision=fs.FS_PRECISION_FP32_REFINE, rho_neg=1.0, rho_pos=1000.0, max_iteration=2000, viscosity=0)


def state(n, seed):
    nx, ny, nz = n
    rng = np.random.default_rng(seed)
    x, y, z = ((np.arange(m) + 0.5) / nx for m in n)
    phi = np.sqrt((x[None, None, :] - 0.5) ** 2 + (y[None, :, None] - 0.4 * ny / nx) ** 2 +
                  (z[:, None, None] - 0.5 * nz / nx) ** 2) - 0.3 * min(n) / nx
    u, v, w = O.zero_walls(0.3 * rng.normal(size=(nz, ny, nx + 1)), 0.3 * rng.normal(size=(nz, ny + 1, nx)),
                           0.3 * rng.normal(size=(nz + 1, ny, nx)))
    return phi, u, v, w


@pytest.mark.parametrize("host_loop", [0, 1])
@pytest.mark.parametrize("n", [(3, 3, 3), (24, 25, 23), (97, 99, 98)])
def test_second_projection_of_the_same_velocity(n, host_loop):
    phi, u, v, w = state(n, 1)
    with fs.Solver(n, 1.0 / n[0], tolerance=1e-8, host_loop=host_loop, **FP32) as s:
        s.upload("phi", phi)
        out = []
        for _ in range(2):
            for k, a in zip("uvw", (u, v, w)):
                s.upload(k, a)
            out.append((s.project(1e-3), s.download("pressure"), [s.download(k) for k in "uvw"]))
    (first, p, vel), (second, q, vel2) = out
    assert first["iterations"] > 0 and second["iterations"] == 0
    assert max(first["rel_residual"], second["rel_residual"]) <= 1e-8
    assert np.array_equal(p, q) and all(np.array_equal(a, b) for a, b in zip(vel, vel2))


@pytest.mark.parametrize("n,levels", [((24, 25, 23), 5), ((97, 99, 98), 7)])
def test_launches_of_a_step_at_rest(n, levels):
    """A fluid at rest without gravity: three projections with nothing to solve.
    More than the red-black solve's look at its guess are two kernels per level at
    most and six others; a cycle would be eight to fourteen."""
    phi = state(n, 1)[0]
    launches = []
    for precond in (fs.FS_PRECOND_DEFAULT, fs.FS_PRECOND_RED_BLACK):
        with fs.Solver(n, 1.0 / n[0], tolerance=1e-8, gravity=(0.0, 0.0, 0.0), pressure_preconditioner=precond,
                       **FP32) as s:
            s.upload("phi", phi)
            rep = s.step(1e-4)
        assert rep["pcg_iterations"] == 0
        launches.append(rep["kernel_launches"])
    assert launches[0] - launches[1] <= 3 * (2 * (levels - 1) + 2)
