"""Contexts of small boxes that solve at the same time, one thread each: results
are those of a context alone, bit for bit, and the solves run beside each other.

Before the resident solves left SMs free, sixteen FP64 contexts of 16^3 took
turns (0.65 ms a projection each); beside each other they take 0.12.  The bound
of half the turn-taking time stands between the two and far from both."""
import threading
import time

import numpy as np
import pytest

import fluid_simulator_backup_b200 as fs
from oracle import fs_oracle as O

pytestmark = pytest.mark.gpu


def state(n, seed):
    rng = np.random.default_rng(seed)
    x = (np.arange(n) + 0.5) / n
    phi = np.sqrt((x[None, None, :] - 0.5) ** 2 + (x[None, :, None] - 0.4) ** 2 + (x[:, None, None] - 0.5) ** 2) - 0.3
    u, v, w = O.zero_walls(0.3 * rng.normal(size=(n, n, n + 1)), 0.3 * rng.normal(size=(n, n + 1, n)),
                           0.3 * rng.normal(size=(n + 1, n, n)))
    return phi, u, v, w, np.zeros((n, n, n))


def project(s, fields):
    for k, a in zip(("phi", "u", "v", "w", "pressure"), fields):
        s.upload(k, a)
    s.project(1e-3)
    return s.download("pressure")


def in_threads(jobs):
    threads = [threading.Thread(target=j) for j in jobs]
    t = time.perf_counter()
    for q in threads:
        q.start()
    for q in threads:
        q.join()
    return time.perf_counter() - t


@pytest.mark.parametrize("n", [16, 33])
@pytest.mark.parametrize("precision,precond", [(fs.FS_PRECISION_FP64, fs.FS_PRECOND_DEFAULT),
                                               (fs.FS_PRECISION_FP32_REFINE, fs.FS_PRECOND_RED_BLACK),
                                               (fs.FS_PRECISION_FP32_REFINE, fs.FS_PRECOND_DEFAULT)])
def test_results_do_not_depend_on_neighbours(n, precision, precond):
    contexts = 8
    fields = [state(n, q) for q in range(contexts)]
    kw = dict(precision=precision, rho_neg=1.0, rho_pos=1000.0, tolerance=1e-8, max_iteration=40000, viscosity=0,
              pressure_preconditioner=precond)
    solvers = [fs.Solver((n, n, n), 1.0 / n, **kw) for _ in range(contexts)]
    alone = [project(s, f) for s, f in zip(solvers, fields)]
    out = [[] for _ in range(contexts)]

    def job(q):
        for _ in range(5):
            out[q].append(project(solvers[q], fields[q]))

    in_threads([lambda q=q: job(q) for q in range(contexts)])
    for q in range(contexts):
        assert len(out[q]) == 5 and all(np.array_equal(p, alone[q]) for p in out[q])
        solvers[q].close()


def test_small_solves_run_beside_each_other():
    n, contexts, repeats = 16, 16, 10
    fields = state(n, 0)
    kw = dict(precision=fs.FS_PRECISION_FP64, rho_neg=1.0, rho_pos=1000.0, tolerance=1e-8, max_iteration=40000,
              viscosity=0)
    solvers = [fs.Solver((n, n, n), 1.0 / n, **kw) for _ in range(contexts)]
    for s in solvers:
        project(s, fields)

    def job(s):
        for _ in range(repeats):
            project(s, fields)

    one = min(in_threads([lambda: job(solvers[0])]) for _ in range(3))
    many = min(in_threads([lambda s=s: job(s) for s in solvers]) for _ in range(3))
    for s in solvers:
        s.close()
    assert many < 0.5 * contexts * one, (many, one)
