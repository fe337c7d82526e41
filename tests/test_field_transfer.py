"""Upload and download of fields at row lengths around a warp and around the
values one pass of a warp takes, with odd and short other extents: FP64 storage
returns the bytes, FP32 storage the values rounded once."""
import numpy as np
import pytest

import fluid_simulator_backup_b200 as fs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [fs.FS_PRECISION_FP64, fs.FS_PRECISION_FP32_REFINE])
@pytest.mark.parametrize("n", [(3, 3, 3), (31, 5, 4), (32, 7, 3), (33, 3, 11), (127, 4, 3), (255, 3, 5), (256, 4, 3), (300, 3, 3)])
def test_round_trip(n, precision):
    rng = np.random.default_rng(n[0])
    with fs.Solver(n, 1.0 / n[0], precision=precision) as s:
        sent = {k: rng.standard_normal(s.shape(k)) for k in ("phi", "u", "v", "w", "pressure")}
        for k, a in sent.items():
            s.upload(k, a)
        for k, a in sent.items():
            stored = a.astype(np.float32).astype(np.float64) if precision == fs.FS_PRECISION_FP32_REFINE and k != "pressure" else a
            assert np.array_equal(s.download(k), stored), k
