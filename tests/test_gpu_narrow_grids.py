"""Row grids of few columns, scattered q-points (which count as rows of one) and single qz blocks: both
sides of the choice between the row kernels and the plain FP64 and FP32 ones, against the oracle at the kernels'
bounds (1e-12 in FP64, 1e-5 in FP32C)."""
import numpy as np
import pytest

import hipgisaxs_b200 as hg
from test_gpu_ff_rows_f64 import cloud

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["real4", "complex4", "real1", "complex1"])
@pytest.mark.parametrize("ncol,nrow,ntri", [
    (1, 1, 40), (1, 200, 700), (1, 2900, 300), (1, 9000, 70), (2, 2600, 300), (3, 3001, 130), (7, 2100, 200),
    (13, 1500, 130), (16, 1600, 130), (15, 1023, 939), (40, 1100, 65), (70, 500, 130),
])
def test_both_kernels(ctx, po, kind, ncol, nrow, ntri):
    rng = np.random.default_rng(100 * ncol + ntri)
    n = ncol * nrow
    qx, qy = rng.uniform(-0.1, 0.1, n), rng.uniform(-2, 2, n)
    z = np.repeat(rng.uniform(0.02, 3, nrow), ncol).astype(complex)
    if kind.startswith("complex"):
        z += 1e-3j * (1 + z.real)
    a, b = z + 0.2, z - 0.2
    qz = z if kind.endswith("1") else np.concatenate([a, -b, b, -a] if kind == "real4" else [a, b, -a, -b])
    g = hg.QGrid.from_arrays(ctx, qx, qy, qz, ncol)
    assert g.mode == (1 if kind == "real4" else 2)
    sd = cloud(rng, ntri)
    R = po.rot_mul(po.rot_axis(2, 0.2), po.rot_axis(1, 0.1))
    ref = po.ff_approx_triangle(sd, qx, qy, qz, R)
    assert po.rel_err(hg.ff_triangles(ctx, g, sd, R, "f64"), ref) < 1e-12
    assert po.rel_err(hg.ff_triangles(ctx, g, sd, R, "f32c"), ref) < 1e-5
    assert po.rel_err(hg.ff_triangles_arrays(ctx, sd, qx, qy, qz, R, "f64"), ref) < 1e-12
