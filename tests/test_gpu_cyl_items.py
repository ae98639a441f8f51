"""Items of the cylinder batch's FP32C pixel pass: regions around a warp's 32 pixels and around the sizes
at which a lane takes another pixel (32,768 pixels each).

Bound: the FP32C tolerance of chi^2 and its gradient, 1e-5 of the FP64 values; a candidate of
a batch equals the same candidate alone bit by bit."""
import numpy as np
import pytest

import hipgisaxs_b200 as hg
from hipgisaxs_b200 import fitting, model

pytestmark = pytest.mark.gpu
DN2 = (-2 * 4.88e-6, -2 * 7.37e-8)
ROIS = [[0, 0, 1, 1], [3, 1, 1, 31], [7, 2, 32, 1], [9, 300, 3, 11], [40, 8, 33, 33], [0, 0, 128, 256],
        [1, 5, 255, 257], [0, 0, 256, 256], [2, 3, 301, 397], [0, 0, 384, 512], [11, 13, 400, 501]]


@pytest.mark.parametrize("reps", [(20, 20, 1), (1, 7, 1)])
def test_items_of_regions(ctx, reps):
    g = hg.QGrid.create(ctx, 516, 420, -2.0, 0.0, 2.0, 3.0, np.deg2rad(0.2), 50.7)
    rowfc = model.propagation_coeffs(ctx, g, [(4.88e-6, 7.37e-8, 0.0, -1)], 50.7, np.deg2rad(0.2), 0, per_row=True)
    abc, _ = model.lattice_vectors("hex")
    models = [fitting.model_block(5 + 0.1 * i, 10 - 0.2 * i, 20 + 0.3 * i, 0.03 * i, 0.05, 11, reps, DN2, (0, 0, 0), 1.0)
              for i in range(len(ROIS))]
    start = fitting.CylinderBatch(ctx, g, rowfc, abc, ROIS, None, None, 1.0, "f64").forward(models)
    scale = 1e4 / max(i.max() for i in start)
    rng = np.random.default_rng(4)
    counts = np.concatenate([(scale * i * rng.uniform(0.2, 0.6, i.shape)).ravel() for i in start])
    (c32, g32), (c64, g64) = (fitting.CylinderBatch(ctx, g, rowfc, abc, ROIS, counts, None, scale, p).eval(models)
                              for p in ("f32c", "f64"))
    at = 0
    for i, r in enumerate(ROIS):
        assert abs(c32[i] - c64[i]) <= 1e-5 * c64[i]
        assert np.linalg.norm(g32[i] - g64[i]) <= 1e-5 * np.linalg.norm(g64[i])
        one = fitting.CylinderBatch(ctx, g, rowfc, abc, [r], counts[at:at + r[2] * r[3]], None, scale, "f32c")
        c1, g1 = one.eval([models[i]])
        assert c1[0] == c32[i] and np.array_equal(g1[0], g32[i])
        at += r[2] * r[3]


@pytest.mark.parametrize("precision", ["f64", "f32c"])
def test_rows_of_regions_of_unequal_height(ctx, precision):
    """Heights around the rows of a warp (4) and of a block (32) beside a tall region, whose batch launches
    more rows than the others have: each candidate equals the same candidate alone bit by bit."""
    rois = [[3, 5, h, 40] for h in (1, 3, 4, 5, 31, 32, 33)] + [[0, 2, 399, 33]]
    g = hg.QGrid.create(ctx, 516, 420, -2.0, 0.0, 2.0, 3.0, np.deg2rad(0.2), 50.7)
    rowfc = model.propagation_coeffs(ctx, g, [(4.88e-6, 7.37e-8, 0.0, -1)], 50.7, np.deg2rad(0.2), 0, per_row=True)
    abc, _ = model.lattice_vectors("hex")
    models = [fitting.model_block(5 + 0.1 * i, 10 - 0.2 * i, 20 + 0.3 * i, 0.03 * i, 0.05, 11, (20, 20, 1), DN2, (0, 0, 0), 1.0)
              for i in range(len(rois))]
    rng = np.random.default_rng(4)
    counts = [rng.uniform(1, 2, r[2] * r[3]) for r in rois]
    c, gr = fitting.CylinderBatch(ctx, g, rowfc, abc, rois, np.concatenate(counts), None, 1.0, precision).eval(models)
    for i, r in enumerate(rois):
        c1, g1 = fitting.CylinderBatch(ctx, g, rowfc, abc, [r], counts[i], None, 1.0, precision).eval([models[i]])
        assert c1[0] == c[i] and np.array_equal(g1[0], gr[i])
