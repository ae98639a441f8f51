"""hgx_ff_tune with the tensor-core kernel among its candidates."""
import numpy as np
import pytest

import hipgisaxs_b200 as hg
from test_gpu_ff_rows_f64 import cloud

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dn2", [(0.0, 0.0), (6e-6, 8e-8)])
def test_the_tensor_core_kernel_is_a_candidate(ctx, po, dn2):
    """256 x 200 pixels x 3,000 triangles, where it takes about half the FP32 kernel's time: it wins, nothing is
    stored, and automatic calls stay as they were, also after another choice had been stored."""
    G = po.Grid(256, 200, -1.9, 0.0, 2.0, 3.0, 0.2, 10.0, dn2)
    g = hg.QGrid.from_arrays(ctx, G.qx, G.qy, G.qz_ext)
    sd = cloud(np.random.default_rng(1), 3000)
    before = hg.ff_triangles(ctx, g, sd, None, "f32c")
    best, ms, times = hg.ff_tune(ctx, g, sd, None, "c128", reps=3)
    assert best == 0 and 0 < ms < min(times.values())
    assert set(times) == ({4, 2, 1, -2, -4, -8} if dn2 == (0.0, 0.0) else {4, 2, 1})
    after = hg.ff_triangles(ctx, g, sd, None, "f32c")
    assert np.array_equal(before, after, equal_nan=True)


def test_a_shape_is_stored_and_replaced(ctx, po):
    """One tile of triangles: the shapes alone are ranked and the choice is used; a later choice replaces it."""
    G = po.Grid(256, 200, -1.9, 0.0, 2.0, 3.0, 0.2, 10.0)
    g = hg.QGrid.from_arrays(ctx, G.qx, G.qy, G.qz_ext)
    sd = cloud(np.random.default_rng(1), 3000)
    untuned = hg.ff_triangles(ctx, g, sd, None, "f32c")
    best = hg.ff_tune(ctx, g, sd[:300], None, "c128", reps=3)[0]
    assert best != 0
    hand = hg.ff_triangles(ctx, g, sd, None, "f32c", pixels_per_thread=best)
    assert np.array_equal(hg.ff_triangles(ctx, g, sd, None, "f32c"), hand, equal_nan=True)
    assert hg.ff_tune(ctx, g, sd, None, "c128", reps=3)[0] == 0
    assert np.array_equal(hg.ff_triangles(ctx, g, sd, None, "f32c"), untuned, equal_nan=True)


def test_pixels_per_thread_refusals(ctx, po):
    G = po.Grid(20, 4, -1.9, 0.0, 2.0, 3.0, 0.2, 10.0)
    g = hg.QGrid.from_arrays(ctx, G.qx, G.qy, G.qz_ext)
    for p in (3, 8, -1, 1 << 20):
        with pytest.raises(hg.HgxError):
            hg.ff_triangles(ctx, g, cloud(np.random.default_rng(1), 30), None, "f32c", pixels_per_thread=p)
