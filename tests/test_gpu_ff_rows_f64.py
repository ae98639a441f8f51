"""The FP64 row kernel of the triangle form factor against the FP64 oracle: norm-wise 1e-12, the
bound of the plain FP64 kernel (each term's phase and phasor err by a few 1e-16, the sums by the
rounding of the additions)."""
import numpy as np
import pytest

import hipgisaxs_b200 as hg

pytestmark = pytest.mark.gpu
TOL64 = 1e-12


def cloud(rng, T, scale=6.0):
    sd = np.zeros((T, 8))
    sd[:, 0] = rng.uniform(0.2, 3.0, T)
    n = rng.normal(size=(T, 3))
    sd[:, 1:4] = n / np.linalg.norm(n, axis=1)[:, None]
    sd[:, 4:7] = rng.normal(scale=scale, size=(T, 3))
    return sd


@pytest.mark.parametrize("kind", ["real", "complex", "one"])
@pytest.mark.parametrize("ncol,nrow,ntri", [
    (2, 3, 1), (31, 5, 63), (33, 4, 64), (65, 3, 65), (129, 2, 129), (257, 2, 300),
    (20, 2, 2000),    # triangles split over CTAs
    (300, 640, 130),  # two pixels per thread
])
def test_edges_of_stagings_rows_and_columns(ctx, po, kind, ncol, nrow, ntri):
    sd = cloud(np.random.default_rng(1000 * ncol + ntri), ntri)
    R = po.rot_mul(po.rot_axis(2, 0.2), po.rot_axis(1, 0.1))
    G = po.Grid(ncol, nrow, -1.87, 0.01, 2.0, 3.0, 0.2, 10.0, (6e-6, 8e-8) if kind != "real" else (0.0, 0.0))
    qz = G.qz_ext[:ncol * nrow].copy() if kind == "one" else G.qz_ext
    g = hg.QGrid.from_arrays(ctx, G.qx, G.qy, qz, ncol)
    assert g.mode == (1 if kind == "real" else 2)
    ref = po.ff_approx_triangle(sd, G.qx, G.qy, qz, R)
    assert po.rel_err(hg.ff_triangles(ctx, g, sd, R, "f64"), ref) < TOL64
    assert po.rel_err(hg.ff_triangles(ctx, g, sd, R, "f64", out_type="c64"), ref) < 1e-7


def test_far_from_the_origin(ctx, po):
    """Phases of some 2,600 rad: their rounding, about 4e-13, is the reference's too."""
    sd = cloud(np.random.default_rng(8), 200)
    sd[:, 4:7] += (1000.0, -700.0, 300.0)
    G = po.Grid(70, 3, -1.87, 0.01, 2.0, 3.0, 0.2, 10.0)
    g = hg.QGrid.from_arrays(ctx, G.qx, G.qy, G.qz_ext, 70)
    assert po.rel_err(hg.ff_triangles(ctx, g, sd, None, "f64"), po.ff_approx_triangle(sd, G.qx, G.qy, G.qz_ext)) < TOL64


@pytest.mark.parametrize("dn2", [(0.0, 0.0), (6e-6, 4e-8)])
@pytest.mark.parametrize("ncol", [64, 131])
def test_reference_shaped_call_while_qz_is_copied(po, ncol, dn2):
    """From the second call with host arrays of the same sizes on, the FP64 row kernel starts from a
    row table read on the host while the 4N qz values are copied and checked: bit for bit the
    device grid's result.  A q-point off its row's value, and blocks that pair only in the rows'
    first q-points, fail the check and are computed from the full qz."""
    G = po.Grid(ncol, 9, -2.0, 0.0, 2.0, 3.0, 0.2, 10.0, dn2)
    sd = cloud(np.random.default_rng(ncol), 150)
    qz_off, qz_pair = G.qz_ext.copy(), G.qz_ext.copy()
    qz_off[3 * ncol + ncol // 2] += 0.01
    qz_pair[2 * G.n + 5 * ncol + 1] *= 1.5
    ctx = hg.Context(0)
    for qz in (G.qz_ext, G.qz_ext, qz_off, G.qz_ext, qz_pair, G.qz_ext):
        want = hg.ff_triangles(ctx, hg.QGrid.from_arrays(ctx, G.qx, G.qy, qz), sd, None, "f64")
        got = hg.ff_triangles_arrays(ctx, sd, G.qx, G.qy, qz, None, "f64")
        ok = np.isfinite(want)  # a q-point at q = 0 is 0 / 0
        assert np.array_equal(ok, np.isfinite(got)) and np.array_equal(got[ok], want[ok])
    ctx.close()
