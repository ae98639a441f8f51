"""The tensor-core row kernel of the FP32C triangle form factor (the automatic choice on row grids).

Bound: the project's FP32C tolerance, 1e-5 norm-wise against the FP64 oracle.  Each term's error
is at most that of the SFU sine and cosine and of the 22- and 24-bit digits, about 1e-6 of the
tile's largest triangle, so sums that do not cancel below a tenth of their terms stay inside.
"""
import numpy as np
import pytest

import hipgisaxs_b200 as hg
from hipgisaxs_b200 import meshes

pytestmark = pytest.mark.gpu
TOL32 = 1e-5


def cloud(rng, T, scale=6.0):
    sd = np.zeros((T, 8))
    sd[:, 0] = rng.uniform(0.2, 3.0, T)
    n = rng.normal(size=(T, 3))
    sd[:, 1:4] = n / np.linalg.norm(n, axis=1)[:, None]
    sd[:, 4:7] = rng.normal(scale=scale, size=(T, 3))
    return sd


def detector(po, ncol, nrow, kind):
    """(qx, qy, qz) of a detector grid: four real blocks, four complex ones, or one complex."""
    G = po.Grid(ncol, nrow, -1.9, 0.0, 2.0, 3.0, 0.2, 10.0, (6e-6, 8e-8) if kind != "real" else (0.0, 0.0))
    return G.qx, G.qy, G.qz_ext[:ncol * nrow].copy() if kind == "one" else G.qz_ext


@pytest.mark.parametrize("kind", ["real", "complex", "one"])
@pytest.mark.parametrize("ncol,nrow,ntri", [
    (2, 3, 1), (17, 5, 31), (127, 2, 32), (128, 2, 33), (129, 2, 511), (64, 3, 512), (257, 2, 513),
    (40, 3, 1500),   # tiles split over CTAs
    (130, 9, 4700),  # ten tiles: stages and accumulators reused
])
def test_edges_of_tiles_chunks_and_columns(ctx, po, kind, ncol, nrow, ntri):
    rng = np.random.default_rng(1000 * ncol + ntri)
    sd = cloud(rng, ntri)
    R = po.rot_mul(po.rot_axis(2, 0.2), po.rot_axis(1, 0.1))
    qx, qy, qz = detector(po, ncol, nrow, kind)
    g = hg.QGrid.from_arrays(ctx, qx, qy, qz, ncol)
    assert g.mode == (1 if kind == "real" else 2)
    ref = po.ff_approx_triangle(sd, qx, qy, qz, R)
    for out_type in ("c128", "c64"):
        f = hg.ff_triangles(ctx, g, sd, R, "f32c", out_type=out_type)
        ok = np.isfinite(ref)  # a q-point at q = 0 is 0 / 0 in both
        assert np.array_equal(ok, np.isfinite(f)) and po.rel_err(f[ok], ref[ok]) < TOL32


def test_wide_phases(ctx, po):
    """One tile spread over 2 um: its in-plane phases take the explicit reduction."""
    sd = cloud(np.random.default_rng(5), 300, scale=400.0)
    qx, qy, qz = detector(po, 130, 4, "real")
    g = hg.QGrid.from_arrays(ctx, qx, qy, qz, 130)
    assert po.rel_err(hg.ff_triangles(ctx, g, sd, None, "f32c"), po.ff_approx_triangle(sd, qx, qy, qz)) < TOL32


def test_slabs_of_row_factors(ctx, po):
    """More row factors than are held at a time: several slabs of rows, against the FP64 kernel."""
    V, F = meshes.star_mesh(15.0, 125, 81)
    sd = meshes.shape_def_from_mesh(V, F)
    g = hg.QGrid.create(ctx, 16, 1500, -1.9, 0.0, 2.0, 3.0, 0.0035, 50.677)
    f64 = hg.ff_triangles(ctx, g, sd, None, "f64")
    assert po.rel_err(hg.ff_triangles(ctx, g, sd, None, "f32c"), f64) < TOL32


@pytest.mark.parametrize("ntri", [514, 1024, 1025, 2048, 2049])
def test_order_of_small_and_large_meshes(ctx, po, ntri):
    """Both ways of ordering the triangles, at the line between them."""
    sd = cloud(np.random.default_rng(ntri), ntri)
    qx, qy, qz = detector(po, 20, 2, "real")
    g = hg.QGrid.from_arrays(ctx, qx, qy, qz, 20)
    assert po.rel_err(hg.ff_triangles(ctx, g, sd, None, "f32c"), po.ff_approx_triangle(sd, qx, qy, qz)) < TOL32


@pytest.mark.parametrize("col,value", [(0, np.nan), (0, np.inf), (2, np.nan), (5, np.nan), (6, np.inf)])
def test_a_triangle_that_is_not_finite_is_not_hidden(ctx, po, col, value):
    sd = cloud(np.random.default_rng(6), 600)
    sd[70, col] = value
    qx, qy, qz = detector(po, 33, 3, "real")
    g = hg.QGrid.from_arrays(ctx, qx, qy, qz, 33)
    assert not np.isfinite(hg.ff_triangles(ctx, g, sd, None, "f32c")).any()


@pytest.mark.parametrize("ncol,nrow,ntri", [(64, 800, 300), (64, 60, 506), (150, 400, 506), (150, 400, 513), (30, 1030, 600)])
def test_both_sides_of_the_kernel_choice(ctx, po, ncol, nrow, ntri):
    """Real blocks near the sizes at which the automatic choice goes from one row kernel to the other."""
    sd = cloud(np.random.default_rng(ncol + ntri), ntri)
    qx, qy, qz = detector(po, ncol, nrow, "real")
    g = hg.QGrid.from_arrays(ctx, qx, qy, qz, ncol)
    assert po.rel_err(hg.ff_triangles(ctx, g, sd, None, "f32c"), po.ff_approx_triangle(sd, qx, qy, qz)) < TOL32


@pytest.mark.parametrize("kind", ["real", "complex"])
@pytest.mark.parametrize("spread", [1.0, 3.0])
def test_triangles_of_uneven_size(ctx, po, kind, spread):
    """Areas over orders of magnitude (log-normal): what a term is off is that of the SFU's sine and cosine
    (2^-21.4) and of the phasors' step (2^-23), 5e-7 of the term, and adds up at random: 1e-6 norm-wise, the error
    of the sums of even triangles, not that of the tile's largest triangle times their number."""
    sd = cloud(np.random.default_rng(3), 600)
    sd[:, 0] = np.exp(spread * np.random.default_rng(4).normal(size=600))
    qx, qy, qz = detector(po, 256, 40, kind)
    g = hg.QGrid.from_arrays(ctx, qx, qy, qz, 256)
    ref = po.ff_approx_triangle(sd, qx, qy, qz)
    f = hg.ff_triangles(ctx, g, sd, None, "f32c")
    ok = np.isfinite(ref)
    assert po.rel_err(f[ok], ref[ok]) < 1e-6


@pytest.mark.parametrize("unit", [1e-33, 1e30])
def test_units_of_the_areas(ctx, po, unit):
    sd = cloud(np.random.default_rng(3), 600)
    sd[:, 0] *= unit
    qx, qy, qz = detector(po, 256, 8, "real")
    g = hg.QGrid.from_arrays(ctx, qx, qy, qz, 256)
    ref = po.ff_approx_triangle(sd, qx, qy, qz)
    ok = np.isfinite(ref)
    assert po.rel_err(hg.ff_triangles(ctx, g, sd, None, "f32c")[ok], ref[ok]) < TOL32


@pytest.mark.parametrize("along", ["qy", "qx"])
@pytest.mark.parametrize("width,ncol", [(0.02, 130), (0.1, 130), (0.01, 1)])
def test_zoomed_grids_around_zero(ctx, po, along, width, ncol):
    """Point by point next to q = 0, where F = S / q^2 and S cancels: a term is off by 5e-7 of |q| |n|, so F by
    5e-7 |q| (surface) / (|q|^2 volume), 3e-6 / (|q| D) for a ball of diameter D; 5e-6 (1 + 1 / (|q| D)) allowed."""
    V, F = meshes.star_mesh(15.0, 64, 33)
    sd = meshes.shape_def_from_mesh(V, F)
    nrow = 160
    u = np.tile(np.linspace(-width, 1.01 * width, ncol) if ncol > 1 else 1e-4, nrow)
    v = np.full(ncol * nrow, 1e-5)
    qx, qy = (v, u) if along == "qy" else (u, v)
    z = np.repeat(np.linspace(1e-4, width, nrow), ncol).astype(complex)
    a, b = z + 1e-4, z - 5e-5
    qz = np.concatenate([a, -b, b, -a])
    g = hg.QGrid.from_arrays(ctx, qx, qy, qz, ncol)
    assert g.mode == 1
    qd = 30.0 * np.sqrt(np.tile(qx ** 2 + qy ** 2, 4) + qz.real ** 2)
    ref = hg.ff_triangles(ctx, g, sd, None, "f64")
    e = np.abs(hg.ff_triangles(ctx, g, sd, None, "f32c") - ref) / np.abs(ref)
    assert np.all(e[qd < 2] < 5e-6 * (1 + 1 / qd[qd < 2]))
