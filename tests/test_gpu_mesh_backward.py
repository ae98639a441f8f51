"""The tensor-core backward pass of the FP32C mesh adjoint (grids wider than 128 columns) against
the plain FP64 forward and adjoint.

Bound: the project's 1e-4 norm-wise for the FP32C vertex gradient.  The counts lie below a
model that every pixel exceeds, so the residuals do not cancel."""
import numpy as np
import pytest

import hipgisaxs_b200 as hg
from hipgisaxs_b200 import fitting, meshes, model

pytestmark = pytest.mark.gpu
SUB = (4.88e-6, 7.37e-8, 0.0, -1)
DN2 = (-2 * 4.88e-6, -2 * 7.37e-8)


def gradients(ctx, po, ncol, nrow, V, F, masked=False):
    G = po.Grid(ncol, nrow, -2.0, 0.0, 2.0, 3.0, 0.2, 10.0)
    g = hg.QGrid.create(ctx, ncol, nrow, -2.0, 0.0, 2.0, 3.0, G.alpha_i, G.k0)
    rowfc = model.propagation_coeffs(ctx, g, [SUB], G.k0, G.alpha_i, 0, per_row=True)
    R = po.rot_mul(po.rot_axis(2, 0.3), po.rot_axis(0, 0.15))
    rng = np.random.default_rng(ncol + len(F))
    mask = (rng.uniform(size=G.n) > 0.1).astype(np.uint32) if masked else None
    inten = fitting.mesh_chi2_grad(ctx, g, V, F, rowfc, DN2, None, None, 1.0, 1.0, R, want_grad=False,
                                   want_intensity=True, precision="f64")[2]
    scale = 1e4 / inten.max()
    counts = scale * inten * rng.uniform(0.2, 0.6, G.n)
    return [fitting.mesh_chi2_grad(ctx, g, V, F, rowfc, DN2, counts, mask, scale, 1.0, R, precision=p)[1]
            for p in ("f32c", "f64")]


@pytest.mark.parametrize("ncol,nrow,nfaces", [
    (128, 3, 129),   # the FP32 kernel
    (129, 2, 1), (160, 2, 127), (192, 3, 128), (225, 2, 129), (256, 5, 511), (257, 4, 513),
    (513, 3, 600),   # three items per row
    (300, 70, 1280),
    (130, 2, 1), (226, 2, 129), (258, 4, 513), (514, 3, 600),
])
def test_edges_of_tiles_chunks_and_rows(ctx, po, ncol, nrow, nfaces):
    V, F = meshes.icosphere(8.0, 3, jitter=0.2, seed=3)
    got, ref = gradients(ctx, po, ncol, nrow, V + [40.0, -25.0, 10.0], F[:nfaces], masked=nrow > 2)
    ok = np.isfinite(ref)  # an odd width has a pixel at q = 0: 0 / 0 in the form factor, in both
    assert np.array_equal(ok, np.isfinite(got)) and (not ok.any() or po.rel_err(got[ok], ref[ok]) < 1e-4)


def test_wide_phases(ctx, po):
    """Tiles of 40 nm: their in-plane phases, up to 85 rad and so 5e-6 rad off in FP32, take the
    explicit reduction."""
    V, F = meshes.icosphere(30.0, 3)
    got, ref = gradients(ctx, po, 140, 3, V, F)
    assert po.rel_err(got, ref) < 1e-4


@pytest.mark.parametrize("unit", [1e-18, 1e-15, 1e20])
def test_units_of_the_counts(ctx, po, unit):
    """Counts and scale in other units: seeds of 1e-31, 1e-25 and 1e21, whose squares leave FP32's range."""
    V, F = meshes.icosphere(8.0, 2, jitter=0.2, seed=3)
    G = po.Grid(140, 3, -2.0, 0.0, 2.0, 3.0, 0.2, 10.0)
    g = hg.QGrid.create(ctx, 140, 3, -2.0, 0.0, 2.0, 3.0, G.alpha_i, G.k0)
    rowfc = model.propagation_coeffs(ctx, g, [SUB], G.k0, G.alpha_i, 0, per_row=True)
    inten = fitting.mesh_chi2_grad(ctx, g, V, F, rowfc, DN2, None, None, 1.0, 1.0, None, want_grad=False,
                                   want_intensity=True, precision="f64")[2]
    scale = unit * 1e4 / inten.max()
    counts = scale * inten * np.random.default_rng(2).uniform(0.2, 0.6, G.n)
    got, ref = [fitting.mesh_chi2_grad(ctx, g, V, F, rowfc, DN2, counts, None, scale, 1.0, None, precision=p)[1]
                for p in ("f32c", "f64")]
    assert np.isfinite(ref).all() and np.abs(ref).max() > 0 and po.rel_err(got, ref) < 1e-4


@pytest.mark.parametrize("ncol,nrow,f64", [(160, 200, True), (2048, 96, False)])  # 5 and 32 slabs
def test_slabs_of_seed_digits_share_their_partial_sums(po, ncol, nrow, f64):
    """Several slabs of rows: their sums add up, and the call's device memory stays below the 1 GiB of
    seed digits, 64 MiB of partial sums and some 150 MiB of arrays that go with the pixels or the faces."""
    import torch
    V, F = meshes.star_mesh(15.0, 500, 328)  # 327,000 faces
    ctx = hg.Context(0)
    gradients(ctx, po, 160, 2, V[:3], np.array([[0, 1, 2]], dtype=np.int32))  # loads the kernels
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    G = po.Grid(ncol, nrow, -2.0, 0.0, 2.0, 3.0, 0.2, 10.0)
    g = hg.QGrid.create(ctx, ncol, nrow, -2.0, 0.0, 2.0, 3.0, G.alpha_i, G.k0)
    rowfc = model.propagation_coeffs(ctx, g, [SUB], G.k0, G.alpha_i, 0, per_row=True)
    counts = np.random.default_rng(4).uniform(1.0, 2.0, G.n)
    args = (ctx, g, V, F, rowfc, DN2, counts, None, 1.0, 1.0, None)
    got = fitting.mesh_chi2_grad(*args, precision="f32c")[1]
    used = free - torch.cuda.mem_get_info()[0]
    ref = fitting.mesh_chi2_grad(*args, precision="f64")[1] if f64 else got
    ctx.close()
    assert used < (1 << 30) + (64 << 20) + (150 << 20)
    assert po.rel_err(got, ref) < 1e-4


@pytest.mark.parametrize("ncol,nrow,nfaces", [(129, 2, 128), (160, 148, 129), (300, 70, 1280)])
def test_blocks_that_follow_one_another_leave_each_other_alone(ctx, po, ncol, nrow, nfaces):
    """One item per block, and several with fewer and more blocks than SMs: the same bits on every call."""
    V, F = meshes.icosphere(8.0, 3, jitter=0.2, seed=3)
    first = gradients(ctx, po, ncol, nrow, V, F[:nfaces])[0]
    for _ in range(5):
        assert np.array_equal(gradients(ctx, po, ncol, nrow, V, F[:nfaces])[0], first, equal_nan=True)
