"""Lattices with repetitions that are not whole numbers, on real qz (sf_lattice_real_kernel and
grain_dwba_real_kernel) against the oracle, whose b-axis numerator takes the unreduced angle.

Bounds: those of the whole repetitions, 1e-11 in FP64 and 1e-5 in FP32C (an angle's rounding, some
1e-15 turn, is the oracle's too, and no point of the structure factors lies within 1e-4 turn of a
peak).  Off the peak of order 0 the b factor grows as 1 / (distance to the peak), so an image's pixel
next to one moves by 4e-11 with the last bit of the scaling, in the oracle as well: images are also
allowed the oracle's own change under 1e-15 of the scaling."""
import copy
import ctypes
import os

import numpy as np
import pytest

import hipgisaxs_b200 as hg
from hipgisaxs_b200 import model
from hipgisaxs_b200.hig import read_hig
from test_gpu_hig_real import BOX, CYL, SPH, TEXT, params

pytestmark = pytest.mark.gpu
HIG = os.path.join(os.path.dirname(os.path.abspath(__file__)), "golden", "hig")
REPS = ["4.5 2.5 3.3", "6 3.25 1", "2.5 7 1.5", "0.5 0.75 1"]


@pytest.mark.parametrize("rep", REPS)
@pytest.mark.parametrize("turn", ["none", "flat", "tilted"])
@pytest.mark.parametrize("kind", ["hex", "hcp", "fcc"])
def test_structure_factor(ctx, po, rep, turn, kind):
    G = po.Grid(31, 17, -1.9, 0.0, 2.0, 3.0, 0.2, 10.0)
    g = hg.QGrid.from_arrays(ctx, G.qx, G.qy, G.qz_ext)
    assert g.mode == 1
    R = {"none": np.eye(3).ravel(), "flat": po.rot_axis(2, 0.4),
         "tilted": po.rot_mul(po.rot_axis(0, 0.3), po.rot_axis(2, 0.4))}[turn]
    abc, _ = model.lattice_vectors(kind)
    rep = [float(v) for v in rep.split()]
    ref = po.sf_lattice(G, abc, rep, [21.5] * 3, (3.0, -2.0, 5.0), R)
    for precision, tol in (("f64", 1e-11), ("f32c", 1e-5)):
        sf = model.sf_lattice(ctx, g, abc, rep, [21.5] * 3, (3.0, -2.0, 5.0), R, precision=precision)
        assert po.rel_err(sf, ref) < tol
        sf = model.sf_lattice(ctx, g, abc, rep, [21.5] * 3, (3.0, -2.0, 5.0), R, out_type="c64", precision=precision)
        assert po.rel_err(sf, ref) < max(tol, 1e-6)


def test_peak_of_order_zero(ctx, po):
    """Angles of zero, where the quotient takes the value N."""
    G = po.Grid(9, 5, -1.9, 0.0, 2.0, 3.0, 0.2, 10.0)
    zero = np.zeros(G.n)
    g = hg.QGrid.from_arrays(ctx, zero, zero, G.qz_ext)
    args = (np.eye(3), [2.5, 3.5, 1.0], [20.0] * 3)
    ref = po.sf_lattice_arrays(*args, [0, 0, 0], None, zero, zero, G.qz_ext)
    assert po.rel_err(model.sf_lattice(ctx, g, *args), ref) < 1e-11


@pytest.mark.parametrize("precision,tol", [("f64", 1e-11), ("f32c", 1e-5)])
@pytest.mark.parametrize("shape", [CYL, SPH, BOX], ids=["cylinder", "sphere", "box"])
@pytest.mark.parametrize("axis,grains,locs,lattice,rep,spacing", [
    ("z", 1, "[[0 0 0]]", "hex", "4.5 2.5 3.3", "0 0 0"),
    ("z", 9, "[[0 0 2.5] [3 2 1]]", "hcp", "6 3.25 1", "150 0 0"),
    ("x", 5, "[[0 0 0]]", "fcc", "4.5 2.5 3.3", "90 0 0"),   # qz in the rotated in-plane q
    ("x", 5, "[[1 0 3]]", "hex", "0.5 0.75 1", "0 0 0"),
    ("z", 9, "[[0 0 0]]", "hcp", "10 7 2", "0 0 0"),         # whole, in both precisions
    ("x", 5, "[[0 0 0]]", "hcp", "6 3 2", "90 0 0"),
])
def test_images(ctx, po, tmp_path, precision, tol, shape, axis, grains, locs, lattice, rep, spacing):
    text = TEXT
    for k, v in (("SHAPE", shape[0]), ("PARAMS", params(*shape[1], n=3)), ("LOCS", locs), ("LATTICE", lattice),
                 ("REP", rep), ("SPACING", spacing), ("GRAINS", str(grains)), ("AXIS", axis)):
        text = text.replace(k, v)
    path = tmp_path / "t.hig"
    path.write_text(text)
    d = read_hig(str(path))
    libc = ctypes.CDLL(None)
    libc.srand(11)
    img = d.compute_gisaxs(ctx, precision=precision)
    ref = []
    for factor in (1.0, 1.0 - 1e-15, 1.0 + 1e-15):
        hig = copy.deepcopy(d.data)
        for st in hig["structures"].values():
            st["scaling_mean"] = [v * factor for v in st["scaling_mean"]]
        libc.srand(11)
        ref.append(po.compute_gisaxs(hig, str(tmp_path)))
    spread = max(np.abs(r - ref[0]).max() for r in ref)
    assert np.abs(img - ref[0]).max() < tol * np.abs(ref[0]).max() + spread


def test_population(ctx, po, tmp_path):
    text = open(os.path.join(HIG, "fit_objective.hig")).read()
    path = tmp_path / "f.hig"
    path.write_text(text.replace("[ 6 6 1 ]", "[ 5.5 3.25 1 ]"))
    d = read_hig(str(path))
    X = np.array([[4.2, 23.0, 7.0], [5.1, 20.5, 14.0], [3.6, 26.0, 2.0]])
    ref_img = np.ones(d.image_size())
    want = []
    for x in X:
        d.fit_update(x)
        want.append(po.fit_distance("sqrt_unit_l2", ref_img, po.compute_gisaxs(d.data, HIG).ravel()))
    for precision, tol in (("f64", 1e-11), ("f32c", 1e-5)):
        pop = d.population(ctx, len(X), ref_img, None, "sqrt_unit_l2", 0.0, precision)
        got = pop.eval(X)
        pop.close()
        assert np.all(np.abs(got - np.ravel(want)) <= tol * np.abs(np.ravel(want)))
