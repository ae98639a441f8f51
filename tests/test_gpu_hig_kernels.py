"""Both sides of the choices between the kernels for real qz (grain_real_plan of a HiG simulation, and the
analytic form factor's thread per pixel or per q-point), against the oracle: 1e-11 in FP64 and 1e-5 in FP32C
of the largest value.  The reference's sphere, (sin x - x cos x) / x^3, loses 3 eps / x^2 of its value next to
q = 0 (twice that in an intensity), which is allowed on top.  Next to a lattice peak its quotient of differences
of exponentials loses eps / (angle to the peak): 1.0e-11 of an fcc image's largest value at a pixel 5.5e-9 turn
off one (against 80 bits), so images of moved elements are also allowed the oracle's own change under 1e-15 of
the scaling."""
import copy
import ctypes

import numpy as np
import pytest

import hipgisaxs_b200 as hg
from hipgisaxs_b200 import model
from hipgisaxs_b200.hig import read_hig
from test_gpu_hig_real import BOX, CYL, SPH, TEXT, params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [CYL, SPH, BOX], ids=["cylinder", "sphere", "box"])
@pytest.mark.parametrize("size,axis,grains,n", [
    ((210, 200), "z", 1, 1), ((210, 200), "z", 1, 4), ((210, 200), "x", 1, 1), ((210, 200), "x", 2, 4),
    ((31, 17), "z", 2, 4), ((31, 17), "z", 3, 4), ((31, 17), "x", 17, 1), ((31, 17), "x", 17, 4), ((31, 17), "x", 2, 4),
])
def test_images(ctx, po, tmp_path, shape, size, axis, grains, n):
    text = TEXT.replace("[ 37 23 ]", "[ %d %d ]" % size)
    for k, v in (("SHAPE", shape[0]), ("PARAMS", params(*shape[1], n=n)), ("LOCS", "[[0 0 0]]"), ("LATTICE", "hex"),
                 ("REP", "10 7 2"), ("SPACING", "0 0 0"), ("GRAINS", str(grains)), ("AXIS", axis)):
        text = text.replace(k, v)
    path = tmp_path / "t.hig"
    path.write_text(text)
    d = read_hig(str(path))
    libc = ctypes.CDLL(None)
    libc.srand(5)
    ref = po.compute_gisaxs(d.data, str(tmp_path))
    lost = 0.0
    if shape is SPH:
        G = po.Grid(*size, -1.0, 0.0, 1.2, 1.5, 0.2, 10.0)
        x = 0.85 * 6 * np.sqrt(np.tile(G.qx ** 2 + G.qy ** 2, 4) + G.qz_ext.real ** 2)
        lost = 2 * 3 * 2.2e-16 / x[x > 0].min() ** 2
    for precision, tol in (("f64", 1e-11 + lost), ("f32c", 1e-5)):
        libc.srand(5)
        img = d.compute_gisaxs(ctx, precision=precision)
        assert np.abs(img - ref).max() < tol * np.abs(ref).max()


@pytest.mark.parametrize("shape", [CYL, SPH, BOX], ids=["cylinder", "sphere", "box"])
@pytest.mark.parametrize("size,grains,n,locs,lattice", [
    ((31, 17), 7, 1, "[[0 0 0] [3 2 1]]", "hex"), ((31, 17), 8, 1, "[[0 0 0] [3 2 1]]", "hex"),
    ((31, 17), 8, 8, "[[3 2 1]]", "hex"), ((210, 200), 1, 8, "[[0 0 0] [3 2 1]]", "hex"),
    ((210, 200), 1, 8, "[[3 2 1]]", "fcc"), ((210, 200), 2, 3, "[[3 2 1] [1 5 0]]", "fcc"),
    ((210, 200), 2, 7, "[[3 2 1]]", "hcp"), ((210, 200), 2, 8, "[[0 0 0]]", "fcc"),
])
def test_images_of_moved_elements(ctx, po, tmp_path, shape, size, grains, n, locs, lattice):
    text = TEXT.replace("[ 37 23 ]", "[ %d %d ]" % size)
    for k, v in (("SHAPE", shape[0]), ("PARAMS", params(*shape[1], n=n)), ("LOCS", locs), ("LATTICE", lattice),
                 ("REP", "4 5 2"), ("SPACING", "150 0 0"), ("GRAINS", str(grains)), ("AXIS", "z")):
        text = text.replace(k, v)
    path = tmp_path / "t.hig"
    path.write_text(text)
    d = read_hig(str(path))
    libc = ctypes.CDLL(None)
    refs = []
    for factor in (1.0, 1.0 - 1e-15, 1.0 + 1e-15):
        hig = copy.deepcopy(d.data)
        for st in hig["structures"].values():
            st["scaling_mean"] = [v * factor for v in st["scaling_mean"]]
        libc.srand(7)
        refs.append(po.compute_gisaxs(hig, str(tmp_path)))
    ref = refs[0]
    spread = max(np.abs(r - ref).max() for r in refs)
    lost = 0.0
    if shape is SPH:
        G = po.Grid(*size, -1.0, 0.0, 1.2, 1.5, 0.2, 10.0)
        x = 0.85 * 6 * np.sqrt(np.tile(G.qx ** 2 + G.qy ** 2, 4) + G.qz_ext.real ** 2)
        lost = 2 * 3 * 2.2e-16 / x[x > 0].min() ** 2
    for precision, tol in (("f64", 1e-11 + lost), ("f32c", 1e-5)):
        libc.srand(7)
        img = d.compute_gisaxs(ctx, precision=precision)
        assert np.abs(img - ref).max() < tol * np.abs(ref).max() + spread


@pytest.mark.parametrize("shape", [CYL, SPH, BOX], ids=["cylinder", "sphere", "box"])
@pytest.mark.parametrize("size", [(31, 17), (200, 151)])
@pytest.mark.parametrize("n", [1, 4])
@pytest.mark.parametrize("tilted", [False, True])
def test_form_factors(ctx, po, shape, size, n, tilted):
    G = po.Grid(*size, -1.9, 0.0, 2.0, 3.0, 0.2, 10.0)
    g = hg.QGrid.from_arrays(ctx, G.qx, G.qy, G.qz_ext)
    P = [dict(type=k, min=0.85 * v, max=1.15 * v, mean=v, deviation=0.05 * v, nvalues=n, stat="gaussian") if n > 1
         else dict(type=k, min=v, max=v, nvalues=1) for k, v in shape[1]]
    R = po.rot_mul(po.rot_axis(0, 0.3), po.rot_axis(2, 0.4)) if tilted else po.rot_axis(2, 0.4)
    ref = po.ff_analytic(G, shape[0], P, transvec=(1.0, 2.0, -3.0), rot=R)
    for precision, tol in (("f64", 1e-11), ("f32c", 1e-5)):
        for out_type in ("c128", "c64"):
            f = model.ff_analytic_params(ctx, g, shape[0], P, transvec=(1.0, 2.0, -3.0), rot=R, out_type=out_type,
                                         precision=precision)
            assert po.rel_err(f, ref) < max(tol, 1e-6 if out_type == "c64" else 0.0)
