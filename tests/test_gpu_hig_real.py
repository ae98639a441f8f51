"""The FP64 grain kernel for real qz (grain_dwba_real_kernel) against the oracle: 1e-11 of the
image's largest value, the bound of the step-by-step FP64 path."""
import ctypes

import numpy as np
import pytest

from hipgisaxs_b200.hig import read_hig

pytestmark = pytest.mark.gpu

TEXT = """hipGisaxsInput = {
	shape = { key = "s", name = "SHAPE", refindex = { delta = 8.5E-06, beta = 3.1E-07 }, PARAMS },
	unitcell = { key = "u1", element = { shape:key = "s", locations = LOCS } },
	layer = { key = "substr", order = -1, refindex = { delta = 9.1E-06, beta = 2.5E-07 } },
	structure = { key = "st1",
		grain = { unitcell:key = "u1", lattice = { type = "LATTICE" }, repetition = [REP], scaling = 21.5 },
		ensemble = { spacing = [SPACING], maxgrains = [GRAINS 1 1],
			orientations = { stat = "range", rot1 = { axis = "AXIS", angles = [0 50] } } } },
	instrumentation = { scattering = { alphai = { min = 0.2 }, photon = { value = 10000, unit = "ev" } },
		detector = { pixelsize = 0.172, sdd = 4000, directbeam = [ 0 0 ] } },
	computation = { runname = "t", outputregion = { type = "qspace", minpoint = [ -1 0 ], maxpoint = [ 1.2 1.5 ] },
		resolution = [ 37 23 ] }
}
"""


def params(*kinds, n=1):
    rows = []
    for kind, v in kinds:
        if n == 1:
            rows.append(f'param = {{ type = "{kind}", min = {v} }}')
        else:
            rows.append(f'param = {{ type = "{kind}", stat = "gaussian", min = {0.85 * v}, max = {1.15 * v}, '
                        f'p1 = {v}, p2 = {0.05 * v}, nvalues = {n} }}')
    return ", ".join(rows)


CYL = ("cylinder", (("radius", 5), ("height", 30)))
SPH = ("sphere", (("radius", 6),))
BOX = ("box", (("xsize", 8), ("ysize", 6), ("height", 10)))


@pytest.mark.parametrize("shape", [CYL, SPH, BOX], ids=["cylinder", "sphere", "box"])
@pytest.mark.parametrize("axis,grains,n,locs,lattice,rep,spacing", [
    ("z", 1, 1, "[[0 0 0]]", "hex", "1 1 1", "0 0 0"),
    ("z", 1, 11, "[[0 0 0]]", "hex", "20 20 1", "0 0 0"),
    ("z", 9, 2, "[[0 0 0]]", "hcp", "10 7 2", "0 0 0"),           # form factors kept over grains
    ("z", 9, 3, "[[0 0 2.5] [3 2 1]]", "fcc", "4 5 6", "150 0 0"),  # offsets, centres, a with z
    ("x", 5, 4, "[[0 0 0] [1 0 3]]", "hcp", "6 3 2", "90 0 0"),   # qz in the rotated in-plane q
])
def test_matches_oracle(ctx, po, tmp_path, shape, axis, grains, n, locs, lattice, rep, spacing):
    text = TEXT
    for k, v in (("SHAPE", shape[0]), ("PARAMS", params(*shape[1], n=n)), ("LOCS", locs), ("LATTICE", lattice),
                 ("REP", rep), ("SPACING", spacing), ("GRAINS", str(grains)), ("AXIS", axis)):
        text = text.replace(k, v)
    path = tmp_path / "t.hig"
    path.write_text(text)
    d = read_hig(str(path))
    libc = ctypes.CDLL(None)
    libc.srand(11)
    img = d.compute_gisaxs(ctx)
    libc.srand(11)
    ref = po.compute_gisaxs(d.data, str(tmp_path))
    assert np.abs(img - ref).max() / np.abs(ref).max() < 1e-11
