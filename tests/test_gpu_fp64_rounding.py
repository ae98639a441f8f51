"""Rounding of the FP64 form factors on real qz (ff_analytic_real_kernel) against the same formulas in 80 bits:
norm-wise 1e-15, a few roundings of 1.1e-16 of phases, sines, quotients and sums, and next to q = 0 as well."""
import numpy as np
import pytest

import hipgisaxs_b200 as hg
from hipgisaxs_b200 import model

pytestmark = pytest.mark.gpu
L = np.longdouble
PI = L(3.141592653589793)


def sinc(x):
    return np.where(np.abs(x) > 1e-14, np.sin(x) / np.where(x == 0, L(1), x), L(1))


def sphere(x):
    z, term = x * x, L(1) / 3
    series = np.zeros_like(x)
    for k in range(14):  # (-1)^k x^2k (2k + 2) / (2k + 3)!
        series = series + term * (-z) ** k
        term = term * L(2 * k + 4) / (L(2 * k + 2) * (2 * k + 4) * (2 * k + 5))
    return np.where(x < 1, series, (np.sin(x) - x * np.cos(x)) / np.where(x == 0, L(1), x ** 3))


def expi(x):
    return np.cos(x) + 1j * np.sin(x)


@pytest.mark.parametrize("tilted", [False, True])
@pytest.mark.parametrize("n", [1, 7])
def test_box_and_sphere(ctx, po, tilted, n):
    G = po.Grid(120, 90, -1.9, 0.0, 2.0, 3.0, 0.2, 10.0)
    g = hg.QGrid.from_arrays(ctx, G.qx, G.qy, G.qz_ext)
    R = po.rot_mul(po.rot_axis(0, 0.3), po.rot_axis(2, 0.4)) if tilted else po.rot_axis(2, 0.4)
    R = np.asarray(R).reshape(3, 3)
    q = [np.tile(G.qx, 4).astype(L), np.tile(G.qy, 4).astype(L), G.qz_ext.real.astype(L)]
    m = [sum(L(R[j, k]) * q[k] for k in range(3)) for j in range(3)]

    def sizes(x):
        return x * (0.85 + 0.3 * np.arange(n) / n) if n > 1 else np.array([x])

    box = [sum(x * sinc(m[j] * x / 2) * (expi(m[j] * x / 2) if j == 2 else 1) for x in sizes(v).astype(L))
           for j, v in enumerate((8.0, 6.0, 10.0))]
    r = np.sqrt(m[0] ** 2 + m[1] ** 2 + m[2] ** 2)
    ball = sum(4 * PI * x ** 3 * sphere(r * x) * expi(m[2] * x) for x in sizes(6.0).astype(L))
    for shape, dims, ref in (("box", (8.0, 6.0, 10.0), box[0] * box[1] * box[2]), ("sphere", (6.0,), ball)):
        f = model.ff_analytic(ctx, g, shape, [(sizes(v), None) for v in dims], rot=R)
        e, a = np.abs(f - ref), np.abs(ref)
        assert np.sqrt((e ** 2).sum() / (a ** 2).sum()) < 1e-15
