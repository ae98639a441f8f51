"""Rounding of the FP32C lattice structure factor on real qz (sf_lattice_real_kernel<float>) against 80-bit
values: norm-wise 1.35e-7, the error of a product of three quotients whose sines, quotients and products are each
rounded about once (six sines of 3e-8 rms each relative, three quotients and two products of 2.9e-8, the phase's
sine and cosine and its product 5e-8: 1.3e-7)."""
import numpy as np
import pytest

import hipgisaxs_b200 as hg
from hipgisaxs_b200 import model

pytestmark = pytest.mark.gpu
L = np.longdouble
TURN = 2 * L("3.14159265358979323846264338327950288")


def factor(theta, n):
    t = theta - TURN * np.rint(theta / TURN)
    s = np.sin(t / 2)
    return np.where(np.abs(s) < 1e-15, L(n), np.sin(n * t / 2) / np.where(s == 0, L(1), s))


@pytest.mark.parametrize("rep", [(20, 7, 3), (100, 10, 2), (5, 4, 1)])
@pytest.mark.parametrize("tilted", [False, True])
def test_against_80_bits(ctx, po, rep, tilted):
    G = po.Grid(200, 90, -1.9, 0.0, 2.0, 3.0, 0.2, 10.0)
    g = hg.QGrid.from_arrays(ctx, G.qx, G.qy, G.qz_ext)
    R = po.rot_mul(po.rot_axis(0, 0.3), po.rot_axis(2, 0.4)) if tilted else po.rot_axis(2, 0.4)
    abc, _ = model.lattice_vectors("hex")
    v = (np.asarray(abc) * 21.5).astype(L)
    R3 = np.asarray(R).reshape(3, 3).astype(L)
    q = [np.tile(G.qx, 4).astype(L), np.tile(G.qy, 4).astype(L), G.qz_ext.real.astype(L)]
    m = [sum(R3[j, k] * q[k] for k in range(3)) for j in range(3)]
    ph = 3 * m[0] - 2 * m[1] + 5 * m[2]
    ref = (factor(sum(v[0, j] * m[j] for j in range(3)), rep[0]) *
           factor(v[1, 0] * m[0] + v[1, 1] * m[1] + v[1, 2] ** 2, rep[1]) *
           factor(sum(v[2, j] * m[j] for j in range(3)), rep[2]) * (np.cos(ph) + 1j * np.sin(ph)))
    sf = model.sf_lattice(ctx, g, abc, rep, (21.5,) * 3, (3.0, -2.0, 5.0), R, precision="f32c")
    e, a = np.abs(sf - ref), np.abs(ref)
    assert np.sqrt((e ** 2).sum() / (a ** 2).sum()) < 1.35e-7
