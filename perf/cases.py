"""Performance cases of the GISAXS library: the calls that a program built on it makes, over the
sizes it makes them at.

A case is a dict; its "kind" names the call, the other entries its sizes and options:

  mesh      form factor of a triangle mesh on a detector grid, device arrays (ff_triangles)
  call      the reference-shaped form-factor call, host arrays in and out (ff_triangles_arrays)
  gradient  chi^2 and vertex gradient of a mesh model (fitting.mesh_chi2_grad)
  batch     chi^2 and gradient of a batch of cylinder-lattice candidates (fitting.CylinderBatch)
  hig       a whole simulation of a HiG description (HiGInput.compute_gisaxs)
  steps     analytic form factor, structure factor, Fresnel coefficients and DWBA sum one by one

Results of the FP32C precision carry single-precision accuracy and are kept in single precision
here (complex64 form factors, float32 images and gradients), as a program that asks for FP32C
stores them; FP64 results stay in double precision.
"""
from __future__ import annotations

import ctypes
import math
import os
import tempfile

import numpy as np
import torch

import hipgisaxs_b200 as hg
from hipgisaxs_b200 import fitting, model
from hipgisaxs_b200.core import ff_triangles, ff_triangles_arrays
from hipgisaxs_b200.hig import read_hig

DEV = "cuda"
PI = 3.141592653589793
ALPHA_I = 0.20 * PI / 180
K0 = 2 * PI / (1.23984 / 10.0)  # 10 keV
# a region off the beam's centre: no pixel falls on q = 0, where the mesh form factor divides by zero
QMIN_Y, QMIN_Z, QMAX_Y, QMAX_Z = -1.937, 0.0, 2.0, 3.0
SUBSTRATE = (4.88e-6, 7.37e-8)  # Si-like delta, beta
DN2 = (-2 * SUBSTRATE[0], -2 * SUBSTRATE[1])
HEX = ((1.0, 0.0, 0.0), (0.5, 0.8660254, 0.0), (0.0, 0.0, 1.0))
HCP = ((1.0, 0.0, 0.0), (0.5, 0.866, 0.0), (0.5, 0.2887, 0.8165))
MAX_EVALS = 2048 * 2048 * 50000  # pixel-triangle products of the largest listed case


def listed():
    return [
        # a quick look at a small particle: launch and preparation latency
        dict(name="mesh_small", kind="mesh", ncol=128, nrow=96, nlon=32, nbands=21, prec="f32c",
             dn2=False, rot=False),
        # a cropped, odd-sized detector region and a turned particle
        dict(name="mesh_ragged", kind="mesh", ncol=601, nrow=301, nlon=123, nbands=51, prec="f32c",
             dn2=False, rot=True),
        # the headline workload: a 50,000-triangle mesh on a full detector
        dict(name="mesh_2048", kind="mesh", ncol=2048, nrow=2048, nlon=250, nbands=101, prec="f32c",
             dn2=False, rot=False),
        # particles inside an absorbing layer: complex qz
        dict(name="mesh_absorbing", kind="mesh", ncol=700, nrow=500, nlon=50, nbands=51, prec="f32c",
             dn2=True, rot=False),
        # the library's default precision, device arrays
        dict(name="mesh_f64", kind="mesh", ncol=1024, nrow=512, nlon=125, nbands=81, prec="f64",
             dn2=False, rot=True),
        # a caller of the reference's interface: host arrays, default precision
        dict(name="call_f64", kind="call", ncol=256, nrow=192, nlon=32, nbands=21),
        # one step of a shape fit
        dict(name="gradient", kind="gradient", ncol=512, nrow=512, nlon=125, nbands=81),
        # one generation of a lattice fit with regions of interest
        dict(name="batch", kind="batch", n=1024, ncand=48, roi_min=96, roi_max=640),
        # one grain of size-distributed cylinders, default precision, image left on the device
        dict(name="hig_grain_f64", kind="hig", n_y=1024, n_z=1024, grains=1, lattice="hex",
             samples=11, prec="f64"),
        # an ensemble of turned grains
        dict(name="hig_ensemble_f64", kind="hig", n_y=600, n_z=300, grains=25, lattice="hcp",
             samples=1, prec="f64"),
        dict(name="hig_ensemble_f32c", kind="hig", n_y=513, n_z=257, grains=18, lattice="hcp",
             samples=1, prec="f32c"),
        # a program that composes the model from its parts
        dict(name="steps", kind="steps", ncol=640, nrow=481, shape="box", samples=5),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _tri(case):
    return 2 * case["nlon"] * (case["nbands"] - 1)


def draw(rng):
    kind = rng.choice(["mesh", "mesh", "mesh", "mesh", "call", "gradient", "batch", "hig", "hig", "steps"])
    if kind == "mesh":
        prec = rng.choice(["f32c", "f32c", "f64"])
        most = MAX_EVALS if prec == "f32c" else 1024 * 1024 * 20000
        while True:
            c = dict(kind=kind, ncol=_log(rng, 64, 2048), nrow=_log(rng, 48, 2048), nlon=_log(rng, 16, 250),
                     nbands=_log(rng, 11, 101), prec=prec, dn2=rng.random() < 0.25, rot=rng.random() < 0.5)
            if c["ncol"] * c["nrow"] * _tri(c) <= most:
                return c
    if kind == "call":
        return dict(kind=kind, ncol=_log(rng, 64, 400), nrow=_log(rng, 48, 300), nlon=_log(rng, 16, 60),
                    nbands=_log(rng, 11, 41))
    if kind == "gradient":
        return dict(kind=kind, ncol=_log(rng, 96, 700), nrow=_log(rng, 64, 600), nlon=_log(rng, 20, 125),
                    nbands=_log(rng, 15, 81))
    if kind == "batch":
        lo = _log(rng, 64, 256)
        return dict(kind=kind, n=rng.choice([512, 768, 1024]), ncand=_log(rng, 1, 96), roi_min=lo,
                    roi_max=min(500, lo + _log(rng, 1, 300)))
    if kind == "hig":
        if rng.random() < 0.4:
            return dict(kind=kind, n_y=_log(rng, 128, 1024), n_z=_log(rng, 96, 1024), grains=1, lattice="hex",
                        samples=rng.randint(1, 15), prec=rng.choice(["f64", "f32c"]))
        return dict(kind=kind, n_y=_log(rng, 100, 600), n_z=_log(rng, 80, 300), grains=rng.randint(2, 25),
                    lattice=rng.choice(["hex", "hcp"]), samples=1, prec=rng.choice(["f64", "f32c"]))
    return dict(kind=kind, ncol=_log(rng, 100, 1200), nrow=_log(rng, 80, 900),
                shape=rng.choice(["box", "cylinder", "sphere"]), samples=rng.randint(1, 11))


# ------------------------------------------------------------------- inputs ----
def _ctx():
    """The program's context, on torch's stream, made on first use."""
    global _CTX
    try:
        return _CTX
    except NameError:
        _CTX = hg.Context(torch.cuda.current_device(), torch.cuda.current_stream())
        return _CTX


def _star(seed, nlon, nbands, radius=15.0):
    """A closed UV-sphere mesh (2 nlon (nbands - 1) faces) whose radius is perturbed by a few
    plane waves of the direction, as (vertices, faces) on the GPU."""
    rng = np.random.default_rng(seed)
    k = torch.tensor(rng.normal(scale=2.5, size=(6, 3)), device=DEV)
    ph = torch.tensor(rng.uniform(0, 2 * PI, 6), device=DEV)
    amp = torch.tensor(rng.normal(scale=0.03, size=6), device=DEV)
    rings = nbands - 1
    th = PI * torch.arange(1, rings + 1, dtype=torch.float64, device=DEV) / nbands
    la = 2 * PI * torch.arange(nlon, dtype=torch.float64, device=DEV) / nlon
    T, L = torch.meshgrid(th, la, indexing="ij")
    T, L = T.reshape(-1), L.reshape(-1)
    u = torch.stack([torch.sin(T) * torch.cos(L), torch.sin(T) * torch.sin(L), torch.cos(T)], 1)
    pole = torch.tensor([[0.0, 0.0, 1.0], [0.0, 0.0, -1.0]], dtype=torch.float64, device=DEV)
    u = torch.cat([pole[:1], u, pole[1:]])
    V = u * (radius * (1 + (amp * torch.sin(u @ k.T + ph)).sum(1)))[:, None]
    j = torch.arange(nlon, device=DEV)
    jn = (j + 1) % nlon
    bot = len(V) - 1
    F = [torch.stack([torch.zeros_like(j), 1 + j, 1 + jn], 1)]
    i = torch.arange(rings - 1, device=DEV)[:, None] * nlon + 1
    a, b, c, d = i + j, i + jn, i + nlon + j, i + nlon + jn
    F += [torch.stack([a, c, b], 2).reshape(-1, 3), torch.stack([b, c, d], 2).reshape(-1, 3)]
    last = 1 + (rings - 1) * nlon
    F.append(torch.stack([torch.full_like(j, bot), last + jn, last + j], 1))
    return V, torch.cat(F).to(torch.int32)


def _normals_centroids(V, F):
    v = V[F.long()]
    return torch.linalg.cross(v[:, 1] - v[:, 0], v[:, 2] - v[:, 0]) / 2, v.mean(1)


def _shape_def(V, F):
    """(T, 8) rows (area, unit normal, centroid, 0): the triangle tuples of the form factor."""
    n, c = _normals_centroids(V, F)
    s = n.norm(dim=1, keepdim=True)
    return torch.cat([s, n / s, c, torch.zeros_like(s)], 1).contiguous()


def _rotation(case, seed):
    if not case.get("rot"):
        return None
    a, b = np.random.default_rng(seed + 7).uniform(0.1, 1.2, 2)
    rz = np.array([[math.cos(a), -math.sin(a), 0], [math.sin(a), math.cos(a), 0], [0, 0, 1.0]])
    rx = np.array([[1.0, 0, 0], [0, math.cos(b), -math.sin(b)], [0, math.sin(b), math.cos(b)]])
    return rz @ rx


def _detector(ncol, nrow, k0=K0, alpha_i=ALPHA_I, lo=(QMIN_Y, QMIN_Z), hi=(QMAX_Y, QMAX_Z), dn2=0.0):
    """The reference's detector grid in 64 bits: qx, qy (nrow, ncol), the four complex qz of each
    row (nrow, 4) and the exit angle of each row."""
    f = torch.float64
    r = torch.arange(nrow, dtype=f, device=DEV)
    al = torch.asin((lo[1] + r * ((hi[1] - lo[1]) / (nrow - 1))) / k0 - math.sin(alpha_i))
    q = lo[0] + torch.arange(ncol, dtype=f, device=DEV) * ((hi[0] - lo[0]) / (ncol - 1))
    ci, cf = math.cos(alpha_i), math.cos(float(al[0]))
    t = ((cf * cf + ci * ci - (q / k0) ** 2) / (2 * cf * ci)).clamp(max=1.0)
    tth = torch.where(q < 0, -1.0, 1.0) * torch.acos(t)
    al = al.flip(0)
    qx = k0 * (torch.cos(al)[:, None] * torch.cos(tth) - ci)
    qy = k0 * (torch.cos(al)[:, None] * torch.sin(tth))
    qz = k0 * (torch.sin(al) + math.sin(alpha_i))
    d = torch.tensor(complex(dn2), dtype=torch.complex128, device=DEV)
    kzi = -k0 * torch.sqrt(math.sin(alpha_i) ** 2 - d)
    kf0 = qz - k0 * math.sin(alpha_i)
    kzf = torch.sqrt(kf0 * kf0 - k0 * k0 * d) * torch.where(kf0 < 0, -1.0, 1.0)
    return qx, qy, torch.stack([kzf - kzi, -kzf - kzi, kzf + kzi, -kzf + kzi], 1), al


def _layer_dn2(case):
    # an absorbing organic layer around the particles
    return complex(2 * 3.0e-6, 2 * 4.0e-8) if case.get("dn2") else 0.0


def _fresnel(al, k0, alpha_i, delta, beta):
    """Per-row coefficients (nrow, 4) of a vacuum layer over one substrate."""
    def amplitude(a):
        s = torch.sin(a).to(torch.complex128)
        k1, k2 = -k0 * torch.sqrt(s * s), -k0 * torch.sqrt(s * s - complex(2 * delta, 2 * beta))
        return (k1 - k2) / (k1 + k2)
    ri = amplitude(torch.tensor([alpha_i], dtype=torch.float64, device=DEV))
    up = al > 0
    rf = torch.where(up, amplitude(torch.where(up, al, torch.ones_like(al))), 0)
    tf = up.to(torch.complex128)
    return torch.stack([tf, rf.conj(), ri * tf, ri * rf.conj()], 1)


def _row_sums(qx, qy, qz, n, c):
    """sum_t (q . n_t) e^{i q . c_t} of one detector row: qx, qy (P), qz (K) complex, n, c (T, 3)."""
    E = torch.exp(1j * (qx[:, None] * c[:, 0] + qy[:, None] * c[:, 1]))
    Z = torch.exp(1j * (c[:, 2:3] * qz))
    B = torch.stack([n[:, j:j + 1] * Z for j in range(3)], 2).reshape(len(c), -1)
    M = (E @ B).reshape(len(qx), len(qz), 3)
    return qx[:, None] * M[:, :, 0] + qy[:, None] * M[:, :, 1] + qz * M[:, :, 2]


def _row_ff(qx, qy, qz, n, c):
    q2 = (qx * qx + qy * qy)[:, None] + (qz.real ** 2 + qz.imag ** 2)
    return -1j * _row_sums(qx, qy, qz, n, c) / q2


def _mesh_intensity(D, rowfc, n, c):
    qx, qy, qz, _ = D
    k = complex(*DN2)
    return torch.stack([(_row_ff(qx[r], qy[r], qz[r], n, c) * (rowfc[r] * k)).sum(1).abs() ** 2
                        for r in range(len(qz))])


def _poisson(rate, seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return torch.poisson(rate, generator=g)


def _target(case, seed):
    """(counts, scale): Poisson counts of a coarse mesh near the fitted one, peak 1e4."""
    D = _detector(case["ncol"], case["nrow"])
    rowfc = _fresnel(D[3], K0, ALPHA_I, *SUBSTRATE)
    n, c = _normals_centroids(*_star(seed + 1, 30, 25, 15.3))
    I = _mesh_intensity(D, rowfc, n, c)
    scale = float(1e4 / I.max())
    return _poisson(scale * I, seed), scale


# ------------------------------------------------------- cylinders on a lattice ----
class _J1(torch.autograd.Function):
    """J1 with its derivative J0 - J1 / x."""

    @staticmethod
    def forward(ctx, x):
        y = torch.special.bessel_j1(x)
        ctx.save_for_backward(x, y)
        return y

    @staticmethod
    def backward(ctx, g):
        x, y = ctx.saved_tensors
        s = torch.where(x == 0, torch.ones_like(x), x)
        return g * (torch.special.bessel_j0(x) - torch.where(x == 0, torch.full_like(x, 0.5), y / s))


def _dirichlet(theta, n):
    """The lattice sum of n cells, sin(n theta / 2) / sin(theta / 2) of the wrapped angle."""
    t = theta - 2 * PI * torch.round(theta.detach() / (2 * PI))
    if n == 1:
        return torch.ones_like(t)
    small = t.detach().abs() < 1e-7
    u = torch.where(small, torch.ones_like(t), t)
    return torch.where(small, torch.full_like(t, float(n)), torch.sin(n * u / 2) / torch.sin(u / 2))


def _radial(qpar, radii):
    out = 0
    for r in radii:
        x = qpar * r
        ok = x.detach() ** 2 > 1e-13
        s = torch.where(ok, x, torch.ones_like(x))
        out = out + torch.where(ok, _J1.apply(s) / s, torch.zeros_like(x)) * (2 * PI * r * r)
    return out


def _heights(qz, heights):
    out = 0
    for h in heights:
        x = qz * h / 2
        ok = x.detach().abs() > 1e-14
        s = torch.where(ok, x, torch.ones_like(x))
        out = out + torch.where(ok, torch.sin(s) / s, torch.ones_like(x)) * h * torch.exp(1j * x)
    return out


def _spread(v, samples, spread=0.05):
    if samples < 2:
        return [v]
    return [v * (1 - 3 * spread + 6 * spread * i / (samples - 1)) for i in range(samples)]


def _batch_setup(case, seed):
    rng = np.random.default_rng(seed)
    n, nc = case["n"], case["ncand"]
    h = rng.integers(case["roi_min"], case["roi_max"] + 1, nc)
    w = rng.integers(case["roi_min"], case["roi_max"] + 1, nc)
    rois = [(int(rng.integers(0, n - a + 1)), int(rng.integers(0, n - b + 1)), int(a), int(b))
            for a, b in zip(h, w)]
    f = 1 + rng.uniform(-0.1, 0.1, (nc, 3))
    theta = [(5 * f[i, 0], 10 * f[i, 1], 20 * f[i, 2], math.radians(rng.uniform(-10, 10))) for i in range(nc)]
    return rois, theta


def _batch_image(D, rowfc, theta, roi):
    """The intensity of one candidate on its region (differentiable in theta)."""
    R, H, a, phi = theta
    r0, c0, h, w = roi
    qx, qy = D[0][r0:r0 + h, c0:c0 + w], D[1][r0:r0 + h, c0:c0 + w]
    mx, my = torch.cos(phi) * qx - torch.sin(phi) * qy, torch.sin(phi) * qx + torch.cos(phi) * qy
    sa = _dirichlet(a * (HEX[0][0] * mx + HEX[0][1] * my), 20)
    sb = _dirichlet(a * (HEX[1][0] * mx + HEX[1][1] * my), 20)
    fr = _radial(torch.sqrt(qx * qx + qy * qy), _spread(R, 11))
    Q = (rowfc[r0:r0 + h] * _heights(D[2][r0:r0 + h].real, _spread(H, 11))).sum(1)
    q2 = (Q.real ** 2 + Q.imag ** 2) * abs(complex(*DN2)) ** 2
    return q2[:, None] * (fr * sa * sb) ** 2


def _batch_target(case, seed):
    """(counts image, scale): Poisson counts of a lattice near the candidates, peak 1e4."""
    D = _detector(case["n"], case["n"])
    rowfc = _fresnel(D[3], K0, ALPHA_I, *SUBSTRATE)
    truth = [torch.tensor(v, dtype=torch.float64, device=DEV) for v in (5.15, 9.6, 20.4, math.radians(5))]
    I = _batch_image(D, rowfc, truth, (0, 0, case["n"], case["n"]))
    scale = float(1e4 / I.max())
    return D, rowfc, _poisson(scale * I, seed), scale


# ----------------------------------------------------------- HiG descriptions ----
HIG = """hipGisaxsInput = {
	shape = { key = "cyl", name = "cylinder", refindex = { delta = 8.5E-06, beta = 3.1E-07 },
		param = { type = "radius", stat = "%(stat)s", min = %(r0).15g, max = %(r1).15g, p1 = %(r).15g, p2 = %(rs).15g, nvalues = %(nv)d },
		param = { type = "height", stat = "%(stat)s", min = %(h0).15g, max = %(h1).15g, p1 = %(h).15g, p2 = %(hs).15g, nvalues = %(nv)d } },
	unitcell = { key = "u1", element = { shape:key = "cyl", locations = [[0 0 0]] } },
	layer = { key = "substr", order = -1, refindex = { delta = 9.1E-06, beta = 2.5E-07 } },
	structure = { key = "st1",
		grain = { unitcell:key = "u1", lattice = { type = "%(lattice)s" }, repetition = [%(rep)s], scaling = %(scaling).15g },
		ensemble = { maxgrains = [%(grains)d %(grains)d 1],
			orientations = { stat = "range", rot1 = { axis = "z", angles = [0 180] } } } },
	instrumentation = { scattering = { alphai = { min = 0.2 }, photon = { value = 10000, unit = "ev" } },
		detector = { pixelsize = 0.172, sdd = 4000, directbeam = [ 0 0 ] } },
	computation = { runname = "case", outputregion = { type = "qspace", minpoint = [ -1 0 ], maxpoint = [ 1 1 ] },
		resolution = [ %(n_y)d %(n_z)d ] }
}
"""


def _hig_values(case, seed):
    rng = np.random.default_rng(seed)
    long = case["lattice"] == "hcp"
    r, h = 5 * rng.uniform(0.9, 1.1), (150 if long else 10) * rng.uniform(0.9, 1.1)
    s = case["samples"]
    w = 0.15 if s > 1 else 0.0
    return dict(stat="gaussian" if s > 1 else "none", r=r, rs=0.05 * r, r0=r * (1 - w), r1=r * (1 + w), h=h,
                hs=0.05 * h, h0=h * (1 - w), h1=h * (1 + w), nv=s, lattice=case["lattice"],
                rep="100 10 2" if long else "20 20 1", scaling=(50 if long else 20) * rng.uniform(0.95, 1.05),
                grains=case["grains"], n_y=case["n_y"], n_z=case["n_z"])


def _stepped(lo, hi, n):
    """The reference's sample values of a distribution between lo and hi."""
    if n < 2:
        return [lo]
    step, v, out = abs(hi - lo) / (n - 1), lo, []
    while True:
        out.append(v)
        v += step
        if not v < hi:
            return out


def _printed(v):
    return float("%.15g" % v)  # the value as the description's text carries it


def _lattice_cylinders(D, rows, radii, heights, lattice, scaling, rep, m):
    """Form factor times structure factor of one turned grain on some rows: (rows, ncol, 4)."""
    qz = D[2][rows].real[:, None, :]
    q = [D[0][rows][:, :, None], D[1][rows][:, :, None], qz]
    mx = m[0][0] * q[0] + m[0][1] * q[1]
    my = m[1][0] * q[0] + m[1][1] * q[1]
    ff = _radial(torch.sqrt(mx * mx + my * my), radii) * _heights(qz, heights)
    va, vb, vc = ([scaling * x for x in v] for v in lattice)
    sf = _dirichlet(va[0] * mx + va[1] * my + va[2] * qz, rep[0])
    sf = sf * _dirichlet(vb[0] * mx + vb[1] * my + vb[2] * vb[2], rep[1])
    return ff * sf * _dirichlet(vc[0] * mx + vc[1] * my + vc[2] * qz, rep[2])


# ------------------------------------------------------------------ prepare ----
def prepare(case, seed):
    kind = case["kind"]
    if kind in ("mesh", "call"):
        sd = _shape_def(*_star(seed, case["nlon"], case["nbands"]))
    if kind == "mesh":
        d = complex(_layer_dn2(case))
        grid = hg.QGrid.create(_ctx(), case["ncol"], case["nrow"], QMIN_Y, QMIN_Z, QMAX_Y, QMAX_Z, ALPHA_I, K0,
                               (d.real, d.imag))
        c64 = case["prec"] == "f32c"
        out = torch.empty(4 * case["ncol"] * case["nrow"], dtype=torch.complex64 if c64 else torch.complex128,
                          device=DEV)
        return dict(case=case, grid=grid, sd=sd, rot=_rotation(case, seed), out=out,
                    out_type="c64" if c64 else "c128")
    if kind == "call":
        qx, qy, qz, _ = _detector(case["ncol"], case["nrow"])
        ext = qz.T[:, :, None].expand(4, case["nrow"], case["ncol"]).reshape(-1)
        return dict(case=case, sd=sd.cpu().numpy(), qx=qx.reshape(-1).cpu().numpy(),
                    qy=qy.reshape(-1).cpu().numpy(), qz=ext.cpu().numpy())
    if kind == "gradient":
        V, F = _star(seed, case["nlon"], case["nbands"])
        counts, scale = _target(case, seed)
        grid = hg.QGrid.create(_ctx(), case["ncol"], case["nrow"], QMIN_Y, QMIN_Z, QMAX_Y, QMAX_Z, ALPHA_I, K0)
        rowfc = model.propagation_coeffs(_ctx(), grid, [(*SUBSTRATE, 0.0, -1)], K0, ALPHA_I, 0, per_row=True)
        return dict(case=case, grid=grid, rowfc=rowfc, verts=V.cpu().numpy(), faces=F.cpu().numpy(),
                    counts=counts.reshape(-1).contiguous(), scale=scale)
    if kind == "batch":
        rois, theta = _batch_setup(case, seed)
        _, _, counts, scale = _batch_target(case, seed)
        n = case["n"]
        grid = hg.QGrid.create(_ctx(), n, n, QMIN_Y, QMIN_Z, QMAX_Y, QMAX_Z, ALPHA_I, K0)
        rowfc = model.propagation_coeffs(_ctx(), grid, [(*SUBSTRATE, 0.0, -1)], K0, ALPHA_I, 0, per_row=True)
        cat = torch.cat([counts[r:r + h, c:c + w].reshape(-1) for r, c, h, w in rois]).cpu().numpy()
        batch = fitting.CylinderBatch(_ctx(), grid, rowfc, np.array(HEX), rois, cat, None, scale, "f32c")
        models = np.array([fitting.model_block(*t, 0.05, 11, (20, 20, 1), DN2, smooth_sampling=True)
                           for t in theta])
        return dict(case=case, batch=batch, grid=grid, models=models)
    if kind == "hig":
        with tempfile.TemporaryDirectory() as tmp:
            path = os.path.join(tmp, "case.hig")
            with open(path, "w") as f:
                f.write(HIG % _hig_values(case, seed))
            d = read_hig(path)
        img = torch.empty(case["n_y"] * case["n_z"], dtype=torch.float64, device=DEV)
        return dict(case=case, hig=d, img=img, seed=seed)
    shape, params = _steps_shape(case, seed)
    grid = hg.QGrid.create(_ctx(), case["ncol"], case["nrow"], QMIN_Y, QMIN_Z, QMAX_Y, QMAX_Z, ALPHA_I, K0)
    n4 = 4 * case["ncol"] * case["nrow"]
    buf = [torch.empty(n4, dtype=torch.complex128, device=DEV) for _ in range(3)]
    return dict(case=case, grid=grid, params=params, shape=shape, ff=buf[0], sf=buf[1], fc=buf[2])


def _steps_shape(case, seed):
    rng = np.random.default_rng(seed)
    n = case["samples"]

    def dist(kind, v):
        if n < 2:
            return dict(type=kind, min=v, max=v, nvalues=1)
        return dict(type=kind, stat="gaussian", min=0.85 * v, max=1.15 * v, mean=v, deviation=0.05 * v, nvalues=n)

    f = rng.uniform(0.9, 1.1, 3)
    if case["shape"] == "box":
        return "box", [dist("xsize", 8 * f[0]), dist("ysize", 6 * f[1]), dist("height", 10 * f[2])]
    if case["shape"] == "cylinder":
        return "cylinder", [dist("radius", 5 * f[0]), dist("height", 10 * f[1])]
    return "sphere", [dist("radius", 6 * f[0])]


# ---------------------------------------------------------------------- run ----
_LIBC = ctypes.CDLL(None)


def run(state):
    case, kind = state["case"], state["case"]["kind"]
    if kind == "mesh":
        return ff_triangles(_ctx(), state["grid"], state["sd"], state["rot"], precision=case["prec"],
                            out=state["out"], out_type=state["out_type"])
    if kind == "call":
        return ff_triangles_arrays(_ctx(), state["sd"], state["qx"], state["qy"], state["qz"])
    if kind == "gradient":
        chi, g, _ = fitting.mesh_chi2_grad(_ctx(), state["grid"], state["verts"], state["faces"], state["rowfc"],
                                           DN2, state["counts"], None, state["scale"])
        return {"chi2": np.float32(chi), "grad": g.astype(np.float32)}
    if kind == "batch":
        chi, g = state["batch"].eval(state["models"])
        return {"chi2": chi.astype(np.float32), "grad": g.astype(np.float32)}
    if kind == "hig":
        _LIBC.srand(state["seed"])  # the orientations are drawn by the C library's rand()
        img = state["hig"].compute_gisaxs(_ctx(), precision=case["prec"], out=state["img"])
        return img.float() if case["prec"] == "f32c" else img
    ctx, grid = _ctx(), state["grid"]
    model.ff_analytic_params(ctx, grid, state["shape"], state["params"], out=state["ff"])
    model.sf_lattice(ctx, grid, HEX, (20, 20, 1), (20.0, 20.0, 20.0), out=state["sf"])
    model.propagation_coeffs(ctx, grid, [(*SUBSTRATE, 0.0, -1)], K0, ALPHA_I, 0, out=state["fc"])
    inten = torch.zeros(case["ncol"] * case["nrow"], dtype=torch.float64, device=DEV)
    model.dwba_combine(ctx, state["fc"], state["sf"], state["ff"], 1.0, inten)
    return {"intensity": inten, "ff": state["ff"]}


# -------------------------------------------------------------------- exact ----
def exact(case, seed):
    kind = case["kind"]
    if kind in ("mesh", "call"):
        n, c = _normals_centroids(*_star(seed, case["nlon"], case["nbands"]))
        rot = _rotation(case, seed)
        if rot is not None:  # R q . n = q . R^T n
            r = torch.tensor(rot, device=DEV)
            n, c = n @ r, c @ r
        qx, qy, qz, _ = _detector(case["ncol"], case["nrow"], dn2=_layer_dn2(case))
        out = torch.empty(4, case["nrow"], case["ncol"], dtype=torch.complex128, device=DEV)
        for r in range(case["nrow"]):
            out[:, r] = _row_ff(qx[r], qy[r], qz[r], n, c).T
        out = out.reshape(-1)
        return out.cpu().numpy() if kind == "call" else out
    if kind == "gradient":
        V, F = _star(seed, case["nlon"], case["nbands"])
        counts, scale = _target(case, seed)
        qx, qy, qz, al = _detector(case["ncol"], case["nrow"])
        fc = _fresnel(al, K0, ALPHA_I, *SUBSTRATE) * complex(*DN2)
        n, c = (t.detach().requires_grad_() for t in _normals_centroids(V, F))
        chi = 0.0
        for r in range(case["nrow"]):
            I = (_row_ff(qx[r], qy[r], qz[r], n, c) * fc[r]).sum(1).abs() ** 2
            x = ((scale * I - counts[r]) ** 2 / counts[r].clamp(min=1)).sum()
            x.backward()
            chi += float(x.detach())
        V.requires_grad_()
        n2, c2 = _normals_centroids(V, F)
        torch.autograd.backward([n2, c2], [n.grad, c.grad])
        return {"chi2": np.float64(chi), "grad": V.grad.cpu().numpy()}
    if kind == "batch":
        rois, theta = _batch_setup(case, seed)
        D, rowfc, counts, scale = _batch_target(case, seed)
        chis, grads = [], []
        for roi, t in zip(rois, theta):
            p = [torch.tensor(float(v), dtype=torch.float64, device=DEV, requires_grad=True) for v in t]
            I = _batch_image(D, rowfc, p, roi)
            r, c, h, w = roi
            C = counts[r:r + h, c:c + w]
            x = ((scale * I - C) ** 2 / C.clamp(min=1)).sum()
            x.backward()
            chis.append(float(x.detach()))
            grads.append([float(v.grad) for v in p])
        return {"chi2": np.array(chis), "grad": np.array(grads)}
    if kind == "hig":
        v = _hig_values(case, seed)
        D = _detector(case["n_y"], case["n_z"], lo=(-1.0, 0.0), hi=(1.0, 1.0))
        fc = _fresnel(D[3], K0, ALPHA_I, 9.1e-6, 2.5e-7)
        radii = _stepped(_printed(v["r0"]), _printed(v["r1"]), v["nv"])
        heights = _stepped(_printed(v["h0"]), _printed(v["h1"]), v["nv"])
        # a description's hexagonal cell has the exact angle, not the table's seven digits
        lattice = HCP if case["lattice"] == "hcp" else (HEX[0], (0.5, math.sqrt(3) / 2, 0.0), HEX[2])
        rep = [int(x) for x in v["rep"].split()]
        scaling = _printed(v["scaling"])
        _LIBC.srand(seed)
        angles = [(0 + (_LIBC.rand() / 2147483647) * 180) * PI / 180 for _ in range(case["grains"] ** 2)]
        k = abs(complex(-2 * 8.5e-6, -2 * 3.1e-7)) ** 2
        img = torch.zeros(case["n_z"], case["n_y"], dtype=torch.float64, device=DEV)
        for a in angles:
            m = ((math.cos(a), -math.sin(a)), (math.sin(a), math.cos(a)))
            A = (_lattice_cylinders(D, slice(None), radii, heights, lattice, scaling, rep, m) *
                 fc[:, None, :]).sum(2)
            img += (A.real ** 2 + A.imag ** 2) * k
        return img.reshape(-1)
    shape, params = _steps_shape(case, seed)
    qx, qy, qz, al = _detector(case["ncol"], case["nrow"])
    q = [qx[:, :, None], qy[:, :, None], qz.real[:, None, :]]
    dims = []
    for p in params:
        vals = _stepped(p["min"], p["max"], p["nvalues"])
        w = [1.0] * len(vals)
        if p.get("stat"):
            w = [math.exp(-(x - p["mean"]) ** 2 / (2 * p["deviation"] ** 2)) / (math.sqrt(2 * PI) * p["deviation"])
                 for x in vals]
        dims.append((vals, w))

    def sinc(x):
        return torch.where(x.abs() > 1e-14, torch.sin(x) / torch.where(x == 0, 1.0, x), 1.0)

    if shape == "cylinder":
        ff = _radial(torch.sqrt(q[0] ** 2 + q[1] ** 2), dims[0][0]) * _heights(q[2], dims[1][0])
    elif shape == "box":
        sx, sy = (sum(w * x * sinc(q[j] * x / 2) for x, w in zip(*dims[j])) for j in (0, 1))
        ff = sx * sy * sum(w * x * sinc(q[2] * x / 2) * torch.exp(0.5j * q[2] * x) for x, w in zip(*dims[2]))
    else:
        qq = torch.sqrt(q[0] ** 2 + q[1] ** 2 + q[2] ** 2)
        ff = sum(w * 4 * PI * ((torch.sin(qq * x) - qq * x * torch.cos(qq * x)) / qq ** 3) * torch.exp(1j * q[2] * x)
                 for x, w in zip(*dims[0]))
    va, vb, _ = ([20.0 * x for x in v] for v in HEX)
    sf = _dirichlet(va[0] * q[0] + va[1] * q[1], 20) * _dirichlet(vb[0] * q[0] + vb[1] * q[1], 20)
    A = (ff * sf * _fresnel(al, K0, ALPHA_I, *SUBSTRATE)[:, None, :]).sum(2)
    return {"intensity": (A.real ** 2 + A.imag ** 2).reshape(-1), "ff": ff.permute(2, 0, 1).reshape(-1)}


# --------------------------------------------------------------------- work ----
def work(case):
    """Inputs read once, outputs written once; operations of the factorised sums: per (pixel,
    triangle) an in-plane phasor (about 12) and its products with the row's four complex phasors
    and three normal components (96), per analytic q-point the samples' transcendentals (about 20
    operations each)."""
    kind = case["kind"]
    if kind in ("mesh", "call", "gradient"):
        px, t = case["ncol"] * case["nrow"], _tri(case)
        flops = 108.0 * px * t
        if kind == "mesh":
            return {"bytes": 16.0 * px + 64.0 * t + px * (32.0 if case["prec"] == "f32c" else 64.0), "flops": flops}
        if kind == "call":
            return {"bytes": 144.0 * px + 64.0 * t, "flops": flops}
        return {"bytes": 24.0 * px + 24.0 * t + 12.0 * t, "flops": 2.5 * flops}
    if kind == "batch":
        px = case["ncand"] * ((case["roi_min"] + case["roi_max"]) / 2) ** 2
        return {"bytes": 24.0 * px, "flops": 150.0 * px}
    if kind == "hig":
        px, g = case["n_y"] * case["n_z"], case["grains"] ** 2
        return {"bytes": 24.0 * px, "flops": px * g * (20.0 * case["samples"] * 5 + 4 * 60.0 + 100.0)}
    px = case["ncol"] * case["nrow"]
    return {"bytes": px * (16.0 + 3 * 64.0 + 8.0), "flops": 4.0 * px * (20.0 * case["samples"] * 3 + 100.0)}
