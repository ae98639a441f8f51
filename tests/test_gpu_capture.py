"""The triangle form factor captured into a CUDA graph: without an allocation inside the capture, and with
every buffer of the graph left in place by later, larger calls.  A replay equals the call itself to the
kernels' bounds (1e-12 in FP64, where a captured call doesn't split its triangles, 1e-5 in FP32C)."""
import numpy as np
import pytest

import hipgisaxs_b200 as hg
from test_gpu_ff_rows_f64 import cloud

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def setup(po, ncol, nrow, ntri, ctx):
    G = po.Grid(ncol, nrow, -1.87, 0.01, 2.0, 3.0, 0.2, 10.0)
    g = hg.QGrid.from_arrays(ctx, G.qx, G.qy, G.qz_ext, ncol)
    sd = torch.tensor(cloud(np.random.default_rng(ncol + ntri), ntri), device="cuda")
    return g, sd, torch.zeros(4 * G.n, dtype=torch.complex128, device="cuda")


def capture(ctx, stream, call):
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, stream=stream):
        call()
    return graph


def replayed(graph, out):
    out.zero_()
    graph.replay()
    torch.cuda.synchronize()
    return out.cpu().numpy()


@pytest.mark.parametrize("precision,warm", [("f64", False), ("f32c", True), ("f32c", False)])
def test_captured_call(po, precision, warm):
    stream = torch.cuda.Stream()
    ctx = hg.Context(0, stream)
    g, sd, out = setup(po, 40, 6, 2000, ctx)
    small = setup(po, 8, 2, 2000, ctx)
    torch.cuda.synchronize()
    if precision == "f32c":  # its tiles, by a call on a smaller grid
        hg.ff_triangles(ctx, small[0], sd, None, precision, out=small[2])
    if warm:
        hg.ff_triangles(ctx, g, sd, None, precision, out=out)
    ctx.synchronize()
    graph = capture(ctx, stream, lambda: hg.ff_triangles(ctx, g, sd, None, precision, out=out))
    first = replayed(graph, out)
    # larger calls in both precisions (FP32C on the same triangles: the tiles are the graph's)
    big = setup(po, 300, 200, 2000, ctx)
    torch.cuda.synchronize()
    for p in ("f64", "f32c"):
        hg.ff_triangles(ctx, big[0], sd, None, p, out=big[2])
    ctx.synchronize()
    again = replayed(graph, out)
    direct = torch.zeros_like(out)
    torch.cuda.synchronize()
    hg.ff_triangles(ctx, g, sd, None, precision, out=direct)
    ctx.synchronize()
    assert np.array_equal(first, again)
    assert po.rel_err(first, direct.cpu().numpy()) < (1e-12 if precision == "f64" else 1e-5)
    del graph
    ctx.close()
