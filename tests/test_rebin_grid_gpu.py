"""The rebin's launch follows its work (particles and cells; the number of
blocks is read from a captured graph), and boxes of any size that do not fit
the cell table are reported."""
import numpy as np
import pytest
import torch

from pysph_b200 import _native as nat
from pysph_b200.engine import Engine, fluid_scheme

pytestmark = pytest.mark.gpu


def _rebin_blocks(eng):
    driver = pytest.importorskip("cuda.bindings.driver")

    def ok(res):
        assert res[0] == driver.CUresult.CUDA_SUCCESS, res[0]
        return res[1:]
    eng.rebin_now()
    g = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(g):
        eng.call("sphb_bin", eng.cur, nat.BIN_IF_NEEDED)
    graph = driver.CUgraph(init_value=g.raw_cuda_graph())
    _, n = ok(driver.cuGraphGetNodes(graph, 0))
    nodes, _ = ok(driver.cuGraphGetNodes(graph, n))
    return [ok(driver.cuGraphKernelNodeGetParams(k))[0].gridDimX for k in nodes[:n]]


def _engine(n, side, dim, **kw):
    rng = np.random.default_rng(n)
    x, y, z = rng.uniform(0, side, (3, n))
    if dim == 2:
        z = 0 * z
    o = np.ones(n)
    arr = dict(x=x, y=y, z=z, u=0 * o, v=0 * o, w=0 * o, m=o, h=0.4 * o, rho=o, p=0 * o, cs=o)
    return Engine([([arr], dict(dt=1e-9))], fluid_scheme(1), dim=dim, precision="fp64", **kw)


@pytest.mark.parametrize("dim,side", [(2, 1000.0), (3, 100.0)])
def test_scattered_particles_get_the_blocks_their_cells_need(dim, side):
    """1,000 particles (four tiles) over a million cells: the scan's 245
    chunks are not left to four blocks."""
    eng = _engine(1000, side, dim)
    assert eng.cell_capacity > 1e6
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert _rebin_blocks(eng) == [2 * sms]
    eng.check_status()


@pytest.mark.parametrize("cells", [4096, 4097, 5 * 4096])
def test_small_engines_wait_for_few_blocks(cells):
    eng = _engine(1000, 10.0, 2, cell_capacity=cells)
    assert _rebin_blocks(eng) == [max(4, -(-cells // 4096))]
    eng.check_status()


@pytest.mark.parametrize("precision", ["fp64", "fp32c"])
@pytest.mark.parametrize("cells", [2.1e6, 2.0 ** 21 - 8, 4.0e6, 3.0e7, 9.9e7])
def test_boxes_whose_cells_overflow_64_bits_are_reported(cells, precision):
    """cells an axis in 3D: 2.1e6 cubed is past 2^63, so a 64-bit product is
    negative and looks as if it fitted the capacity.  The grid is refused, and
    the engine works again with the particles back."""
    rng = np.random.default_rng(1)
    n = 300
    x, y, z = rng.uniform(0, 1, (3, n))
    o = np.ones(n)
    arr = dict(x=x, y=y, z=z, u=0 * o, v=0 * o, w=0 * o, m=o, h=0.1 * o, rho=o, p=0 * o, cs=o)
    eng = Engine([([arr], dict(dt=1e-9))], fluid_scheme(1), dim=3, precision=precision)
    eng.density()
    eng.check_status()
    want = eng.get(0, "rho")
    start = {c: eng.get(0, c) for c in "xyz"}
    for c in "xyz":
        eng.exchange_in(0, c, start[c] * (cells * eng.cell_size()))
    eng.density()
    assert eng.status() & nat.ST_GRID_OVERFLOW
    for c in "xyz":
        eng.exchange_in(0, c, start[c])
    eng.rebin_now()
    eng.clear_status()
    eng.rebin_now()
    eng.density()
    eng.check_status()
    assert torch.allclose(eng.get(0, "rho"), want, rtol=1e-6, atol=0)
