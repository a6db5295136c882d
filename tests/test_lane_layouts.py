"""The lane layouts of the FP32 product kernels: channel counts around the tile sizes of every layout, batches that do not
fill a warp's cells, and calls small enough that several blocks share a cell (gradients added with atomics).  Small calls
choose few of the layouts, so each is pinned once."""
import numpy as np
import pytest
import torch

from util import crandn, np_c, rel_err

pytestmark = pytest.mark.gpu

TOL = 1e-5


@pytest.fixture(scope="module")
def G():
    import gelib_b200
    assert torch.cuda.is_available(), "these tests need a CUDA device"
    gelib_b200._lib.lib()
    return gelib_b200


@pytest.mark.parametrize("n1,n2", [(16, 16), (15, 16), (17, 18), (16, 15), (8, 8), (9, 7), (7, 8), (12, 10), (5, 24), (24, 6), (33, 5)])
@pytest.mark.parametrize("B,lmax", [(1, 2), (3, 3), (77, 2), (600, 1)])
def test_uniform_vectors(G, oracle, n1, n2, B, lmax):
    run(G, oracle, B, {l: n1 for l in range(lmax + 1)}, {l: n2 for l in range(lmax + 1)}, lmax)


@pytest.mark.parametrize("tx,ty,maxl", [({0: 12, 1: 9, 2: 7, 3: 5}, {0: 10, 1: 7, 2: 3}, 3), ({0: 40, 3: 6}, {1: 17, 2: 16}, -1)])
@pytest.mark.parametrize("B", [2, 150])
def test_ragged_vectors(G, oracle, tx, ty, maxl, B):
    run(G, oracle, B, tx, ty, maxl)


# the layouts of the kernels: {n1 and n2 of a warp's tile, cells of a warp}, in their order
FWD = [(16, 32, 1), (8, 32, 1), (16, 16, 2), (1, 16, 8), (8, 8, 8), (8, 8, 4), (4, 8, 8), (1, 4, 32), (16, 4, 8)]
BWD = [(32, 32, 1), (16, 16, 2), (8, 8, 8), (8, 8, 4), (8, 16, 2), (1, 16, 8), (4, 4, 8), (16, 2, 8)]


@pytest.fixture
def pinned(G):
    def pin(fwd, bwd):
        for name, value in (("fwd", "simt"), ("bwd", "simt"), ("col", "0"), ("fwd_layout", fwd), ("bwd_layout", bwd)):
            G._lib.set_option(name, value)

    yield pin
    for name in ("fwd", "bwd", "col", "fwd_layout", "bwd_layout"):
        G._lib.set_option(name, "auto")


@pytest.mark.parametrize("kernel,index", [("fwd", i) for i in range(len(FWD))] + [("bwd", i) for i in range(len(BWD))])
@pytest.mark.parametrize("d1,d2", [(0, 0), (-1, 1), (1, -1), (1, 2)])
def test_every_layout_around_its_tile(G, oracle, pinned, kernel, index, d1, d2):
    """A pinned layout (a call that it does not fit would be refused), with cells that do not fill a warp."""
    n1, n2, cells = (FWD if kernel == "fwd" else BWD)[index]
    n1, n2 = max(5, n1 + d1), max(1, n2 + d2)  # a narrow x has kernels of its own
    pinned(index if kernel == "fwd" else "auto", index if kernel == "bwd" else "auto")
    run(G, oracle, cells + 3, {0: n1, 2: n1}, {1: n2, 2: n2}, 3)


def run(G, oracle, B, tx, ty, maxl):
    V = G.backend.SO3vec.view
    mk = lambda s, tau: {l: crandn(s + l, B, 2 * l + 1, n) for l, n in tau.items()}
    tr = oracle.cg_type(tx, ty, maxl)
    x, y, g = mk(1, tx), mk(50, ty), mk(100, tr)
    nx, ny, ng = ({l: np_c(t) for l, t in d.items()} for d in (x, y, g))
    dx, dy, dg = ([t.cuda() for t in d.values()] for d in (x, y, g))
    r = [torch.empty(B, 2 * l + 1, n, dtype=torch.complex64, device="cuda") for l, n in tr.items()]
    V(r).addCGproduct(V(dx), V(dy), overwrite=True)
    want = {l: np.zeros((B, 2 * l + 1, n), np.complex64) for l, n in tr.items()}
    oracle.vec_cg(want, nx, ny)
    for t, w in zip(r, want.values()):
        assert rel_err(t, w) < TOL
    xg, yg = [torch.ones_like(t) for t in dx], [torch.ones_like(t) for t in dy]
    G.backend.SO3vec.addCGproduct_back01(V(xg), V(yg), V(dg), V(dx), V(dy))
    wx, wy = {l: np.ones_like(t) for l, t in nx.items()}, {l: np.ones_like(t) for l, t in ny.items()}
    oracle.vec_cg_back0(wx, ng, ny)
    oracle.vec_cg_back1(wy, ng, nx)
    for t, w in zip(xg + yg, list(wx.values()) + list(wy.values())):
        assert rel_err(t, w) < TOL
