"""The column kernels (diagonal products, products with a one-channel x): every direction against the CPU oracle at the
edges of their range -- column counts that do not fill a warp, pairs with more output l than one pass holds, types with
gaps, truncated outputs, accumulation, broadcast operands, strided operands, grids -- and non-finite inputs.  Each case runs
by the rules ("auto": few cells, so mostly the walk split over blocks), pinned to one and to two columns per lane with the
walk in one piece, which the rules leave to calls too large for the oracle, and pinned to each way of splitting the walk."""
import numpy as np
import pytest
import torch

from util import crandn, np_c, rel_err

pytestmark = pytest.mark.gpu

TOL = 1e-5
TOL_BIG = 1e-4  # sums over maxl >= 6


@pytest.fixture(scope="module")
def G():
    import gelib_b200
    assert torch.cuda.is_available(), "these tests need a CUDA device"
    gelib_b200._lib.lib()
    return gelib_b200


@pytest.fixture(params=["auto", "one", "two"] + ["split%d" % k for k in range(1, 13)])
def col(request, G):
    G._lib.set_option("col", request.param)
    yield request.param
    G._lib.set_option("col", "auto")


def parts(seed, B, tau, bcast=False):
    return {l: crandn(seed + l, 1 if bcast else B, 2 * l + 1, n) for l, n in tau.items()}


def vec(G, d):
    return G.backend.SO3vec.view(list(d.values()))


def cuda(d):
    return {l: t.cuda() for l, t in d.items()}


U = lambda lmax, n: {l: n for l in range(lmax + 1)}

CASES = [
    # (diagonal, batch, x, y, maxl)
    (True, 1, {0: 1}, {0: 1}, -1), (True, 3, U(2, 5), U(2, 5), 2), (True, 11, U(3, 12), U(3, 12), 3), (True, 1000, U(2, 3), U(2, 3), 2),
    (True, 5, U(4, 33), U(3, 33), 4), (True, 2, U(8, 32), U(8, 32), 8), (True, 2, {8: 7}, {8: 7}, 15), (True, 2, {6: 20}, {5: 20}, -1),
    (True, 4, {1: 9, 4: 9}, {0: 9, 2: 9, 8: 9}, 6), (True, 3, U(3, 4), {12: 4, 20: 4}, -1), (True, 4700, U(1, 33), U(1, 33), 1),
    (False, 5, U(3, 1), U(3, 16), 3), (False, 33, U(6, 1), U(6, 16), 6), (False, 7, U(2, 1), U(4, 40), -1), (False, 300, U(2, 1), U(2, 7), 2),
    (False, 2, {0: 1, 7: 1}, {3: 65}, -1),
    (True, 5, U(2, 34), U(2, 34), 2), (True, 2, {6: 48, 8: 48}, {0: 48, 7: 48}, 8), (False, 9, {0: 1, 5: 1}, U(4, 24), 5),
    (True, 2, {9: 17}, {9: 17}, 4),  # beyond the column kernels: one cell per CTA
]


def check(G, oracle, diag, B, tx, ty, maxl, xb=False, yb=False):
    tr = oracle.cg_type(tx, ty, maxl, diag)
    x, y = parts(1, B, tx, xb), parts(100, B, ty, yb)
    g, r0 = parts(200, B, tr), parts(300, B, tr)
    nx, ny, ng = ({l: np_c(t) for l, t in d.items()} for d in (x, y, g))
    tol = TOL_BIG if max(tr) >= 6 or xb or yb else TOL
    dx, dy, dg = cuda(x), cuda(y), cuda(g)
    for overwrite in (True, False):
        r = cuda(r0)
        (vec(G, r).addDiagCGproduct if diag else vec(G, r).addCGproduct)(vec(G, dx), vec(G, dy), overwrite=overwrite)
        want = {l: np.zeros((B, 2 * l + 1, n), np.complex64) if overwrite else np_c(r0[l]).copy() for l, n in tr.items()}
        oracle.vec_cg(want, nx, ny, diag)
        for l in tr:
            assert rel_err(r[l], want[l]) < tol, ("forward", overwrite, l)
    wx, wy = {l: np.ones_like(t) for l, t in nx.items()}, {l: np.ones_like(t) for l, t in ny.items()}
    oracle.vec_cg_back0(wx, ng, ny, diag)
    oracle.vec_cg_back1(wy, ng, nx, diag)
    V = G.backend.SO3vec
    ones = lambda d: {l: torch.ones_like(t) for l, t in d.items()}
    xg, yg = ones(dx), ones(dy)
    (V.addDiagCGproduct_back01 if diag else V.addCGproduct_back01)(vec(G, xg), vec(G, yg), vec(G, dg), vec(G, dx), vec(G, dy))
    xg1, yg1 = ones(dx), ones(dy)
    (vec(G, xg1).addDiagCGproduct_back0 if diag else vec(G, xg1).addCGproduct_back0)(vec(G, dg), vec(G, dy))
    (vec(G, yg1).addDiagCGproduct_back1 if diag else vec(G, yg1).addCGproduct_back1)(vec(G, dg), vec(G, dx))
    for got in (xg, xg1):
        for l in wx:
            assert rel_err(got[l], wx[l]) < tol, ("xg", l)
    for got in (yg, yg1):
        for l in wy:
            assert rel_err(got[l], wy[l]) < tol, ("yg", l)


@pytest.mark.parametrize("diag,B,tx,ty,maxl", CASES)
def test_products_and_gradients(G, oracle, col, diag, B, tx, ty, maxl):
    check(G, oracle, diag, B, tx, ty, maxl)


@pytest.mark.parametrize("diag,tx,ty", [(True, U(3, 12), U(3, 12)), (True, U(2, 40), U(2, 40)), (False, U(2, 1), U(2, 16))])
@pytest.mark.parametrize("xb,yb", [(True, False), (False, True)])
def test_operand_broadcast_over_the_batch(G, oracle, col, diag, tx, ty, xb, yb):
    check(G, oracle, diag, 9, tx, ty, 3, xb, yb)


@pytest.mark.parametrize("pad", [3, 4])
@pytest.mark.parametrize("diag,n", [(True, 12), (True, 20), (False, 12)])
def test_strided_rows_and_grids(G, oracle, col, diag, n, pad):
    """Operands cut out of larger tensors (rows a multiple of 16 bytes apart or not), on a contiguous grid and on one that
    is no arithmetic progression of cells and goes to the other kernels (with 20 channels: one cell per CTA)."""
    nx = n if diag else 1
    for grid, cut in (((3,), False), ((3,), True), ((2, 3), False)):
        def make(seed, l, ch, odd):
            t = crandn(seed, 4, *[k + (cut and i == 0) for i, k in enumerate(grid)], 2 * l + 1, ch + (pad if odd else 0)).cuda()
            return t[:, :grid[0]][..., :ch] if odd or cut else t
        x = {l: make(l, l, nx, True) for l in range(3)}
        y = {l: make(10 + l, l, n, l == 1) for l in range(3)}
        cells = 4 * int(np.prod(grid))
        flat = lambda d: {l: np_c(t.contiguous().reshape(cells, 2 * l + 1, -1)) for l, t in d.items()}
        tr = oracle.cg_type({l: nx for l in x}, {l: n for l in y}, 2, diag)
        r = {l: torch.empty(4, *grid, 2 * l + 1, c, dtype=torch.complex64, device="cuda") for l, c in tr.items()}
        (vec(G, r).addDiagCGproduct if diag else vec(G, r).addCGproduct)(vec(G, x), vec(G, y), overwrite=True)
        want = {l: np.zeros((cells, 2 * l + 1, c), np.complex64) for l, c in tr.items()}
        oracle.vec_cg(want, flat(x), flat(y), diag)
        for l in tr:
            assert rel_err(r[l].reshape(cells, 2 * l + 1, -1), want[l]) < TOL, (grid, cut, l)
        g = {l: torch.randn_like(t) for l, t in r.items()}
        yg = {l: torch.zeros(4, *grid, 2 * l + 1, n, dtype=torch.complex64, device="cuda") for l in y}
        if diag:
            xg = {l: torch.zeros(4, *grid, 2 * l + 1, n, dtype=torch.complex64, device="cuda") for l in x}
            G.backend.SO3vec.addDiagCGproduct_back01(vec(G, xg), vec(G, yg), vec(G, g), vec(G, x), vec(G, y))
            wx = {l: np.zeros((cells, 2 * l + 1, n), np.complex64) for l in x}
            oracle.vec_cg_back0(wx, flat(g), flat(y), diag)
            for l in wx:
                assert rel_err(xg[l].reshape(cells, 2 * l + 1, -1), wx[l]) < TOL, (grid, cut, l)
        else:
            vec(G, yg).addCGproduct_back1(vec(G, g), vec(G, x))
        wy = {l: np.zeros((cells, 2 * l + 1, n), np.complex64) for l in y}
        oracle.vec_cg_back1(wy, flat(g), flat(x), diag)
        for l in wy:
            assert rel_err(yg[l].reshape(cells, 2 * l + 1, -1), wy[l]) < TOL, (grid, cut, l)


@pytest.mark.parametrize("l", [1, 4, 8])
def test_an_infinity_stays_in_its_band(G, oracle, col, l):
    """x[m1] = inf reaches the rows that m1 couples to and no other."""
    tx, ty = {l: 6}, {l: 6}
    x, y = parts(1, 3, tx), parts(50, 3, ty)
    x[l][1, 0, 2] = complex(float("inf"), 0.)
    tr = oracle.cg_type(tx, ty, 15, True)
    g = parts(90, 3, tr)
    g[0][2, 0, 1] = complex(float("inf"), 0.)
    dx, dy, dg = cuda(x), cuda(y), cuda(g)
    r = {k: torch.empty(3, 2 * k + 1, n, dtype=torch.complex64, device="cuda") for k, n in tr.items()}
    vec(G, r).addDiagCGproduct(vec(G, dx), vec(G, dy), overwrite=True)
    want = {k: np.zeros((3, 2 * k + 1, n), np.complex64) for k, n in tr.items()}
    with np.errstate(all="ignore"):
        oracle.vec_cg(want, {k: np_c(t) for k, t in x.items()}, {k: np_c(t) for k, t in y.items()}, True)
        for k in tr:
            assert (np.isfinite(np_c(r[k])) == np.isfinite(want[k])).all(), k
        xg = {l: torch.zeros_like(dx[l])}
        yg = {l: torch.zeros_like(dy[l])}
        x[l][1, 0, 2] = 1.
        dx = cuda(x)
        G.backend.SO3vec.addDiagCGproduct_back01(vec(G, xg), vec(G, yg), vec(G, dg), vec(G, dx), vec(G, dy))
        wx = {l: np.zeros_like(np_c(x[l]))}
        oracle.vec_cg_back0(wx, {k: np_c(t) for k, t in g.items()}, {k: np_c(t) for k, t in y.items()}, True)
    assert (np.isfinite(np_c(xg[l])) == np.isfinite(wx[l])).all()


@pytest.mark.parametrize("diag,B,tx,ty,maxl", [
    (True, 16, U(4, 8), U(4, 8), 4), (True, 500, U(3, 12), U(3, 12), 3), (True, 30, U(8, 16), U(8, 16), 8), (True, 40, U(3, 15), U(5, 15), 5),
    (True, 4, U(3, 4), {9: 4, 12: 4, 20: 4}, -1), (False, 33, U(6, 1), U(6, 16), 6), (False, 500, U(4, 1), U(4, 8), 4),
])
def test_gradients_are_repeatable(G, oracle, col, diag, B, tx, ty, maxl):
    """Few columns: blocks share the walk, yet a gradient row is added to in one order (but for splits by pairs, the last)."""
    if col in ("split9", "split10", "split11", "split12"):
        pytest.skip("several blocks add to a row")
    tr = oracle.cg_type(tx, ty, maxl, diag)
    x, y, g = cuda(parts(1, B, tx)), cuda(parts(100, B, ty)), cuda(parts(200, B, tr))
    x0, y0 = cuda(parts(300, B, tx)), cuda(parts(400, B, ty))
    first = None
    for _ in range(10):
        xg, yg = {l: t.clone() for l, t in x0.items()}, {l: t.clone() for l, t in y0.items()}
        y1 = {l: t.clone() for l, t in y0.items()}
        if diag:
            G.backend.SO3vec.addDiagCGproduct_back01(vec(G, xg), vec(G, yg), vec(G, g), vec(G, x), vec(G, y))
            vec(G, y1).addDiagCGproduct_back1(vec(G, g), vec(G, x))
        else:
            vec(G, y1).addCGproduct_back1(vec(G, g), vec(G, x))
        got = [torch.view_as_real(t) for d in (xg, yg, y1) for t in d.values()]
        first = first or got
        assert all(torch.equal(a, b) for a, b in zip(first, got))
