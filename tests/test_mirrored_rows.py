"""The mirrored-row kernels (diagonal products and products with a one-channel x on a full chip) pinned on small calls, with
one and with two columns per lane, against the CPU oracle: column counts that do not fill a warp, blocks that touch several
cells, pairs with more output l than an item holds, lopsided pairs, types with gaps, truncated outputs, accumulation, single
gradients, broadcast operands, strided rows, and non-finite inputs, which must reach only what they are a factor of."""
import numpy as np
import pytest
import torch

from test_column_kernels import CASES, U, check, cuda, parts, vec
from util import np_c

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def G():
    import gelib_b200
    assert torch.cuda.is_available(), "these tests need a CUDA device"
    gelib_b200._lib.lib()
    return gelib_b200


@pytest.fixture(params=["one", "two"])
def mir(request, G):
    G._lib.set_option("mir", request.param)
    yield request.param
    G._lib.set_option("mir", "auto")


EXTRA = [(False, 40, U(2, 1), U(6, 6), 6), (False, 3, {12: 1, 20: 1}, U(3, 10), -1), (True, 70, U(3, 1), U(3, 1), 3)]


@pytest.mark.parametrize("diag,B,tx,ty,maxl", CASES + EXTRA)
def test_products_and_gradients(G, oracle, mir, diag, B, tx, ty, maxl):
    check(G, oracle, diag, B, tx, ty, maxl)


@pytest.mark.parametrize("diag,tx,ty", [(True, U(3, 12), U(3, 12)), (False, U(2, 1), U(2, 16))])
@pytest.mark.parametrize("xb,yb", [(True, False), (False, True)])
def test_operand_broadcast_over_the_batch(G, oracle, mir, diag, tx, ty, xb, yb):
    check(G, oracle, diag, 9, tx, ty, 3, xb, yb)


def crandn_padded(seed, B, l, ch, pad):
    t = torch.randn(B, 2 * l + 1, ch + pad, 2, generator=torch.Generator().manual_seed(seed))
    return torch.view_as_complex(t).cuda()[..., :ch]


@pytest.mark.parametrize("diag,n", [(True, 12), (False, 12)])
@pytest.mark.parametrize("pad", [3, 4])
def test_strided_rows(G, oracle, mir, diag, n, pad):
    B, nx = 5, n if diag else 1
    x = {l: crandn_padded(l, B, l, nx, pad) for l in range(4)}
    y = {l: crandn_padded(10 + l, B, l, n, pad) for l in range(4)}
    tr = oracle.cg_type({l: nx for l in x}, {l: n for l in y}, 3, diag)
    r = {l: torch.empty(B, 2 * l + 1, c, dtype=torch.complex64, device="cuda") for l, c in tr.items()}
    (vec(G, r).addDiagCGproduct if diag else vec(G, r).addCGproduct)(vec(G, x), vec(G, y), overwrite=True)
    want = {l: np.zeros((B, 2 * l + 1, c), np.complex64) for l, c in tr.items()}
    hx, hy = ({l: np_c(t.contiguous()) for l, t in d.items()} for d in (x, y))
    oracle.vec_cg(want, hx, hy, diag)
    for l in tr:
        assert np.abs(np_c(r[l]) - want[l]).max() < 1e-5 * np.abs(want[l]).max()
    yg = {l: torch.zeros_like(t) for l, t in y.items()}
    g = cuda(parts(50, B, tr))
    (vec(G, yg).addDiagCGproduct_back1 if diag else vec(G, yg).addCGproduct_back1)(vec(G, g), vec(G, x))
    wy = {l: np.zeros_like(t) for l, t in hy.items()}
    oracle.vec_cg_back1(wy, {l: np_c(t) for l, t in g.items()}, hx, diag)
    for l in wy:
        assert np.abs(np_c(yg[l]) - wy[l]).max() < 1e-5 * np.abs(wy[l]).max()


@pytest.mark.parametrize("value", [float("inf"), float("nan")])
@pytest.mark.parametrize("diag", [True, False])
def test_non_finite_inputs_stay_where_they_belong(G, oracle, mir, diag, value):
    """One non-finite number in x, in y, in g: exactly the outputs that it is a factor of become non-finite, as in the oracle
    (which multiplies by every coefficient inside a band, zeros among them, and by none outside)."""
    B, n = 3, 8
    tx, ty = U(3, n if diag else 1), U(3, n)
    tr = oracle.cg_type(tx, ty, 3, diag)
    for where in ("x", "y", "g"):
        x, y, g = parts(1, B, tx), parts(100, B, ty), parts(200, B, tr)
        {"x": x, "y": y, "g": g}[where][2][1, 1, 0] = value
        nx, ny, ng = ({l: np_c(t) for l, t in d.items()} for d in (x, y, g))
        r = {l: torch.empty(B, 2 * l + 1, c, dtype=torch.complex64, device="cuda") for l, c in tr.items()}
        (vec(G, r).addDiagCGproduct if diag else vec(G, r).addCGproduct)(vec(G, cuda(x)), vec(G, cuda(y)), overwrite=True)
        want = {l: np.zeros((B, 2 * l + 1, c), np.complex64) for l, c in tr.items()}
        oracle.vec_cg(want, nx, ny, diag)
        yg = cuda({l: torch.zeros_like(t) for l, t in y.items()})
        xg = cuda({l: torch.zeros_like(t) for l, t in x.items()})
        wy, wx = ({l: np.zeros_like(t) for l, t in d.items()} for d in (ny, nx))
        oracle.vec_cg_back1(wy, ng, nx, diag)
        pairs = [(r, want), (yg, wy)]
        if diag:
            G.backend.SO3vec.addDiagCGproduct_back01(vec(G, xg), vec(G, yg), vec(G, cuda(g)), vec(G, cuda(x)), vec(G, cuda(y)))
            oracle.vec_cg_back0(wx, ng, ny, diag)
            pairs.append((xg, wx))
        else:
            vec(G, yg).addCGproduct_back1(vec(G, cuda(g)), vec(G, cuda(x)))
        for got, exp in pairs:
            for l in exp:
                assert (np.isfinite(np_c(got[l])) == np.isfinite(exp[l])).all(), (where, l)


@pytest.mark.parametrize("diag,n,batches", [(True, 66, (3, 1100)), (True, 70, (1100, 3)), (False, 32, (4, 2100)), (False, 16, (4200, 4))])
def test_a_type_of_few_items_is_captured_at_another_batch(G, oracle, diag, n, batches):
    """Types of a handful of items leave these kernels when there are many columns: whichever batch comes first plans both."""
    tx, ty = {0: n if diag else 1, 1: n if diag else 1}, {1: n}
    tr = oracle.cg_type(tx, ty, 1, diag)

    def call(B):
        x, y = cuda(parts(1, B, tx)), cuda(parts(9, B, ty))
        r = {l: torch.empty(B, 2 * l + 1, c, dtype=torch.complex64, device="cuda") for l, c in tr.items()}
        return lambda: (vec(G, r).addDiagCGproduct if diag else vec(G, r).addCGproduct)(vec(G, x), vec(G, y), overwrite=True), r

    call(batches[0])[0]()
    f, r = call(batches[1])
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        f()
    graph.replay()
    torch.cuda.synchronize()
    got = {l: t.clone() for l, t in r.items()}
    f()
    for l in got:
        assert float((got[l] - r[l]).abs().max()) <= 1e-5 * float(r[l].abs().max())


def test_row_pair_gradient_by_the_rule(G, oracle):
    """Enough columns for the row-pair gradient to be taken by its rule, in the last cells of which the oracle is asked: the
    choice of kernel changes nothing, and a first small call plans what the large one runs."""
    n, lmax, B = 20, 3, 4900
    tx, ty = U(lmax, 1), U(lmax, n)
    tr = oracle.cg_type(tx, ty, lmax, False)
    cells = slice(B - 3, B)

    def call(B):
        x, g = parts(1, B, tx), parts(20, B, tr)
        dx, dg = cuda(x), cuda(g)
        yg = {l: torch.zeros(B, 2 * l + 1, n, dtype=torch.complex64, device="cuda") for l in ty}
        return (lambda: vec(G, yg).addCGproduct_back1(vec(G, dg), vec(G, dx))), yg, x, g

    call(3)[0]()
    f, yg, x, g = call(B)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        f()
    graph.replay()
    torch.cuda.synchronize()
    want = {l: np.zeros((3, 2 * l + 1, n), np.complex64) for l in ty}
    oracle.vec_cg_back1(want, {l: np_c(t[cells]) for l, t in g.items()}, {l: np_c(t[cells]) for l, t in x.items()})
    for l in want:
        assert np.abs(np_c(yg[l][cells]) - want[l]).max() < 1e-5 * np.abs(want[l]).max()
