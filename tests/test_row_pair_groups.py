"""The row-pair gradient where an item holds eight output l, and where a pair has more than an item holds and is split into groups
that add to the same rows, against the CPU oracle; and that pinned calls run the mirrored-row and row-pair kernels at all."""
import pytest
import torch

from test_column_kernels import U, check, cuda, parts, vec

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def G():
    import gelib_b200
    assert torch.cuda.is_available(), "these tests need a CUDA device"
    gelib_b200._lib.lib()
    return gelib_b200


@pytest.fixture(autouse=True)
def pinned(G):
    G._lib.set_option("mir", "one")
    yield
    G._lib.set_option("mir", "auto")


# output l of the largest pairs: 8; 9 in two groups, beside pairs of 8; 9; 15 in groups of seven and eight; 13 and 12; ten, cut off by maxl
GROUPS = [(33, U(7, 1), U(7, 3), 7), (9, U(8, 1), U(8, 9), 8), (40, {4: 1}, {4: 10}, -1), (5, {7: 1}, {7: 5}, -1), (17, {6: 1, 7: 1}, {6: 4}, -1),
          (11, {1: 1, 5: 1}, {5: 33, 6: 33}, 10)]


@pytest.mark.parametrize("B,tx,ty,maxl", GROUPS)
def test_groups_of_a_pair(G, oracle, B, tx, ty, maxl):
    check(G, oracle, False, B, tx, ty, maxl)


# every kernel sums in one order of its own
@pytest.mark.parametrize("diag,B,tx,ty,maxl", [(False,) + c for c in GROUPS] + [(True, 11, U(3, 12), U(3, 12), 3), (True, 2, U(8, 32), U(8, 32), 8),
                                                                              (False, 5, U(3, 1), U(3, 16), 3), (False, 33, U(6, 1), U(6, 16), 6)])
def test_pinned_calls_run_these_kernels(G, oracle, diag, B, tx, ty, maxl):
    tr = oracle.cg_type(tx, ty, maxl, diag)
    x, y, g = cuda(parts(1, B, tx)), cuda(parts(100, B, ty)), cuda(parts(200, B, tr))

    def results(mir):
        G._lib.set_option("mir", mir)
        r, yg = {l: torch.empty_like(t) for l, t in g.items()}, {l: torch.zeros_like(t) for l, t in y.items()}
        (vec(G, r).addDiagCGproduct if diag else vec(G, r).addCGproduct)(vec(G, x), vec(G, y), overwrite=True)
        (vec(G, yg).addDiagCGproduct_back1 if diag else vec(G, yg).addCGproduct_back1)(vec(G, g), vec(G, x))
        return r, yg

    same = [all(torch.equal(a[l], b[l]) for l in a) for a, b in zip(results("one"), results("0"))]
    assert same == [False, diag]  # diagonal products of several channels have no row-pair gradient
