"""The column kernels by their own rules (the walk in as many runs as the number of columns asks for, one or two columns per lane)
and the older kernels behind them, with the mirrored-row and row-pair kernels off: what they serve when those decline -- a handful of
items on many columns, outputs whose rows are not dense."""
import pytest
import torch

from test_column_kernels import CASES, U, check

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def G():
    import gelib_b200
    assert torch.cuda.is_available(), "these tests need a CUDA device"
    gelib_b200._lib.lib()
    return gelib_b200


@pytest.fixture(params=["auto", "0"])
def col(request, G):
    G._lib.set_option("mir", "0")
    G._lib.set_option("col", request.param)
    yield request.param
    G._lib.set_option("col", "auto")
    G._lib.set_option("mir", "auto")


@pytest.mark.parametrize("diag,B,tx,ty,maxl", CASES + [(True, 2, U(8, 128), U(8, 128), 8), (False, 4, U(4, 1), {0: 32, 2: 32}, 6), (False, 3, U(2, 1), {1: 5, 2: 5}, 4)])
def test_products_and_gradients(G, oracle, col, diag, B, tx, ty, maxl):
    check(G, oracle, diag, B, tx, ty, maxl)


@pytest.mark.parametrize("diag,tx,ty", [(True, U(3, 12), U(3, 12)), (True, U(2, 40), U(2, 40)), (False, U(2, 1), U(2, 16))])
@pytest.mark.parametrize("xb,yb", [(True, False), (False, True)])
def test_operand_broadcast_over_the_batch(G, oracle, col, diag, tx, ty, xb, yb):
    check(G, oracle, diag, 9, tx, ty, 3, xb, yb)
