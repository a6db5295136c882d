"""That the native host side takes the plain forms of operand, and leaves the others to the Python code: equal results of both
(test_native_host.py) would not show a native function that declines every call."""
import pytest
import torch

from test_native_host import FORMS, leaf, operand

pytestmark = pytest.mark.gpu


@pytest.fixture
def G(monkeypatch):
    import gelib_b200
    assert torch.cuda.is_available(), "these tests need a CUDA device"
    return gelib_b200


class Counts:
    """The native functions; remembers which calls they took."""

    def __init__(self, module):
        self.module, self.took = module, []

    def __getattr__(self, name):
        def call(*args):
            r = getattr(self.module, name)(*args)
            self.took.append((name, r is not None))
            return r
        return call


@pytest.fixture
def counts(G, monkeypatch):
    c = Counts(G._lib.native())
    assert hasattr(c.module, "vec_forward") and c.module.__name__ == "gelib_b200._native"
    monkeypatch.setattr(G._lib, "_native", c)
    return c


@pytest.mark.parametrize("lx,ly,how,need", FORMS)
@pytest.mark.parametrize("kind", ["vec", "diag", "part", "diagpart"])
def test_products(G, counts, kind, lx, ly, how, need):
    diag, arr, n = kind.startswith("diag"), len(lx) > 1, 3 if kind.startswith("diag") else 2
    if kind.endswith("part"):
        x, y = leaf(G, operand(1, lx, 2, 3, how), need[0], how, arr), leaf(G, operand(2, ly, 1, n, "plain"), need[1], "plain", arr)
        cls = G.SO3partArr if arr else G.SO3part
        out = [(G.DiagCGproduct if diag else G.CGproduct)(cls(x) if how == "Parameter" else x, y, 2)]
    else:
        x, y = ([leaf(G, operand(k + l, d, l, c, h), m, h, arr) for l in ls]
                for k, d, c, h, m, ls in ((0, lx, 3, how, need[0], (1, 2)), (5, ly, n, "plain", need[1], (0, 2))))
        V = G.SO3vecArr if arr else G.SO3vec
        out = list((G.DiagCGproduct if diag else G.CGproduct)(V(*x), V(*y), 3).parts.values())
    if any(need):
        torch.autograd.backward(out, [torch.ones_like(t) for t in out])
    kind = "part" if kind.endswith("part") else "vec"
    plain = how != "conj" and len(lx) <= 3
    assert counts.took == [(kind + "_forward", plain)] + [(kind + "_backward", plain)] * any(need)


@pytest.mark.parametrize("how", ["plain", "conj", "swapped"])
def test_gathers(G, counts, how):
    gmap = G.gather_map.sources_targets([0, 1, 1, 3], [0, 0, 4, 2], 4, 5)
    r = G.gather(leaf(G, operand(3, (2, 4), 1, 3, how), 1, how, True), gmap, 0)
    r.backward(torch.ones_like(r))
    assert counts.took == [("gather", how != "conj"), ("gather", True)]
