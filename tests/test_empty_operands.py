"""An operand without cells against one that has some: nothing is computed, and the output is zero, not what its memory held."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def empty_memory_is_nan():
    torch.use_deterministic_algorithms(True)  # fills torch.empty with NaN
    yield
    torch.use_deterministic_algorithms(False)


@pytest.mark.parametrize("kind", ["vec", "diag", "part", "diagpart"])
@pytest.mark.parametrize("lead_x,lead_y,lead", [((0,), (1,), (1,)), ((5,), (0,), (5,)), ((0,), (0,), (0,)), ((2, 0), (2, 1), (2, 1))])
def test_products(kind, lead_x, lead_y, lead):
    import gelib_b200 as G
    part, vec = (G.SO3part, G.SO3vec) if len(lead) == 1 else (G.SO3partArr, G.SO3vecArr)
    make = lambda d, l: part(torch.ones(*d, 2 * l + 1, 3, dtype=torch.complex64, device="cuda"))
    f = G.DiagCGproduct if kind.startswith("diag") else G.CGproduct
    if kind.endswith("part"):
        out = {2: f(make(lead_x, 1), make(lead_y, 1), 2)}
    else:
        out = f(vec(*[make(lead_x, l) for l in (0, 1)]), vec(*[make(lead_y, l) for l in (0, 1)])).parts
    for l, p in out.items():
        assert tuple(p.shape[:-1]) == lead + (2 * l + 1,)
        assert not bool(p.as_subclass(torch.Tensor).abs().ne(0).any())


def test_fused_first_layer():
    import gelib_b200 as G
    y = G.SO3vec(*[G.SO3part(torch.ones(0, 2 * l + 1, 3, dtype=torch.complex64, device="cuda")) for l in (0, 1)])
    for p in G.SO3vec.spharm_CGproduct(1, torch.ones(4, 3, 1, device="cuda"), y).parts.values():
        assert not bool(p.as_subclass(torch.Tensor).abs().ne(0).any())


def test_with_parities():
    import gelib_b200 as G
    make = lambda b, mu: G.O3part(torch.ones(b, 2 * mu[0] + 1, 3, dtype=torch.complex64, device="cuda"), mu)
    out = list(G.CGproduct(G.O3vec(make(0, (1, -1))), G.O3vec(make(4, (1, -1)))).parts.values())
    for p in out + [make(0, (1, -1)).CGproduct(make(4, (1, -1)), (2, 1))]:
        assert p.size(0) == 4 and not bool(p.as_subclass(torch.Tensor).abs().ne(0).any())
