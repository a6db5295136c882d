"""The native host side of the products against the Python code that it stands in for: equal outputs and gradients over the
forms of operand that both take, and equal errors where both refuse."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def G():
    import gelib_b200
    assert torch.cuda.is_available(), "these tests need a CUDA device"
    gelib_b200._lib.lib()
    return gelib_b200


class Declines:
    def __getattr__(self, name):
        return lambda *args: None


@pytest.fixture
def python_only(G, monkeypatch):
    def switch():
        monkeypatch.setattr(G._lib, "_native", Declines())
    return switch


def rand(seed, *shape):
    return torch.randn(*shape, 2, generator=torch.Generator().manual_seed(seed)).cuda()


def crand(seed, *shape):
    return torch.view_as_complex(rand(seed, *shape))


# operands of a product: lead dimensions of x and y, what is done to x, which sides need a gradient
FORMS = [((5,), (5,), "plain", (1, 1)), ((5,), (1,), "plain", (1, 1)), ((5,), (5,), "plain", (1, 0)), ((5,), (5,), "plain", (0, 1)),
         ((5,), (5,), "plain", (0, 0)), ((2, 3), (2, 3), "plain", (1, 1)), ((2, 3), (2, 1), "plain", (1, 1)), ((2, 2, 3), (2, 2, 3), "plain", (1, 1)),
         ((2, 1, 2, 3), (2, 1, 2, 3), "plain", (1, 1)), ((5,), (5,), "conj", (1, 1)), ((5,), (5,), "cut", (1, 1)), ((5,), (5,), "swapped", (1, 1)),
         ((5,), (5,), "Parameter", (1, 1))]


def operand(seed, lead, l, n, how):
    if how == "conj":
        return crand(seed, *lead, 2 * l + 1, n).conj()
    if how == "cut":
        return crand(seed, *lead, 2 * l + 1, n + 3)[..., 1:n + 1]
    if how == "swapped":
        return crand(seed, *lead, n, 2 * l + 1).transpose(-1, -2)
    return crand(seed, *lead, 2 * l + 1, n)


def leaf(G, t, need, how, arr):
    t = t.detach()
    if how == "Parameter":
        return torch.nn.Parameter(t, requires_grad=bool(need))
    return (G.SO3partArr if arr else G.SO3part)(t).requires_grad_(bool(need))


def outcome(f):
    try:
        out = f()
    except Exception as e:  # noqa: BLE001
        return type(e), str(e)
    return out


def same(a, b):
    assert type(a) is type(b), (a, b)
    if not isinstance(a, list):
        assert a == b
        return
    assert len(a) == len(b)
    for s, t in zip(a, b):
        assert type(s) is type(t) and (s is None or (s.shape == t.shape and s.stride() == t.stride()))
        if s is not None:
            p, q = s.detach().as_subclass(torch.Tensor), t.detach().as_subclass(torch.Tensor)
            assert torch.allclose(p, q, rtol=1e-5, atol=1e-5)


@pytest.mark.parametrize("lx,ly,how,need", FORMS)
@pytest.mark.parametrize("kind", ["vec", "diag", "part", "diagpart"])
def test_outputs_and_gradients(G, python_only, kind, lx, ly, how, need):
    diag = kind.startswith("diag")
    arr = len(lx) > 1

    def run():
        nx, ny = (3, 3) if diag else (3, 2)
        if kind.endswith("part"):
            x = leaf(G, operand(1, lx, 2, nx, how), need[0], how, arr)
            y = leaf(G, operand(2, ly, 1, ny, "plain"), need[1], "plain", arr)
            cls = G.SO3partArr if arr else G.SO3part
            xs, ys = [x], [y]
            out = [(G.DiagCGproduct if diag else G.CGproduct)(cls(x) if how == "Parameter" else x, y, 2)]
        else:
            xs = [leaf(G, operand(l, lx, l, nx, how), need[0], how, arr) for l in (1, 2)]
            ys = [leaf(G, operand(5 + l, ly, l, ny, "plain"), need[1], "plain", arr) for l in (0, 2)]
            V = G.SO3vecArr if arr else G.SO3vec
            out = list((G.DiagCGproduct if diag else G.CGproduct)(V(*xs), V(*ys), 3).parts.values())
        grads = []
        if any(need):
            g = [crand(40 + i, *t.shape) for i, t in enumerate(out)]
            torch.autograd.backward(out, g)
            grads = [t.grad for t in xs + ys]
        return out + grads

    native = outcome(run)
    python_only()
    same(native, outcome(run))


@pytest.mark.parametrize("bad", ["batch", "dtype", "cpu", "channels", "twice", "rank"])
def test_refusals(G, python_only, bad):
    def run():
        x = [crand(l, 4, 2 * l + 1, 3) for l in (0, 1)]
        y = [crand(l, 4, 2 * l + 1, 3) for l in (0, 1)]
        if bad == "batch":
            y = [t[:3] for t in y]
        if bad == "dtype":
            y[1] = y[1].to(torch.complex128)
        if bad == "cpu":
            y = [t.cpu() for t in y]
        if bad == "channels":
            y = [t[..., :2] for t in y]
        if bad == "twice":
            y = [y[1], y[1].clone()]
        if bad == "rank":
            y = [t[0] for t in y]
        return list(G.DiagCGproduct(G.SO3vec(*x), G.SO3vec(*y), 1).parts.values())

    native = outcome(run)
    python_only()
    same(native, outcome(run))


@pytest.mark.parametrize("how", ["plain", "conj", "swapped"])
@pytest.mark.parametrize("lead,dim", [((2, 4), 0), ((2, 3, 4), 1)])
def test_gather(G, python_only, how, lead, dim):
    gmap = G.gather_map.sources_targets([0, 1, 1, 3], [0, 0, 4, 2], 4, 5)

    def run():
        x = leaf(G, operand(3, lead, 1, 3, how), 1, how, True)
        r = G.gather(x, gmap, dim)
        r.backward(crand(9, *r.shape))
        return [r, x.grad]

    native = outcome(run)
    python_only()
    same(native, outcome(run))
