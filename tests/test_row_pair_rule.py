"""When the gradient of y for a one-channel x goes to the row-pair kernel: never where the sums would become less accurate than
those of the kernel that took the call otherwise."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def G():
    import gelib_b200
    assert torch.cuda.is_available(), "these tests need a CUDA device"
    gelib_b200._lib.lib()
    return gelib_b200


def crand(*shape):
    return torch.view_as_complex(torch.randn(*shape, 2, device="cuda"))


class Call:
    """Operands of the gradient of y, parts l = 0 .. maxl, at least `cols` columns."""

    def __init__(self, G, maxl, n, cols):
        torch.manual_seed(maxl * 64 + n)
        self.G, self.maxl, self.n, cells = G, maxl, n, -(-cols // n)
        V = G.backend.SO3vec.view
        self.x = [crand(cells, 2 * l + 1, 1) for l in range(maxl + 1)]
        self.y = [crand(cells, 2 * l + 1, n) for l in range(maxl + 1)]
        tau = V(self.x).get_tau().CGproduct(V(self.y).get_tau(), maxl)
        self.g = [crand(cells, 2 * l + 1, k) for l, k in tau.get_parts().items()]

    def gradient(self, mir):
        V = self.G.backend.SO3vec.view
        yg = [torch.zeros_like(t) for t in self.y]
        self.G._lib.set_option("mir", mir)
        try:
            assert V(yg).addCGproduct_back1(V(self.g), V(self.x))
        finally:
            self.G._lib.set_option("mir", "auto")
        return yg

    def in_64_bits(self, cells):
        lib, n = self.G._lib.lib(), self.n
        x, g = ([t[:cells].to(torch.complex128) for t in v] for v in (self.x, self.g))
        offs = [0] * len(g)
        yg = [torch.zeros(cells, 2 * l + 1, n, dtype=torch.complex128, device="cuda") for l in range(self.maxl + 1)]
        for l1 in range(self.maxl + 1):
            for l2 in range(self.maxl + 1):
                for l in range(abs(l1 - l2), min(l1 + l2, self.maxl) + 1):
                    for m1 in range(-l1, l1 + 1):
                        lo, hi = max(-l2, -l - m1), min(l2, l - m1)
                        c = torch.tensor([lib.gelib_CGcoefficient(l1, l2, l, m1, m2) for m2 in range(lo, hi + 1)],
                                         dtype=torch.float64, device="cuda")
                        rows = g[l][:, lo + m1 + l:hi + m1 + l + 1, offs[l]:offs[l] + n]
                        yg[l2][:, lo + l2:hi + l2 + 1] += c[None, :, None] * rows * x[l1][:, m1 + l1:m1 + l1 + 1].conj()
                    offs[l] += n
        return yg


def relative_error(got, want):
    num = sum(float((a[:w.size(0)].to(torch.complex128) - w).abs().square().sum()) for a, w in zip(got, want))
    return (num / sum(float(w.abs().square().sum()) for w in want)) ** 0.5


@pytest.mark.parametrize("maxl,n,cols", [(5, 16, 420000), (5, 20, 420000), (6, 20, 130000), (6, 24, 130000), (7, 24, 100000),
                                         (8, 12, 100000), (8, 20, 100000)])
def test_sums_are_no_less_accurate_than_without_the_row_pair_kernel(G, maxl, n, cols):
    # thousands of sums each: the errors' own scatter is under a percent, and 3 % are allowed
    call = Call(G, maxl, n, cols)
    want = call.in_64_bits(200)
    assert relative_error(call.gradient("auto"), want) < 1.03 * relative_error(call.gradient("0"), want)


# every row is summed in one order, so that two runs of one kernel agree bit for bit
@pytest.mark.parametrize("maxl,n,cols,taken", [
    (3, 12, 100000, False), (3, 20, 400000, False), (3, 1, 100000, False), (3, 6, 400000, False), (3, 32, 130000, False),
    (4, 5, 100000, False), (4, 12, 400000, False), (4, 15, 200000, False), (4, 20, 200000, False), (4, 32, 130000, False),
    (5, 8, 200000, False), (5, 12, 200000, False), (5, 20, 200000, False), (6, 9, 200000, False), (6, 15, 200000, False), (6, 20, 130000, False),
    (8, 15, 98000, False), (3, 9, 200000, True), (3, 17, 210000, True), (4, 23, 210000, True), (4, 32, 400000, True), (5, 16, 420000, True),
    (6, 16, 130000, True), (6, 31, 130000, True), (7, 8, 98000, True), (8, 32, 98000, True)])
def test_calls_that_the_row_pair_kernel_takes(G, maxl, n, cols, taken):
    call = Call(G, maxl, n, cols)
    auto, pinned, others = (call.gradient(mir) for mir in ("auto", "one", "0"))
    assert all(torch.equal(a, b) for a, b in zip(auto, pinned if taken else others))
    assert not all(torch.equal(a, b) for a, b in zip(pinned, others))


def test_a_signature_that_it_never_takes_gets_no_plan(G):
    # device memory for a plan cannot be had during capture
    call = Call(G, 3, 40, 100000)
    want = call.gradient("0")
    V = G.backend.SO3vec.view
    yg = [torch.zeros_like(t) for t in call.y]
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        V(yg).addCGproduct_back1(V(call.g), V(call.x))
    graph.replay()
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for a, b in zip(yg, want))
