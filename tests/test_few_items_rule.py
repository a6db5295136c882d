"""Forward products of a one-channel x with a handful of items: from 40000 columns on the narrow kernel takes them."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lx,ly,maxl,n", [(1, 1, 1, 16), (1, 1, 2, 20)])
@pytest.mark.parametrize("cols,mirrored", [(62000, False), (36000, True)])
def test_the_narrow_kernel_takes_them(lx, ly, maxl, n, cols, mirrored):
    import gelib_b200 as G
    V, cells = G.backend.SO3vec.view, cols // n
    gen = torch.Generator(device="cuda").manual_seed(n)
    crand = lambda *s: torch.view_as_complex(torch.randn(*s, 2, device="cuda", generator=gen))
    x, y = [crand(cells, 2 * l + 1, 1) for l in range(lx + 1)], [crand(cells, 2 * l + 1, n) for l in range(ly + 1)]
    tau = V(x).get_tau().CGproduct(V(y).get_tau(), maxl).get_parts()

    def product(mir):
        r = [torch.empty(cells, 2 * l + 1, k, dtype=torch.complex64, device="cuda") for l, k in tau.items()]
        G._lib.set_option("mir", mir)
        try:
            assert V(r).addCGproduct(V(x), V(y), overwrite=True)
        finally:
            G._lib.set_option("mir", "auto")
        return r

    # each kernel sums in one order, and the two orders differ
    auto, same, other = product("auto"), product("two" if mirrored else "0"), product("0" if mirrored else "two")
    assert all(torch.equal(a, b) for a, b in zip(auto, same))
    assert not all(torch.equal(a, b) for a, b in zip(auto, other))
