"""The channel-mixing kernels at the edges of their tiles -- odd channel counts on either side, 1, 2 and 64 channels, rows that
do not fill a tile, inputs on 8-byte boundaries -- against float64, within the rounding of their float32 sums."""
import pytest
import torch

pytestmark = pytest.mark.gpu

SIZES = [(1, 1, 1), (3, 2, 64), (1025, 64, 2), (259, 63, 33), (67, 17, 16), (513, 16, 16), (4097, 4, 5), (100, 64, 64), (33, 31, 32), (7, 1, 64)]


@pytest.mark.parametrize("aligned", [True, False])
@pytest.mark.parametrize("rows,n_in,n_out", SIZES)
def test_edges(rows, n_in, n_out, aligned):
    from gelib_b200 import backend
    gen = torch.Generator().manual_seed(rows + n_in)

    def make(*shape):
        n = torch.Size(shape).numel()
        t = torch.view_as_complex(torch.randn(n + 1, 2, generator=gen)).cuda()
        return (t[:-1] if aligned else t[1:]).view(shape)

    x, g, w = make(rows, n_in), make(rows, n_out), make(n_in, n_out)
    d = lambda t: t.to(torch.complex128)
    # a complex sum of k products in float32 errs by at most about (2 k + 2) 2^-24 of the sum of the products' absolute values
    for got, a, b in ((backend.mix(x, w), d(x), d(w)), (backend.mix(g, w, adjoint=True), d(g), d(w).conj().T),
                      (backend.mix_back_w(x, g, n_in, n_out), d(x).conj().T, d(g))):
        bound = (2 * a.size(1) + 2) * 2.0 ** -24 * 2 * (a.abs() @ b.abs())
        assert ((d(got) - a @ b).abs() <= bound).all()
