"""The mixing kernels over several tiles per block, on both sides of the lines where their tiles change, and the accuracy of their
sums, against 64 bits on the device."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def gb():
    import gelib_b200
    assert torch.cuda.is_available(), "these tests need a CUDA device"
    gelib_b200._lib.lib()
    return gelib_b200.backend


def crand(seed, *shape):
    return torch.view_as_complex(torch.randn(*shape, 2, device="cuda", generator=torch.Generator(device="cuda").manual_seed(seed)))


def relative_error(got, want):
    return float((got.to(want.dtype) - want).abs().square().sum().sqrt() / want.abs().square().sum().sqrt())


def wide(t):
    return t.to(torch.complex128)


def test_wide_weight_gradients_are_as_accurate_as_narrow_ones(gb):
    # more than 32 x 32 channels leave fewer groups of rows to a block, and a thread more rows to add up; the blocks' own sums, in
    # varying order, are common to both
    def error(n):
        x, g = crand(1, 400000, n), crand(2, 400000, n)
        return relative_error(gb.mix_back_w(x, g, n, n), wide(x).conj().T @ wide(g))

    narrow = error(32)
    assert error(48) < 1.15 * narrow and error(64) < 1.15 * narrow


# several tiles and a partial last one for every block; few rows, and both sides of the lines
SIZES = [(200003, 16, 16), (40001, 64, 64), (310007, 8, 8), (80021, 32, 32), (70001, 16, 32), (70001, 32, 16), (300011, 5, 3), (150001, 33, 31),
         (1, 7, 9), (295, 5, 3), (297, 32, 4), (9999, 5, 3), (10000, 16, 8), (10001, 16, 8), (10001, 64, 2), (30011, 3, 5), (9473, 12, 20)]


@pytest.mark.parametrize("aligned", [True, False])
@pytest.mark.parametrize("rows,n_in,n_out", SIZES)
def test_several_tiles_per_block(gb, rows, n_in, n_out, aligned):
    off = 0 if aligned else 1  # eight bytes off a 16-byte boundary

    def operand(seed, n):
        return crand(seed, rows * n + off)[off:].view(rows, n)

    x, w, g = operand(1, n_in), crand(2, n_in, n_out), operand(3, n_out)
    # an element's error is at most the number of its roundings, 2 n + 1, times half an ulp of the terms' absolute sum
    for got, a, b in ((gb.mix(x, w), wide(x), wide(w)), (gb.mix(g, w, adjoint=True), wide(g), wide(w).conj().T)):
        bound = (2 * a.size(1) + 1) * 2.0 ** -24 * 2 ** 0.5 * (a.abs() @ b.abs())
        assert bool(((wide(got) - a @ b).abs() <= bound).all())
    # a tile left out or taken twice shows by more than a percent; sums of 32-bit numbers in random order by some 1e-6
    assert relative_error(gb.mix_back_w(x, g, n_in, n_out), wide(x).conj().T @ wide(g)) < 1e-5


def test_two_channels_are_summed_in_one_chain(gb):
    # fma in double rounded to float: the chain of four multiply-adds, and two halves of two added at the end
    x, w = crand(1, 200000, 2), crand(2, 2, 16)
    a, b = torch.view_as_real(x).double(), torch.view_as_real(w).double()

    def fma(p, q, s):
        return (p * q + s).float().double()

    def mac(re, im, k):
        xr, xi, wr, wi = a[:, k, None, 0], a[:, k, None, 1], b[k, :, 0], b[k, :, 1]
        return fma(-xi, wi, fma(xr, wr, re)), fma(xi, wr, fma(xr, wi, im))

    zero = torch.zeros(200000, 16, dtype=torch.float64, device="cuda")
    first = mac(zero, zero, 0)
    chain = torch.complex(*mac(*first, 1))
    second = mac(zero, zero, 1)
    halves = torch.complex((first[0] + second[0]).float().double(), (first[1] + second[1]).float().double())
    want = wide(x) @ wide(w)
    assert relative_error(chain, want) < relative_error(halves, want)
    assert relative_error(gb.mix(x, w), want) < 1.01 * relative_error(chain, want)
