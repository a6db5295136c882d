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
