"""What the native host side does with arguments that are not plain: it leaves them to the Python code."""
import sys

import pytest
import torch


def vec(G, device, n):
    gen = torch.Generator().manual_seed(n)
    return G.SO3vec(*[torch.randn(3, 2 * l + 1, n, dtype=torch.complex64, generator=gen).to(device) for l in (0, 1, 2)])


def test_numbers_that_are_no_32_bit_ints_are_declined(cabi):
    from gelib_b200 import _lib
    x = [torch.zeros(2, 3, 1, dtype=torch.complex64)]
    for maxl in (sys.maxsize, 2 ** 40, -2 ** 70, True, 1.0, None):
        assert _lib.native().vec_forward(x, x, maxl, False) is None
        assert _lib.native().part_forward(x[0], x[0], maxl, False) is None


def test_a_maxl_beyond_32_bits_gets_as_far_as_the_device_check(cabi):
    import gelib_b200 as G
    with pytest.raises(RuntimeError, match="CUDA"):
        vec(G, "cpu", 2).CGproduct(vec(G, "cpu", 3), sys.maxsize)


@pytest.mark.gpu
def test_maxl_of_sys_maxsize_keeps_every_l():
    import gelib_b200 as G
    x, y = vec(G, "cuda", 2), vec(G, "cuda", 3)
    want, got = x.CGproduct(y), x.CGproduct(y, sys.maxsize)
    assert list(got.parts) == list(want.parts) == [0, 1, 2, 3, 4]
    for l, p in want.parts.items():
        assert torch.equal(p, got.parts[l])
