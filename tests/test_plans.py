"""A product's plans do not depend on the batch: once a signature has run at one batch size, a call at any other builds and
uploads nothing, so it can be captured in a CUDA graph (device memory cannot be allocated there)."""
import pytest
import torch

from util import crandn

pytestmark = pytest.mark.gpu

U = lambda ls, n: {l: n for l in ls}


@pytest.fixture(scope="module")
def G():
    import gelib_b200
    assert torch.cuda.is_available(), "these tests need a CUDA device"
    gelib_b200._lib.lib()
    return gelib_b200


# types that no other test uses, so that the first call here is the first of the signature; batches on both sides of the
# lines at which the lane layout, the number of runs or the kernel changes
CASES = [
    (False, U((0, 2, 3), 15), U((0, 2, 3), 14), 3, (2, 2500)),
    (False, U((0, 2, 3), 14), U((0, 2, 3), 15), 3, (2500, 2)),
    (False, U((1, 2), 7), U((0, 1, 2), 7), 2, (4, 3000)),
    (False, {0: 11, 2: 9}, {0: 7, 1: 3}, 2, (1500, 3)),
    (True, U((0, 2, 3), 11), U((1, 2, 3), 11), 3, (4000, 4)),
    (True, U((0, 2, 3), 13), U((1, 2, 3), 13), 3, (4, 4000)),
    (True, U((2, 6), 18), U((2, 6), 18), 6, (3, 2400)),
    (False, U((0, 2, 6), 1), U((0, 2, 6), 14), 6, (5, 12000)),
    (False, U((0, 3, 6), 1), U((0, 3, 6), 14), 6, (12000, 5)),
    (False, U((0, 3, 6), 1), U((0, 3, 6), 31), 6, (5, 6000)),
]


@pytest.mark.parametrize("diag,tx,ty,maxl,batches", CASES)
def test_a_signature_is_captured_at_another_batch_than_it_was_warmed_up_at(G, oracle, diag, tx, ty, maxl, batches):
    V = G.backend.SO3vec
    tr = oracle.cg_type(tx, ty, maxl, diag)
    both = diag or min(tx.values()) > 1

    def buffers(B):
        mk = lambda seed, tau: [crandn(seed + l, B, 2 * l + 1, n).cuda() for l, n in tau.items()]
        x, y, g = mk(1, tx), mk(50, ty), mk(100, tr)
        return x, y, g, [torch.empty_like(t) for t in g], [torch.zeros_like(t) for t in x], [torch.zeros_like(t) for t in y]

    def step(x, y, g, r, xg, yg):
        for t in xg + yg:
            t.zero_()
        vx, vy, vg, vr, vxg, vyg = (V.view(p) for p in (x, y, g, r, xg, yg))
        if diag:
            vr.addDiagCGproduct(vx, vy, overwrite=True)
            V.addDiagCGproduct_back01(vxg, vyg, vg, vx, vy)
        else:
            vr.addCGproduct(vx, vy, overwrite=True)
            if both:
                V.addCGproduct_back01(vxg, vyg, vg, vx, vy)
            else:
                vyg.addCGproduct_back1(vg, vx)
        return r + yg + (xg if both else [])

    warm, other = batches
    step(*buffers(warm))
    b = buffers(other)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = step(*b)
    graph.replay()
    torch.cuda.synchronize()
    got = [t.clone() for t in out]
    want = step(*b)
    torch.cuda.synchronize()
    for a, w in zip(got, want):
        assert float((a - w).abs().max()) <= 1e-5 * float(w.abs().max())  # gradients summed with atomics: not bitwise
