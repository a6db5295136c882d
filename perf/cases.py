"""The Clebsch-Gordan workloads that a program on this package runs, at the sizes it runs them.

Every case goes through the public Python API and, where it says "train", through autograd: the pass returns the product
and the gradients for a given upstream gradient.  Families ("kind"):

  part   one SO3part.CGproduct, one (l1,l2)->l term
  vec    SO3vec CGproduct, every term with l <= maxl
  diag   SO3vec DiagCGproduct: channel n pairs with channel n
  cloud  first layer on a point cloud: spherical harmonics of the points, the features mixed by per-l weights, their product
  array  message passing: the SO3vecs of an array of atoms are gathered over a neighbour map and multiplied with the atoms' own

A type is written "l:channels,l:channels,..".  All tensors are complex64 (the points float32).
"""
import math

import torch

import gelib_b200 as gelib


def _uniform(maxl, n, minl=0):
    return ",".join("%d:%d" % (l, n) for l in range(minl, maxl + 1))


def listed():
    return [
        # one product on a handful of objects, no gradients: a call made from a loop, bound by its latency
        dict(name="part_infer_tiny", kind="part", train=False, b=16, l1=1, l2=2, l=2, n1=4, n2=4),
        # one product of two l=2 parts in training, 32 channels: the single-term configuration of the benchmark
        dict(name="part_train", kind="part", train=True, b=1024, l1=2, l2=2, l=2, n1=32, n2=32),
        # a small network on a small batch of molecules: few channels, low l, launches and host work count
        dict(name="vec_train_small", kind="vec", train=True, b=64, x=_uniform(2, 8), y=_uniform(2, 8), maxl=2),
        # the usual layer of an equivariant network: 16 channels, l up to 4
        dict(name="vec_train_mid", kind="vec", train=True, b=1000, x=_uniform(4, 16), y=_uniform(4, 16), maxl=4),
        # a layer whose channel counts fall with l, odd ones among them, on a ragged batch
        dict(name="vec_train_ragged", kind="vec", train=True, b=777, x="0:12,1:9,2:7,3:5", y="0:10,1:7,2:3", maxl=3),
        # one pair of wide parts with every l that it couples to (l = 1..7): the second configuration of the benchmark
        dict(name="vec_train_wide", kind="vec", train=True, b=2048, x="3:64", y="4:64", maxl=-1),
        # the largest layer: l up to 6 with 32 channels each, the headline configuration, a quarter of its batch
        dict(name="vec_train_large", kind="vec", train=True, b=1024, x=_uniform(6, 32), y=_uniform(6, 32), maxl=6),
        # evaluation of a trained layer: the forward product alone, without gradients, on an odd batch
        dict(name="vec_infer", kind="vec", train=False, b=2047, x=_uniform(4, 32), y=_uniform(4, 32), maxl=4),
        # the diagonal product of a wide network: l up to 8, 128 channels
        dict(name="diag_train_large", kind="diag", train=True, b=2048, x=_uniform(8, 128), y=_uniform(8, 128), maxl=8),
        # the diagonal product of a small network: a channel count below a warp and not a power of two
        dict(name="diag_train_small", kind="diag", train=True, b=500, x=_uniform(3, 12), y=_uniform(3, 12), maxl=3),
        # first layer on a point cloud: one harmonic channel against 16 mixed feature channels, gradients of features and weights
        dict(name="cloud_train", kind="cloud", train=True, b=65536, lmax=6, n=16),
        # message passing on a batch of molecules: 29 atoms, a neighbour map with a quarter of the pairs
        dict(name="array_train", kind="array", train=True, b=32, atoms=29, density=0.25, x=_uniform(2, 8), maxl=2),
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    """One more case of a family's range; its batch is cut until it costs no more than the largest listed case."""
    kind = rng.choice(["part", "vec", "vec", "vec", "diag", "diag", "cloud", "array"])
    train = kind == "array" or kind == "cloud" or rng.random() < 0.75
    if kind == "part":
        l1, l2 = rng.randint(0, 6), rng.randint(0, 6)
        case = dict(kind=kind, train=train, b=_log_int(rng, 1, 4096), l1=l1, l2=l2, l=rng.randint(abs(l1 - l2), l1 + l2),
                    n1=_log_int(rng, 1, 64), n2=_log_int(rng, 1, 64))
    elif kind == "vec":
        shape = rng.choice(["uniform", "uniform", "wide", "ragged"])
        if shape == "uniform":
            n = rng.choice([32, 16, _log_int(rng, 2, 64)])
            lx = rng.randint(1, 6)
            case = dict(x=_uniform(lx, n), y=_uniform(lx, n), maxl=lx)
        elif shape == "wide":
            case = dict(x="%d:%d" % (rng.randint(0, 5), 32 * rng.randint(1, 3)), y="%d:%d" % (rng.randint(0, 5), 32 * rng.randint(1, 3)),
                        maxl=-1)
        else:
            lx, ly = rng.randint(1, 5), rng.randint(1, 5)
            case = dict(x=",".join("%d:%d" % (l, rng.randint(1, 40)) for l in range(lx + 1)),
                        y=",".join("%d:%d" % (l, rng.randint(1, 40)) for l in range(ly + 1)), maxl=max(lx, ly))
        case = dict(kind=kind, train=train, shape=shape, b=_log_int(rng, 4, 4096), **case)
    elif kind == "diag":
        n, lx, ly = _log_int(rng, 4, 128), rng.randint(1, 8), rng.randint(1, 8)
        case = dict(kind=kind, train=train, b=_log_int(rng, 16, 4096), x=_uniform(lx, n), y=_uniform(ly, n), maxl=max(lx, ly))
    elif kind == "cloud":
        case = dict(kind=kind, train=train, b=_log_int(rng, 256, 65536), lmax=rng.randint(1, 6), n=_log_int(rng, 4, 32))
    else:
        lx, n = rng.randint(1, 3), _log_int(rng, 2, 32)
        case = dict(kind=kind, train=train, b=_log_int(rng, 1, 64), atoms=rng.randint(3, 40), density=0.25, x=_uniform(lx, n), maxl=lx)
    most = [work(c) for c in listed()]
    share = 0.125 if case.get("shape") == "ragged" else 1.0  # odd channel counts run on the general kernels
    most = {k: share * max(w[k] for w in most) for k in ("bytes", "flops")}
    while case["b"] > 1 and any(work(case)[k] > most[k] for k in most):
        case["b"] = max(1, case["b"] * 2 // 3)
    return case


def _tau(text):
    return {int(p.split(":")[0]): int(p.split(":")[1]) for p in text.split(",")}


def _types(case):
    """(type of x, type of y, maxl, diagonal) of the product in the case."""
    if case["kind"] == "part":
        return {case["l1"]: case["n1"]}, {case["l2"]: case["n2"]}, None, False
    if case["kind"] == "cloud":
        return {l: 1 for l in range(case["lmax"] + 1)}, {l: case["n"] for l in range(case["lmax"] + 1)}, case["lmax"], False
    return _tau(case["x"]), _tau(case["x"] if case["kind"] == "array" else case["y"]), case["maxl"], case["kind"] == "diag"


def _product_type(case):
    tx, ty, maxl, diag = _types(case)
    out = {}
    for l1, n1 in tx.items():
        for l2, n2 in ty.items():
            for l in range(abs(l1 - l2), l1 + l2 + 1):
                if (l == case["l"]) if maxl is None else (maxl == -1 or l <= maxl):
                    out[l] = out.get(l, 0) + (n1 if diag else n1 * n2)
    return dict(sorted(out.items()))


def _crandn(gen, *shape):
    return torch.view_as_complex(torch.randn(*shape, 2, device="cuda", generator=gen))


def prepare(case, seed):
    """Features, weights, maps and the upstream gradient, re and im ~ N(0,1); points on the sphere with radii U(0.5, 2)."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    tx, ty, maxl, _ = _types(case)
    lead = [case["b"], case["atoms"]] if case["kind"] == "array" else [case["b"]]
    part = gelib.SO3partArr if case["kind"] == "array" else gelib.SO3part
    train = case["train"]

    def features(tau):
        return [part(_crandn(gen, *lead, 2 * l + 1, n)).requires_grad_(train) for l, n in tau.items()]

    s = dict(case=case, maxl=maxl, g=None)
    if train:
        s["g"] = [_crandn(gen, *lead, 2 * l + 1, n) for l, n in _product_type(case).items()]
    if case["kind"] == "cloud":
        d = torch.randn(case["b"], 3, 1, device="cuda", generator=gen)
        radius = 0.5 + 1.5 * torch.rand(case["b"], 1, 1, device="cuda", generator=gen)
        s["points"] = (d / d.norm(dim=1, keepdim=True) * radius).contiguous()
        s["y"] = features(ty)
        s["w"] = [(_crandn(gen, n, n) / math.sqrt(n)).requires_grad_(train) for n in ty.values()]
        s["leaves"] = s["y"] + s["w"]
    elif case["kind"] == "array":
        pairs = torch.rand(case["atoms"], case["atoms"], device="cuda", generator=gen) < case["density"]
        s["map"] = gelib.gather_map.from_matrix(pairs, case["atoms"], case["atoms"])
        s["x"] = features(tx)
        s["leaves"] = s["x"]
    else:
        s["x"], s["y"] = features(tx), features(ty)
        s["leaves"] = s["x"] + s["y"]
    return s


def run(state):
    """One forward product, and in training its gradients."""
    case, kind = state["case"], state["case"]["kind"]
    if kind == "part":
        z = gelib.CGproduct(state["x"][0], state["y"][0], case["l"])
        out = [z]
    else:
        if kind == "cloud":
            u = gelib.SO3vec.spharms(case["lmax"], state["points"])
            v = gelib.SO3vec(*state["y"]) * gelib.SO3weights(*state["w"])
            z = gelib.CGproduct(u, v, maxl=state["maxl"])
        elif kind == "array":
            x = gelib.SO3vecArr(*state["x"])
            z = gelib.CGproduct(gelib.gather(x, state["map"]), x, maxl=state["maxl"])
        else:
            x, y = gelib.SO3vec(*state["x"]), gelib.SO3vec(*state["y"])
            z = (gelib.DiagCGproduct if kind == "diag" else gelib.CGproduct)(x, y, maxl=state["maxl"])
        out = list(z.parts.values())
    if not case["train"]:
        return {"product": out}
    return {"product": out, "grads": list(torch.autograd.grad(out, state["leaves"], grad_outputs=state["g"]))}


def work(case):
    """Bytes: features, points, weights and upstream gradient read once, product and gradients written once.  Operations:
    per band entry (m1,m2) of a pair (l1,l2) one complex product of x and y, which every output l shares (8), or two with
    the gradient (16), and one real-by-complex multiply-add per output l (4), for each channel of the output."""
    tx, ty, _, diag = _types(case)
    tr = _product_type(case)
    cells = case["b"] * case.get("atoms", 1)

    def floats(tau):
        return 2 * sum((2 * l + 1) * n for l, n in tau.items())

    terms = pairs = 0
    for l1, n1 in tx.items():
        for l2, n2 in ty.items():
            w = n1 if diag else n1 * n2
            for m1 in range(-l1, l1 + 1):
                for m2 in range(-l2, l2 + 1):
                    k = sum(1 for l in tr if abs(l1 - l2) <= l <= l1 + l2 and l >= abs(m1 + m2))
                    terms += w * k
                    pairs += w * (k > 0)
    small = {"cloud": 3 + floats(ty), "array": floats(tx)}.get(case["kind"], floats(tx) + floats(ty))  # floats read per cell
    grads = {"cloud": floats(ty), "array": floats(tx)}.get(case["kind"], floats(tx) + floats(ty))
    mix = sum((2 * l + 1) * n * n for l, n in ty.items()) if case["kind"] == "cloud" else 0
    flops = cells * (4 * terms + 8 * pairs + 8 * mix)
    total = 4 * cells * (small + floats(tr))
    if case["train"]:
        needed = 8 if case["kind"] == "cloud" else 16  # the harmonics need no gradient
        flops += cells * (4 * terms + needed * pairs + 16 * mix)
        total += 4 * cells * (floats(tr) + grads)
    return {"bytes": total, "flops": flops}


def tolerance(case):
    """Sums in 32 bits.  Against sums in 64 bits the products differ by up to 4e-7 of the result (3e-6 in single values) and
    the gradients by up to 3e-7; two runs that add the weight gradients of 65536 points in another order differ by 7e-7."""
    return {"rel": 4e-6 if case["kind"] == "cloud" else 2e-6, "max": 3e-5}
