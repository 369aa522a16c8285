"""What the performance of this framework is measured on.

Each case is work that a program gives the framework through its public entry
points: a code called on CUDA tensors (``code(*xs)``), a contraction tree
(``NestedEinsum`` / ``SlicedEinsum``), ``cost_and_gradient`` or
``BatchedEinsum``.  A case is a dict of plain values:

* kind "flat": one contraction ``code`` of one or two tensors with the extents
  ``sizes`` ("a=48,b=48"), element type ``dtype`` and memory order ``order``
  ("col": column-major, as a Julia array; "row": as torch makes them);
* kind "nested": ein"(ijk,jkl),klm->im" with every extent ``d``;
* kind "network": a random 3-regular graph of ``n`` vertices (graph seed
  ``graph``), one bond-2 tensor per vertex, ``open`` vertices with a free leg
  in the output; greedy order, sliced to 2^``slice`` elements (0: unsliced);
  ``grad``: cost_and_gradient instead of the value;
* kind "mps": ``njobs`` transfer contractions (ab,bcd),de->ace of uneven bond
  dimensions, multiples of ``step``, as two grouped launches.
"""
import importlib.util
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _package():
    if "omeinsum_b200" not in sys.modules:
        pkg = os.path.join(ROOT, "omeinsum.jl_b200")
        spec = importlib.util.spec_from_file_location("omeinsum_b200", os.path.join(pkg, "__init__.py"),
                                                      submodule_search_locations=[pkg])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["omeinsum_b200"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["omeinsum_b200"]


ome = _package()

DTYPES = {"f32": torch.float32, "f64": torch.float64, "c32": torch.complex64, "c64": torch.complex128,
          "i64": torch.int64, "trop": torch.float32}
WIDE = {"f32": torch.float64, "f64": torch.float64, "c32": torch.complex128, "c64": torch.complex128,
        "i64": torch.float64, "trop": torch.float64}
FLOPS_PER_MAC = {"f32": 2, "f64": 2, "c32": 8, "c64": 8, "i64": 2, "trop": 2}


def listed():
    return [
        # the smallest whole call: a two-step tree on tensors of a few KB (launches and host path)
        {"name": "nested_small", "kind": "nested", "d": 16},
        # the dense four-leg contraction of the rule suite: a 2304^3 GEMM
        {"name": "gemm_f32", "kind": "flat", "code": "abcd,cdef->abef", "dtype": "f32", "order": "col",
         "sizes": "a=48,b=48,c=48,d=48,e=48,f=48"},
        # the same on extents that divide nothing and rows that start on 4 bytes (1369 x 1369 x 1369)
        {"name": "gemm_f32_odd", "kind": "flat", "code": "abcd,cdef->abef", "dtype": "f32", "order": "col",
         "sizes": "a=37,b=37,c=37,d=37,e=37,f=37"},
        # batched matrix product in Julia's layout, the batch mode innermost
        {"name": "batched_f32", "kind": "flat", "code": "bij,bjk->bik", "dtype": "f32", "order": "col",
         "sizes": "b=512,i=64,j=64,k=64"},
        # ComplexF32, the element type of quantum circuits, in torch's row-major order
        {"name": "gemm_c32", "kind": "flat", "code": "abcd,cdef->abef", "dtype": "c32", "order": "row",
         "sizes": "a=32,b=32,c=32,d=32,e=32,f=32"},
        # Float64, Julia's default element type, on odd extents (1681 x 1681 x 1681)
        {"name": "gemm_f64_odd", "kind": "flat", "code": "abcd,cdef->abef", "dtype": "f64", "order": "col",
         "sizes": "a=41,b=41,c=41,d=41,e=41,f=41"},
        # Int64 counting: the rule suite's long-K contraction, exact
        {"name": "gemm_i64", "kind": "flat", "code": "ijk,jkl->il", "dtype": "i64", "order": "col",
         "sizes": "i=256,j=256,k=256,l=256"},
        # a five-mode permutation on odd extents (160 MB each way)
        {"name": "permute_odd", "kind": "flat", "code": "abcde->ecadb", "dtype": "f32", "order": "col",
         "sizes": "a=31,b=33,c=29,d=35,e=39"},
        # the value of a sliced network: a 3-regular graph with a few open legs
        {"name": "network_f32", "kind": "network", "dtype": "f32", "n": 160, "graph": 2, "open": 4, "slice": 26,
         "grad": False},
        # the ground-state energy of a spin glass on a 3-regular graph (max-plus)
        {"name": "network_trop", "kind": "network", "dtype": "trop", "n": 120, "graph": 3, "open": 0, "slice": 0,
         "grad": False},
        # one optimisation step: value and gradients of a network with every vertex tensor a parameter
        {"name": "network_grad", "kind": "network", "dtype": "f32", "n": 100, "graph": 2, "open": 0, "slice": 0,
         "grad": True},
        # a DMRG-style sweep over many sites at once: uneven ComplexF32 transfers, grouped
        {"name": "mps_c32", "kind": "mps", "njobs": 2048, "step": 8, "shapes": 9},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["gemm", "gemm", "batched", "unary", "nested", "network", "network", "mps"])
    if kind == "nested":
        return {"kind": "nested", "d": _log(rng, 4, 64)}
    if kind == "mps":
        return {"kind": "mps", "njobs": _log(rng, 64, 4096), "step": rng.choice([1, 4, 8]),
                "shapes": rng.randrange(1000)}
    if kind == "network":
        dtype = rng.choice(["f32", "f32", "f64", "trop", "c32"])
        grad = dtype != "trop" and rng.random() < 0.4
        cut = 0 if grad else rng.choice([0, 16, 20])
        return {"kind": "network", "dtype": dtype, "n": 2 * rng.randint(20, 60), "graph": rng.randrange(1000),
                "open": 0 if grad else rng.randint(0, 4), "slice": cut, "grad": grad}
    order = rng.choice(["col", "col", "row"])
    if kind == "unary":
        code = rng.choice(["abcde->ecadb", "ijk->kji", "ijk->j", "ijk->ik", "ij->j", "ii->", "ii->i"])
        dtype = rng.choice(["f32", "f32", "f64", "c32", "i64"])
        labels = sorted(set(code) - set(",->"))
        total = _log(rng, 1 << 12, 1 << 26)
        if code.startswith("ii"):
            return {"kind": "flat", "code": code, "dtype": dtype, "order": order, "sizes": "i=%d" % _log(rng, 64, 8192)}
        cuts = [rng.uniform(0.6, 1.4) for _ in labels]
        ext = [max(2, int(round(total ** (c / sum(cuts))))) for c in cuts]
        return {"kind": "flat", "code": code, "dtype": dtype, "order": order,
                "sizes": ",".join("%s=%d" % p for p in zip(labels, ext))}
    if kind == "batched":
        dtype = rng.choice(["f32", "f32", "f64", "c32"])
        ext = {"b": _log(rng, 32, 2048), "i": _log(rng, 8, 128), "j": _log(rng, 8, 128), "k": _log(rng, 8, 128)}
        return {"kind": "flat", "code": "bij,bjk->bik", "dtype": dtype, "order": order,
                "sizes": ",".join("%s=%d" % p for p in ext.items())}
    code = rng.choice(["abcd,cdef->abef", "ij,jk->ki", "ijk,jkl->il", "iaj,jbk->iabk"])
    dtype = rng.choice(["f32", "f32", "f32", "f64", "c32", "c64", "i64", "trop"])
    labels = sorted(set(code) - set(",->"))
    macs = _log(rng, 1 << 15, (1 << 34) if dtype == "f32" else (1 << 32))
    cuts = [rng.uniform(0.6, 1.4) for _ in labels]
    ext = [max(3, int(round(macs ** (c / sum(cuts))))) for c in cuts]
    if rng.random() < 0.4:   # half of real extents are round
        ext = [max(4, 4 * (e // 4)) for e in ext]
    return {"kind": "flat", "code": code, "dtype": dtype, "order": order,
            "sizes": ",".join("%s=%d" % p for p in zip(labels, ext))}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------


def _sizes(case):
    return {k: int(v) for k, v in (p.split("=") for p in case["sizes"].split(","))}


def _values(shape, dtype, order, g, dev):
    """normal(0,1) values (integers in [-8, 8] for i64) of the given shape and memory order."""
    mem = tuple(shape)[::-1] if order == "col" else tuple(shape)
    if dtype == "i64":
        x = torch.randint(-8, 9, mem, generator=g, device=dev, dtype=torch.int64)
    else:
        x = torch.randn(mem, generator=g, device=dev, dtype=DTYPES[dtype])
        if dtype in ("c32", "c64"):
            x = x * math.sqrt(2.0)
    return x.permute(*range(len(mem) - 1, -1, -1)) if order == "col" else x


def _parse(code):
    lhs, iy = code.split("->")
    return lhs.split(","), iy


def _graph(n, seed):
    """Edges of a random 3-regular graph (pairing model, resampled until simple)."""
    rng = np.random.default_rng(seed)
    while True:
        pairs = rng.permutation(np.repeat(np.arange(n), 3)).reshape(-1, 2)
        pairs = np.sort(pairs, axis=1)
        if np.all(pairs[:, 0] != pairs[:, 1]) and len(np.unique(pairs, axis=0)) == len(pairs):
            return [tuple(map(int, p)) for p in pairs]


_TREES = {}


def _network(case):
    """(contraction tree or sliced tree, labels per vertex, output labels): the order search is done once per
    network, as a program that contracts it again and again does."""
    key = tuple(case[k] for k in ("n", "graph", "open", "slice"))
    if key not in _TREES:
        n, nopen = case["n"], case["open"]
        edges = _graph(n, case["graph"])
        inc = [[] for _ in range(n)]
        for i, (a, b) in enumerate(edges):
            inc[a].append(i)
            inc[b].append(i)
        out = []
        for v in range(nopen):
            inc[v * (n // max(nopen, 1))].append(len(edges) + v)
            out.append(len(edges) + v)
        sd = {i: 2 for i in range(len(edges) + nopen)}
        tree = ome.optimize_code(ome.EinCode([tuple(v) for v in inc], tuple(out)), sd,
                                 ome.GreedyMethod(nrepeat=10, seed=case["graph"]))
        code = tree
        if case["slice"]:
            code = ome.slice_code(tree, sd, ome.GreedySlicer(sc_target=case["slice"]))
        _TREES[key] = (tree, code, inc, out, sd)
    return _TREES[key]


def _network_values(case, inc, g, dev):
    dtype = case["dtype"]
    if dtype == "trop":   # +-1 couplings spread over the vertices: energies are whole numbers
        return [torch.randint(0, 2, (2,) * len(v), generator=g, device=dev).mul(2).sub(1).to(torch.float32)
                for v in inc]
    return [torch.randn((2,) * len(v), generator=g, device=dev, dtype=DTYPES[dtype]) *
            (math.sqrt(2.0 / 3.0) if dtype == "c32" else 1 / math.sqrt(3.0)) for v in inc]


def _mps_shapes(case):
    rng = np.random.default_rng(case["shapes"])
    step, top = case["step"], 128 // case["step"]
    lo = 8 // step
    return [(*(int(step * rng.integers(max(lo, 1), top + 1)) for _ in range(4)), int(rng.choice([2, 4])))
            for _ in range(case["njobs"])]


def _flat_views(shapes, dev, g=None):
    """Column-major complex64 tensors of the given shapes in one buffer, each on a 256-byte boundary."""
    offs, n = [], 0
    for s in shapes:
        offs.append(n)
        n += -(-int(np.prod(s)) // 32) * 32
    flat = torch.zeros(n, dtype=torch.complex64, device=dev)
    if g is not None:
        flat.copy_(torch.randn(n, dtype=torch.complex64, device=dev, generator=g)).mul_(math.sqrt(2.0))
    views = []
    for s, o in zip(shapes, offs):
        st = [int(np.prod(s[:d])) for d in range(len(s))]
        views.append(torch.as_strided(flat, s, st, o))
    return flat, views


def _inputs(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    g = torch.Generator(device=dev).manual_seed(seed)
    if case["kind"] == "nested":
        return [torch.rand((case["d"],) * 3, generator=g, device=dev).permute(2, 1, 0) for _ in range(3)]
    if case["kind"] == "flat":
        sd = _sizes(case)
        return [_values([sd[l] for l in ix], case["dtype"], case["order"], g, dev) for ix in _parse(case["code"])[0]]
    if case["kind"] == "network":
        return _network_values(case, _network(case)[2], g, dev)
    shapes = _mps_shapes(case)
    return [_flat_views(s, dev, g)[1] for s in ([(a, b) for a, b, d, e, c in shapes],
                                                [(b, c, d) for a, b, d, e, c in shapes],
                                                [(d, e) for a, b, d, e, c in shapes])]


def prepare(case, seed):
    xs = _inputs(case, seed)
    kind = case["kind"]
    if kind == "nested":
        return {"call": ome.ein("(ijk,jkl),klm->im"), "xs": xs}
    if kind == "flat":
        if case["dtype"] == "trop":
            xs = [ome.TropicalTensor(x) for x in xs]
        return {"call": ome.ein(case["code"]), "xs": xs}
    if kind == "network":
        if case["dtype"] == "trop":
            xs = [ome.TropicalTensor(x) for x in xs]
        return {"call": _network(case)[1], "xs": xs, "grad": case["grad"]}
    shapes = _mps_shapes(case)
    dev = xs[0][0].device
    _, mids = _flat_views([(a, c, d) for a, b, d, e, c in shapes], dev)
    flat, outs = _flat_views([(a, c, e) for a, b, d, e, c in shapes], dev)
    first = ome.BatchedEinsum(ome.ein("ab,bcd->acd"), list(zip(xs[0], xs[1])), mids)
    second = ome.BatchedEinsum(ome.ein("acd,de->ace"), list(zip(mids, xs[2])), outs)
    return {"batches": [first, second], "out": flat}


def run(state):
    if "batches" in state:
        for b in state["batches"]:
            b.run()
        return state["out"]
    if state.get("grad"):
        cost, grads = ome.cost_and_gradient(state["call"], state["xs"])
        return [cost, torch.stack(grads)]
    y = state["call"](*state["xs"])
    return y.data if isinstance(y, ome.TropicalTensor) else y


# ---------------------------------------------------------------------------
# what a pass cannot do without, and its value in 64 bits
# ---------------------------------------------------------------------------


def work(case):
    kind = case["kind"]
    if kind == "nested":
        d = case["d"]
        return {"bytes": 4 * (3 * d ** 3 + d * d), "flops": 2 * (d ** 4 + d ** 4)}
    if kind == "flat":
        sd = _sizes(case)
        ixs, iy = _parse(case["code"])
        es = torch.empty((), dtype=DTYPES[case["dtype"]]).element_size()
        elems = sum(math.prod(sd[l] for l in set(ix)) for ix in ixs) + math.prod(sd[l] for l in iy)
        labels = set("".join(ixs)) | set(iy)
        macs = math.prod(sd[l] for l in labels) if len(ixs) > 1 else 0
        return {"bytes": es * elems, "flops": FLOPS_PER_MAC[case["dtype"]] * macs}
    if kind == "network":
        _, code, inc, out, sd = _network(case)
        es = torch.empty((), dtype=DTYPES[case["dtype"]]).element_size()
        times = 3 if case["grad"] else 1
        nbytes = es * (times - 1 if case["grad"] else 1) * sum(2 ** len(v) for v in inc) + es * 2 ** len(out)
        return {"bytes": nbytes,
                "flops": times * FLOPS_PER_MAC[case["dtype"]] * 2.0 ** ome.contraction_complexity(code, sd).tc}
    shapes = _mps_shapes(case)
    return {"bytes": 8 * sum(a * b + b * c * d + d * e + a * c * e for a, b, d, e, c in shapes),
            "flops": 8 * sum(a * b * c * d + a * c * d * e for a, b, d, e, c in shapes)}


def _maxplus(ixs, xs, iy):
    """max over the summed labels of the sum of the inputs, in pieces of at most 2^27 elements."""
    labels = list(iy) + sorted({l for ix in ixs for l in ix} - set(iy))
    ext = {l: e for ix, x in zip(ixs, xs) for l, e in zip(ix, x.shape)}
    total = math.prod(ext[l] for l in labels)
    if total > 1 << 27:   # cut the largest label in two
        l = max(labels, key=lambda q: ext[q])
        half = ext[l] // 2
        parts = [_maxplus(ixs, [x.narrow(ix.index(l), s, c) if l in ix else x for ix, x in zip(ixs, xs)], iy)
                 for s, c in ((0, half), (half, ext[l] - half))]
        return torch.cat(parts, dim=iy.index(l)) if l in iy else torch.maximum(*parts)
    full = 0.0
    for ix, x in zip(ixs, xs):
        have = [l for l in labels if l in ix]
        x = x.permute([ix.index(l) for l in have])
        full = full + x.reshape([ext[l] if l in ix else 1 for l in labels])
    full = full.expand([ext[l] for l in labels])
    return full.reshape([ext[l] for l in iy] + [-1]).amax(-1) if len(labels) > len(iy) else full


def _contract(ixs, xs, iy, tropical):
    ixs, iy = [list(ix) for ix in ixs], list(iy)
    if tropical:
        return _maxplus(ixs, xs, iy)
    ids = {}
    for l in [l for ix in ixs for l in ix] + iy:
        ids.setdefault(l, len(ids))
    args = [a for ix, x in zip(ixs, xs) for a in (x, [ids[l] for l in ix])]
    return torch.einsum(*args, [ids[l] for l in iy])


def _tree_value(node, xs, tropical):
    if node.isleaf:
        return xs[node.tensorindex]
    return _contract(node.eins.ixs, [_tree_value(a, xs, tropical) for a in node.args], node.eins.iy, tropical)


def exact(case, seed):
    kind = case["kind"]
    xs = _inputs(case, seed)
    if kind == "nested":
        i, j, k = (x.double() for x in xs)
        return torch.einsum("ijk,jkl,klm->im", i, j, k)
    if kind == "mps":
        shapes = _mps_shapes(case)
        dev = xs[0][0].device
        flat, outs = _flat_views([(a, c, e) for a, b, d, e, c in shapes], dev)
        flat = flat.to(torch.complex128)
        pos = 0
        for x1, x2, x3, o in zip(*xs, outs):
            v = torch.einsum("ab,bcd,de->eca", *(x.to(torch.complex128) for x in (x1, x2, x3)))
            flat[pos:pos + v.numel()] = v.reshape(-1)
            pos += -(-v.numel() // 32) * 32
        return flat
    dtype = case["dtype"]
    wide = [x.to(WIDE[dtype]) for x in xs]
    if kind == "flat":
        ixs, iy = _parse(case["code"])
        if case["code"] == "ii->":
            v = torch.diagonal(wide[0]).sum()
        elif case["code"] == "ii->i":
            v = torch.diagonal(wide[0]).clone()
        else:
            v = _contract(ixs, wide, iy, dtype == "trop")
        return v.round().to(torch.int64) if dtype == "i64" else v   # whole sums below 2^53
    tree = _network(case)[0]
    if ome.contraction_complexity(tree, _network(case)[4]).sc > 31:
        return None
    if case["grad"]:
        wide = [x.requires_grad_() for x in wide]
        cost = _tree_value(tree, wide, False)
        cost.backward(torch.ones_like(cost))
        return [cost.detach(), torch.stack([x.grad for x in wide])]
    return _tree_value(tree, wide, dtype == "trop")
