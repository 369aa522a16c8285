"""The tiny programs of contraction trees (one launch for the nodes whose whole
subtree is small): trees of mixed sizes, around the limits of a node's work and
of a launch's nodes, sliced and unsliced, every element type, with gradients.

Tolerances: exact for Int64, Bool and max-plus; helpers' 1e-12 for FP64 and
ComplexF64; FP32 / ComplexF32 within 1e-5 of the same tree in 64 bits."""
import numpy as np
import pytest
import torch

import ome_oracle as O
import omeinsum_b200 as ome
from helpers import alg_of, assert_match, gen, to_np, to_dev

pytestmark = pytest.mark.gpu


def chain(n, ext, rng):
    """A ring of n matrices with extents from `ext`, contracted as a random
    tree, one label of the ring in the output."""
    sizes = {i: int(rng.choice(ext)) for i in range(n)}
    ixs = [(i, (i + 1) % n) for i in range(n)]
    parts = [(ome.NestedEinsum(i), ixs[i], {i}) for i in range(n)]
    while len(parts) > 1:
        k = int(rng.integers(0, len(parts) - 1))
        (a, la, sa), (b, lb, sb) = parts[k], parts[k + 1]
        rest = {l for p in parts[:k] + parts[k + 2:] for l in p[1]} | {0}
        keep = tuple(dict.fromkeys(l for l in (*la, *lb) if l in rest))
        if len(parts) == 2:
            keep = (0,)
        if rng.integers(0, 2):
            keep = keep[::-1]
        parts[k:k + 2] = [(ome.NestedEinsum([a, b], ome.EinCode([la, lb], keep)), keep, sa | sb)]
    return parts[0][0], ixs, sizes


def oracle_tree(ne):
    if ne.isleaf:
        return O.leaf(ne.tensorindex)
    return O.Node(args=[oracle_tree(a) for a in ne.args], ixs=[list(ix) for ix in ne.eins.ixs], iy=list(ne.eins.iy))


@pytest.mark.parametrize("dt", ["f64", "f32", "c128", "c64", "i64", "bool", "trop"])
@pytest.mark.parametrize("n,ext", [(3, [2]), (17, [2, 3]), (40, [1, 2, 5, 16]), (130, [2, 4]), (24, [20, 40, 41])])
def test_ring_of_matrices(n, ext, dt):
    rng = np.random.default_rng(n)
    tree, ixs, sizes = chain(n, ext, rng)
    xs = [gen(rng, [sizes[l] for l in ix], dt) for ix in ixs]
    if dt in ("f64", "f32", "c128", "c64"):
        xs = [x / np.sqrt(x.shape[1]).astype(x.real.dtype) for x in xs]
    if dt == "i64":
        xs = [x % 3 - 1 for x in xs]
    wide = [x.astype(np.float64 if dt == "f32" else np.complex128) if dt in ("f32", "c64") else x for x in xs]
    want = O.nested_einsum(oracle_tree(tree), wide, sizes, alg_of(dt))
    got = tree(*[to_dev(x, dt) for x in xs])
    assert_match(to_np(got), want, dt)
    row = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in xs]
    if dt == "trop":
        row = [ome.TropicalTensor(t) for t in row]
    again = tree(*row)
    assert_match(to_np(again), want, dt)
    sliced = ome.SlicedEinsum([0, n // 2], tree)
    assert_match(to_np(sliced(*row)), want, dt)
    if dt in ("f64", "c128", "i64"):
        y = to_dev(gen(rng, [sizes[0]], dt), dt)
        y0 = to_np(y).copy()
        ome.einsum_(tree, row, y, 2, 3)
        assert_match(to_np(y), 2 * want + 3 * y0, dt)


@pytest.mark.parametrize("n,ext,dt", [(n, ext, dt) for dt in ("f64", "c128", "f32")
                                      for n, ext in ((3, [2]), (17, [2, 3]), (60, [1, 2, 5]), (90, [2, 4]),
                                                     (20, [20, 40, 41]))
                                      if not (dt == "f32" and n == 90)])   # (round-off amplified by 90 factors)
def test_ring_gradients(n, ext, dt):
    """Gradients of every matrix against torch's in 64 bits (torch's complex
    gradient is the conjugate convention that the reference's pullback has)."""
    rng = np.random.default_rng(100 + n)
    tree, ixs, sizes = chain(n, ext, rng)
    xs = [gen(rng, [sizes[l] for l in ix], dt) for ix in ixs]
    xs = [x / np.sqrt(x.shape[1]).astype(x.real.dtype) for x in xs]
    dy = gen(rng, [sizes[0]], dt)
    y, grads = ome.cost_and_gradient(tree, [to_dev(x, dt) for x in xs], dy=to_dev(dy, dt))
    ts = [torch.from_numpy(x.astype(np.float64 if dt == "f32" else x.dtype)).requires_grad_() for x in xs]
    m = torch.eye(sizes[0], dtype=ts[0].dtype)
    for t in ts:
        m = m @ t
    v = torch.diagonal(m)
    v.backward(torch.from_numpy(dy.astype(np.float64 if dt == "f32" else dy.dtype)))
    assert_match(to_np(y), v.detach().numpy(), dt, 1e-10 if dt != "f32" else None)
    for g, t in zip(grads, ts):
        assert_match(to_np(g), t.grad.numpy(), dt, 1e-10 if dt != "f32" else None)


@pytest.mark.parametrize("dt", ["f32", "c64"])
@pytest.mark.parametrize("n,ext", [(9, [2, 3]), (17, [2, 3]), (12, [5, 30])])
def test_float32_trees_in_float64(n, ext, dt):
    """Trees of eight and more Float32 / ComplexF32 nodes are evaluated in
    64 bits and rounded once: norm-wise below 1e-7 (half an ulp is 6e-8), also
    onto old values and for gradients with a cotangent."""
    rng = np.random.default_rng(500 + n)
    tree, ixs, sizes = chain(n, ext, rng)
    wide_t = np.float64 if dt == "f32" else np.complex128
    xs = [gen(rng, [sizes[l] for l in ix], dt) for ix in ixs]
    xs = [x / np.sqrt(x.shape[1]).astype(x.real.dtype) for x in xs]
    ts = [torch.from_numpy(x.astype(wide_t)).requires_grad_() for x in xs]
    m = torch.eye(sizes[0], dtype=ts[0].dtype)
    for t in ts:
        m = m @ t
    v = torch.diagonal(m)
    dy = gen(rng, [sizes[0]], dt)
    v.backward(torch.from_numpy(dy.astype(wide_t)))
    want = v.detach().numpy()
    dev = [to_dev(x, dt) for x in xs]
    assert_match(to_np(tree(*dev)), want, dt, 1e-7)
    y0 = gen(rng, [sizes[0]], dt)
    y = to_dev(y0, dt)
    ome.einsum_(tree, dev, y, 2, 3)
    assert_match(to_np(y), 2 * want + 3 * y0.astype(wide_t), dt, 3e-7)
    got, grads = ome.cost_and_gradient(tree, dev, dy=to_dev(dy, dt))
    assert_match(to_np(got), want, dt, 1e-7)
    for g, t in zip(grads, ts):
        assert_match(to_np(g), t.grad.numpy(), dt, 1e-7)
