"""Repeated calls on plain CUDA tensors: a code's descriptors are kept by the
layout of its inputs and a tree's by the tree's structure, so that a call with
another layout, other values or a changed tree gives what a first call gives.
Tolerances: helpers' (FP64 1e-12, FP32 1e-5)."""
import numpy as np
import pytest
import torch

import omeinsum_b200 as ome
from helpers import assert_match, gen, oracle, parse, to_np

pytestmark = pytest.mark.gpu


def layouts(x):
    """The same values column-major, row-major, as every second element of a
    larger array, and expanded along the first mode (all rows equal)."""
    t = torch.from_numpy(x).cuda()
    big = torch.zeros([2 * s for s in x.shape], dtype=t.dtype, device="cuda")
    big[tuple(slice(None, None, 2) for _ in x.shape)] = t
    return [torch.from_numpy(np.asfortranarray(x)).cuda(), t.contiguous(),
            big[tuple(slice(None, None, 2) for _ in x.shape)]]


@pytest.mark.parametrize("dt", ["f32", "f64", "c64"])
def test_flat_calls_by_layout(dt):
    rng = np.random.default_rng(1)
    code = "abc,cbd->da"
    ixs, iy = parse(code)
    c = ome.ein(code)
    for sizes in (dict(a=5, b=3, c=4, d=6), dict(a=20, b=9, c=4, d=33), dict(a=5, b=3, c=4, d=6)):
        xs = [gen(rng, [sizes[l] for l in ix], dt) for ix in ixs]
        want = oracle(ixs, iy, xs, sizes, dt)
        for x in layouts(xs[0]):
            for y in layouts(xs[1]):
                assert_match(to_np(c(x, y)), want, dt)
                assert_match(to_np(ome.einsum(c, [x, y])), want, dt)
    with pytest.raises(ome.DimensionMismatch):
        c(torch.zeros(5, 3, 4, device="cuda"), torch.zeros(4, 2, 6, device="cuda"))
    with pytest.raises(ome.ArgumentError):
        c(torch.zeros(5, 3, device="cuda"), torch.zeros(4, 3, 6, device="cuda"))
    e = torch.randn(4, 1, 3, device="cuda").expand(4, 5, 3).permute(1, 2, 0)   # stride 0 along a
    y = torch.randn(4, 3, 6, device="cuda")
    want = np.einsum("abc,cbd->da", e.cpu().double().numpy(), y.cpu().double().numpy())
    assert_match(to_np(c(e, y)), want, "f32")


@pytest.mark.parametrize("sizes", [dict(i=3, j=4, k=5, l=6, m=7), dict(i=20, j=17, k=19, l=23, m=12)])
def test_tree_calls_by_layout_and_structure(sizes):
    """Small inputs are read in place, larger ones copied; a tree whose lists
    were changed between calls is planned again."""
    rng = np.random.default_rng(2)
    tree = ome.ein("(ijk,jkl),klm->im")
    xs = [gen(rng, [sizes[l] for l in ix], "f64") for ix in ("ijk", "jkl", "klm")]
    want = np.einsum("ijk,jkl,klm->im", *xs)
    for k in range(3):
        args = [layouts(x)[(k + i) % 3] for i, x in enumerate(xs)]
        for _ in range(2):
            assert_match(to_np(tree(*args)), want, "f64")
    sliced = ome.SlicedEinsum(["l"], tree)
    for k in range(3):
        assert_match(to_np(sliced(*[layouts(x)[k] for x in xs])), want, "f64")
    sliced.slicing[0] = "j"
    assert_match(to_np(sliced(*[layouts(x)[1] for x in xs])), want, "f64")
    tree.eins = ome.EinCode(tree.eins.ixs, ("m", "i"))
    assert_match(to_np(tree(*[layouts(x)[1] for x in xs])), want.T, "f64")
    assert_match(to_np(sliced(*[layouts(x)[0] for x in xs])), want.T, "f64")


def test_gradient_of_any_layout():
    rng = np.random.default_rng(3)
    tree = ome.ein("(ij,jk),ki->")
    xs = [gen(rng, s, "f64") for s in ((5, 6), (6, 7), (7, 5))]
    grads = [np.einsum("jk,ki->ij", xs[1], xs[2]), np.einsum("ij,ki->jk", xs[0], xs[2]),
             np.einsum("ij,jk->ki", xs[0], xs[1])]
    for k in range(3):
        y, dx = ome.cost_and_gradient(tree, [layouts(x)[k] for x in xs])
        assert_match(to_np(y), np.einsum("ij,jk,ki->", *xs), "f64")
        for g, w in zip(dx, grads):
            assert_match(to_np(g), w, "f64")
