"""Where trees of small nodes run without or beyond one tiny program: inputs
whose strides its descriptors cannot hold (the nodes then run one by one, as on
a device that cannot place its cluster of sixteen blocks), and more levels than
one launch takes.  Tolerances: the other tree tests'; FP32 and ComplexF32 trees
of eight nodes or more are evaluated in 64 bits and rounded once (5e-8)."""
import numpy as np
import pytest
import torch

import ome_oracle as O
import omeinsum_b200 as ome
from helpers import alg_of, assert_match, gen, to_dev, to_np
from test_gpu_parity import kernel_names
from test_gpu_tiny_programs import oracle_tree

pytestmark = pytest.mark.gpu


def product(n):
    """m0 m1 ... as a tree as deep as it can be."""
    tree = ome.NestedEinsum(0)
    for i in range(1, n):
        tree = ome.NestedEinsum([tree, ome.NestedEinsum(i)], ome.EinCode([(0, i), (i, i + 1)], (0, i + 1)))
    return tree


def matrices(n, e, dt, seed):
    rng = np.random.default_rng(seed)
    xs = [gen(rng, (e, e), dt) for _ in range(n)]
    if dt == "i64":
        return [x % 3 - 1 for x in xs]
    return xs if dt == "trop" else [(x / np.sqrt(e)).astype(x.dtype) for x in xs]


def in_64_bits(tree, xs, dt, sizes):
    if dt in ("f32", "c64"):
        xs = [x.astype(np.float64 if dt == "f32" else np.complex128) for x in xs]
    return O.nested_einsum(oracle_tree(tree), xs, sizes, alg_of(dt))


TOL = {"f32": 5e-8, "c64": 5e-8}


def far(x, dt):
    """x with columns 2^25 elements apart."""
    t = to_dev(x, dt)
    t = t.data if dt == "trop" else t
    y = torch.empty(4 << 25, dtype=t.dtype, device="cuda").as_strided((4, 4), (1, 1 << 25))
    y.copy_(t)
    return ome.TropicalTensor(y) if dt == "trop" else y


@pytest.mark.parametrize("dt", ["f64", "f32", "c64", "i64", "trop"])
def test_strides_beyond_a_program(dt):
    n = 11
    tree, sizes = product(n), {i: 4 for i in range(n + 1)}
    xs = matrices(n, 4, dt, 31)
    want = in_64_bits(tree, xs, dt, sizes)
    near = [to_dev(x, dt) for x in xs]
    got, names = kernel_names(lambda: tree(*near))
    assert "k_tiny" in names, names
    assert_match(to_np(got), want, dt, TOL.get(dt))
    mixed = list(near)
    mixed[6] = far(xs[6], dt)
    got, names = kernel_names(lambda: tree(*mixed))
    assert "k_tiny" not in names, names
    assert_match(to_np(got), want, dt)
    assert_match(to_np(ome.SlicedEinsum([3], tree)(*mixed)), want, dt)
    assert_match(to_np(tree(*near)), want, dt, TOL.get(dt))


@pytest.mark.parametrize("dt", ["f64", "f32", "c64"])
@pytest.mark.parametrize("n,strided", [(11, True), (150, False)])
def test_gradients(dt, n, strided):
    e = 4
    inner = product(n)
    tree = ome.NestedEinsum([inner], ome.EinCode([(0, n)], ()))
    xs = matrices(n, e, dt, 32)
    wide_t = np.complex128 if dt == "c64" else np.float64
    ts = [torch.from_numpy(x.astype(wide_t)).requires_grad_() for x in xs]
    m = ts[0]
    for t in ts[1:]:
        m = m @ t
    m = m.sum()
    (m.real if dt == "c64" else m).backward()
    dev = [to_dev(x, dt) for x in xs]
    if strided:
        dev[6] = far(xs[6], dt)
    y, grads = ome.cost_and_gradient(tree, dev)
    tol = None if strided else TOL.get(dt)
    tol_g = 1e-10 if dt == "f64" and n > 100 else tol   # (150 factors' round-off at a condition of about 1e2)
    assert_match(to_np(y), m.detach().numpy(), dt, tol_g)
    for g, t in zip(grads, ts):
        assert_match(to_np(g), t.grad.numpy(), dt, tol_g)


@pytest.mark.parametrize("dt", ["f32", "c64", "i64", "trop"])
def test_more_levels_than_a_launch(dt):
    """149 levels: three launches of at most 64."""
    n, e = 150, 3
    tree, sizes = product(n), {i: e for i in range(n + 1)}
    xs = matrices(n, e, dt, 33)
    got, names = kernel_names(lambda: tree(*[to_dev(x, dt) for x in xs]))
    assert names.count("k_tiny") >= 3, names
    assert_match(to_np(got), in_64_bits(tree, xs, dt, sizes), dt, TOL.get(dt))


@pytest.mark.parametrize("dt", ["f64", "f32"])
@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
def test_non_finite(dt, value):
    n, e = 12, 3
    tree, sizes = product(n), {i: e for i in range(n + 1)}
    xs = matrices(n, e, dt, 34)
    xs[5][1, 2] = value
    want = in_64_bits(tree, xs, dt, sizes)
    got = to_np(tree(*[to_dev(x, dt) for x in xs])).astype(np.float64)
    assert np.array_equal(np.isnan(got), np.isnan(want)) and np.array_equal(np.isposinf(got), np.isposinf(want)) \
        and np.array_equal(np.isneginf(got), np.isneginf(want))
