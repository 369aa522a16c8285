"""Float32 / ComplexF32 trees between 2^26 and 2^32 multiply-adds: evaluated in
64 bits and rounded once.  Norm-wise 5e-8 (one rounding of every element leaves
2.5e-8 .. 3.5e-8; a rounding at each of the 13 nodes sqrt(13) times that)."""
import numpy as np
import pytest
import torch

import omeinsum_b200 as ome
from omeinsum_b200 import _lib
from omeinsum_b200.plan import get_plan
from helpers import assert_match, gen, to_dev, to_np
from test_gpu_tiny_programs import chain


@pytest.mark.gpu
@pytest.mark.parametrize("dt", ["f32", "c64"])
def test_value_and_gradients(dt):
    rng = np.random.default_rng(8)
    n = 14
    tree, ixs, sizes = chain(n, [240, 250, 255], rng)
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
    dev = [to_dev(x, dt) for x in xs]
    assert_match(to_np(tree(*dev)), v.detach().numpy(), dt, 5e-8)
    got, grads = ome.cost_and_gradient(tree, dev, dy=to_dev(dy, dt))
    assert_match(to_np(got), v.detach().numpy(), dt, 5e-8)
    for g, t in zip(grads, ts):
        assert_match(to_np(g), t.grad.numpy(), dt, 5e-8)


def test_large_buffers_stay_in_float32():
    """A tree whose values would take more than 1 GiB in Float64 keeps the
    workspace of its Float32 plan."""
    size = {i: 2 for i in range(27)}   # nine bond-2 vertices of three legs: their outer product, summed at the end
    acc, lab = ome.NestedEinsum(0), (0, 1, 2)
    for i in range(1, 9):
        leg = (3 * i, 3 * i + 1, 3 * i + 2)
        acc = ome.NestedEinsum([acc, ome.NestedEinsum(i)], ome.EinCode([lab, leg], lab + leg))
        lab = lab + leg
    tree = ome.NestedEinsum([ome.NestedEinsum([acc], ome.EinCode([lab], lab[:2]))], ome.EinCode([lab[:2]], ()))
    p32 = get_plan(tree, size, _lib.F32, 0)
    plain = get_plan(tree, size, _lib.F32, 1)     # (plain Float32: never in Float64)
    assert p32.grad_bytes < 1.2 * plain.grad_bytes


@pytest.mark.gpu
@pytest.mark.parametrize("server", ["TNServer", "NativeTNServer"])
@pytest.mark.parametrize("grad", [False, True])
def test_served_within_a_float32_budget(server, grad):
    """A server whose budget holds the tree's Float32 buffers but not its
    Float64 ones runs the job (in Float32)."""
    rng = np.random.default_rng(9)
    tree, ixs, sd = chain(12, [170], rng)
    tree = ome.NestedEinsum([tree], ome.EinCode([(0,)], ()))
    xs = [gen(rng, [170, 170], "f32") / np.float32(np.sqrt(170)) for _ in ixs]
    plain, full = get_plan(tree, sd, _lib.F32, 1), get_plan(tree, sd, _lib.F32, 0)
    budget = plain.grad_bytes if grad else plain.forward_bytes
    assert budget < (full.grad_bytes if grad else full.forward_bytes)
    srv = getattr(ome, server)(n_slots=1, hbm_budget_bytes=budget)
    job = ome.Job(tree, [to_dev(x, "f32") for x in xs], grad=grad)
    st = srv.run_trace([job])
    srv.close()
    assert st["completed"] == 1, st
    ts = [torch.from_numpy(x.astype(np.float64)).requires_grad_() for x in xs]
    v = torch.diagonal(torch.linalg.multi_dot(ts)).sum()
    assert_match(to_np(job.value), v.detach().numpy(), "f32")
    if grad:
        v.backward()
        for g, t in zip(job.grads, ts):
            assert_match(to_np(g), t.grad.numpy(), "f32")
