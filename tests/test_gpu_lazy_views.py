"""Tensors whose conjugate or negative torch has not carried out yet (their
memory holds the other value): conj(), and the imaginary part of a conjugate."""
import pytest
import torch

import omeinsum_b200 as ome

pytestmark = pytest.mark.gpu


def chain():
    return ome.ein("(ij,jk),kl->il")


def inputs(dtype):
    g = torch.Generator(device="cuda").manual_seed(4)
    xs = [torch.randn(5, 5, dtype=torch.complex128, generator=g, device="cuda").conj() for _ in range(3)]
    return xs if dtype.is_complex else [x.imag for x in xs]


@pytest.mark.parametrize("dtype", [torch.complex128, torch.float64])
def test_values(dtype):
    xs = inputs(dtype)
    assert all(x.is_conj() or x.is_neg() for x in xs)
    cp = [x.clone().resolve_conj().resolve_neg() for x in xs]
    want = cp[0] @ cp[1] @ cp[2]
    for got in (chain()(*xs), ome.SlicedEinsum(["j"], chain())(*xs), ome.ein("ij,jk,kl->il")(*xs),
                ome.ein("ij,jk->ik")(ome.ein("ij,jk->ik")(xs[0], xs[1]), xs[2])):
        torch.testing.assert_close(got, want, rtol=1e-12, atol=1e-12)


@pytest.mark.parametrize("dtype", [torch.complex128, torch.float64])
def test_gradients(dtype):
    xs = inputs(dtype)
    dy = xs[0].clone().resolve_conj().resolve_neg().conj() if dtype.is_complex else inputs(dtype)[0].contiguous()
    y, grads = ome.cost_and_gradient(chain(), xs, dy=dy)
    cp = [x.clone().resolve_conj().resolve_neg().requires_grad_() for x in xs]
    want = cp[0] @ cp[1] @ cp[2]
    want.backward(dy.clone().resolve_conj().resolve_neg())
    torch.testing.assert_close(y, want.detach(), rtol=1e-12, atol=1e-12)
    for a, c in zip(grads, cp):
        torch.testing.assert_close(a, c.grad, rtol=1e-12, atol=1e-12)
    scalar = ome.ein("(ij,jk),ki->")
    y, grads = ome.cost_and_gradient(scalar, xs)
    cp = [x.clone().resolve_conj().resolve_neg().requires_grad_() for x in xs]
    want = torch.trace(cp[0] @ cp[1] @ cp[2])
    (want.real if dtype.is_complex else want).backward()
    torch.testing.assert_close(y, want.detach(), rtol=1e-12, atol=1e-12)
    for a, c in zip(grads, cp):
        torch.testing.assert_close(a, c.grad, rtol=1e-12, atol=1e-12)
