"""What repeated calls keep of contraction trees: nothing that keeps a tree
alive, and the prepared calls by structure, not by object."""
import gc
import weakref

import pytest
import torch

import omeinsum_b200 as ome
from omeinsum_b200 import engine, plan

pytestmark = pytest.mark.gpu

CODE = "(ij,jk),kl->il"


def inputs():
    g = torch.Generator(device="cuda").manual_seed(1)
    return [torch.randn(6, 6, dtype=torch.float64, generator=g, device="cuda") for _ in range(3)]


@pytest.mark.parametrize("make", [lambda: ome.ein(CODE), lambda: ome.SlicedEinsum(["j"], ome.ein(CODE))])
def test_trees_are_given_back(make):
    xs = inputs()
    n0 = len(getattr(engine._TLS, "trees", {}))
    for _ in range(3):
        t = make()
        want = xs[0] @ xs[1] @ xs[2]
        torch.testing.assert_close(t(*xs), want)
        torch.testing.assert_close(t(*xs), want)
        refs = [weakref.ref(t), weakref.ref(t.eins if isinstance(t, ome.SlicedEinsum) else t.args[0])]
        del t
        gc.collect()
        assert all(r() is None for r in refs)
    gc.collect()
    assert len(engine._TLS.trees) <= n0


def test_a_new_object_takes_over_prepared_calls(monkeypatch):
    xs = inputs()
    want = xs[0] @ xs[1] @ xs[2]
    ome.ein(CODE)(*xs)

    def refuse(*a):
        raise AssertionError("planned again")

    with monkeypatch.context() as m:
        m.setattr(plan, "get_plan", refuse)
        torch.testing.assert_close(ome.ein(CODE)(*xs), want)
    # an equal tree that is changed afterwards, and one with another structure
    a, b = ome.ein(CODE), ome.ein(CODE)
    torch.testing.assert_close(a(*xs), want)
    b(*xs)
    b.eins = ome.EinCode(b.eins.ixs, ("l", "i"))
    torch.testing.assert_close(b(*xs), want.T)
    torch.testing.assert_close(a(*xs), want)
    a.args[0].eins = ome.EinCode([("j", "i"), ("j", "k")], ("i", "k"))
    torch.testing.assert_close(a(*xs), xs[0].T @ xs[1] @ xs[2])
    torch.testing.assert_close(ome.ein(CODE)(*xs), want)


def test_many_trees():
    """More live trees than are kept, called in turn."""
    xs = inputs()
    want = xs[0] @ xs[1] @ xs[2]
    trees = [ome.ein(CODE) for _ in range(2 * plan._STATES_MAX + 3)]
    for _ in range(2):
        for t in trees[::5] + trees[:3]:
            torch.testing.assert_close(t(*xs), want)
    for t in trees:
        t(*xs)
    assert len(engine._TLS.trees) <= plan._STATES_MAX
