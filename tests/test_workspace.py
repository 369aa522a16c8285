"""The per-device context's workspace when the device has less memory than a
plan's peak: the least that the plan runs in will do."""
import numpy as np
import pytest
import torch

import omeinsum_b200 as ome
from omeinsum_b200 import _lib
from omeinsum_b200.plan import get_plan
from helpers import assert_match, gen, to_dev, to_np
from test_gpu_tiny_programs import chain

MB = 1 << 20


@pytest.fixture
def fake(monkeypatch):
    """Contexts of a device with 900 MB; the sizes that were asked for."""
    asked = []

    class Fake:
        def __init__(self, device, size):
            asked.append(size // MB)
            if size > 900 * MB:
                raise MemoryError("fake")
            self.workspace_bytes, self.refused, self.open = size, float("inf"), True

        def close(self):
            self.open = False

    monkeypatch.setattr(_lib, "Context", Fake)
    monkeypatch.setattr(_lib, "_contexts", {})
    monkeypatch.setattr(torch.cuda, "synchronize", lambda d=None: None)
    return asked


def test_growth(fake):
    c = _lib.context(0)
    assert c.workspace_bytes == _lib.DEFAULT_WORKSPACE and _lib.context(0, 200 * MB) is c
    d = _lib.context(0, 300 * MB)
    assert d.workspace_bytes == 512 * MB and not c.open and d.open
    e = _lib.context(0, 600 * MB)          # twice the old one is not there
    assert e.workspace_bytes == 600 * MB and not d.open
    assert fake == [256, 512, 1024, 600]


def test_least(fake):
    c = _lib.context(0, 300 * MB)
    d = _lib.context(0, 2000 * MB, 700 * MB)
    assert d.workspace_bytes == 700 * MB and not c.open
    n = len(fake)
    for _ in range(3):                     # (not tried again for as much or more)
        assert _lib.context(0, 2000 * MB, 700 * MB) is d
        assert _lib.context(0, 3000 * MB, 500 * MB) is d
    assert len(fake) == n
    assert _lib.context(0, 800 * MB, 100 * MB).workspace_bytes == 800 * MB


def test_refused(fake):
    _lib.context(0, 300 * MB)
    with pytest.raises(MemoryError):
        _lib.context(0, 2000 * MB)
    assert not _lib._contexts              # (no closed context stays behind)
    assert _lib.context(0).open


@pytest.mark.gpu
@pytest.mark.parametrize("grad", [False, True])
def test_tree_in_its_least_workspace(monkeypatch, grad):
    rng = np.random.default_rng(10)
    tree, ixs, sd = chain(12, [250], rng)
    tree = ome.NestedEinsum([tree], ome.EinCode([(0,)], ()))
    xs = [gen(rng, [250, 250], "f32") / np.float32(np.sqrt(250)) for _ in ixs]
    p = get_plan(tree, sd, _lib.F32, 0)
    least, peak = (p.grad_min, p.grad_bytes) if grad else (p.forward_min, p.forward_bytes)
    assert least < peak

    class Small(_lib.Context):
        def __init__(self, device, size):
            if size > least:
                raise MemoryError("fake")
            super().__init__(device, size)

    monkeypatch.setattr(_lib, "Context", Small)
    monkeypatch.setattr(_lib, "_contexts", {})
    monkeypatch.setattr(_lib, "DEFAULT_WORKSPACE", 0)
    dev = [to_dev(x, "f32") for x in xs]
    ts = [torch.from_numpy(x.astype(np.float64)).requires_grad_() for x in xs]
    v = torch.diagonal(torch.linalg.multi_dot(ts)).sum()
    for _ in range(2):
        if grad:
            y, grads = ome.cost_and_gradient(tree, dev)
            v.backward(retain_graph=True) if ts[0].grad is None else None
            for g, t in zip(grads, ts):
                assert_match(to_np(g), t.grad.numpy(), "f32")
        else:
            y = tree(*dev)
        assert_match(to_np(y), v.detach().numpy(), "f32")
    assert _lib._contexts[0].workspace_bytes == least
    _lib.release_workspaces()
