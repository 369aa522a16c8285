"""Float32 nodes of sliced trees: one order of summation for every node,
whatever kernel and tile serve it, so that the tree's value does not move when
a faster kernel takes a node over.  All comparisons are bit for bit."""
import numpy as np
import pytest
import torch

import omeinsum_b200 as ome
from helpers import gen, to_dev, to_np
from test_gpu_parity import kernel_names
from test_gpu_tiny_programs import chain

pytestmark = pytest.mark.gpu


def node_in_float32(ixs, xs, iy, sizes):
    """The node's value summed in Float32 term by term, a rounding per
    multiply-add (the product and sum are formed in 64 bits, where the product
    is exact)."""
    summed = [l for l in dict.fromkeys([l for ix in ixs for l in ix]) if l not in iy]
    assert len(summed) <= 1
    out = np.zeros([sizes[l] for l in iy], dtype=np.float32)
    for j in range(sizes[summed[0]] if summed else 1):
        ops = []
        for ix, x in zip(ixs, xs):
            sl = tuple(j if l in summed else slice(None) for l in ix)
            have = [l for l in ix if l not in summed]
            ops += [x[sl].astype(np.float64), [iy.index(l) for l in have]]
        out = (np.einsum(*ops, list(range(len(iy)))) + out.astype(np.float64)).astype(np.float32)
    return out


def tree_in_float32(ne, xs, sizes):
    if ne.isleaf:
        return xs[ne.tensorindex]
    return node_in_float32(ne.eins.ixs, [tree_in_float32(a, xs, sizes) for a in ne.args], ne.eins.iy, sizes)


def drop(ne, label):
    if ne.isleaf:
        return ne
    cut = lambda ix: tuple(l for l in ix if l != label)
    return ome.NestedEinsum([drop(a, label) for a in ne.args],
                            ome.EinCode([cut(ix) for ix in ne.eins.ixs], cut(ne.eins.iy)))


@pytest.mark.parametrize("n,ext", [(5, [2]), (17, [2, 3]), (40, [1, 2, 5]), (130, [2, 4])])
def test_small_nodes(n, ext):
    rng = np.random.default_rng(70 + n)
    tree, ixs, sizes = chain(n, ext, rng)
    cut = n // 2
    sizes[cut] = 2
    xs = [gen(rng, [sizes[l] for l in ix], "f32") for ix in ixs]
    got = to_np(ome.SlicedEinsum([cut], tree)(*[to_dev(x, "f32") for x in xs]))
    want = 0.0
    for s in range(2):
        part = [x[tuple(s if l == cut else slice(None) for l in ix)] for ix, x in zip(ixs, xs)]
        want = want + tree_in_float32(drop(tree, cut), part, sizes).astype(np.float64)
    assert np.array_equal(got, want.astype(np.float32))


def test_packed_gemm_rows():
    """A GEMM on k_gemm_packed (rows of B on 4-byte boundaries): 256 rows give
    the same bits alone, among 2560 (another tile count, other K splits) and
    with the output's modes exchanged (operands exchanged in the kernel)."""
    g = torch.Generator(device="cuda").manual_seed(3)
    k, n = 1025, 8191
    a = torch.randn(2, k, 2560, generator=g, device="cuda")
    a[1] = 0   # the second slice adds nothing
    a = a.permute(2, 1, 0)
    b = torch.randn(n, k, generator=g, device="cuda").t()

    def call(x, out):
        node = ome.NestedEinsum([ome.NestedEinsum(0), ome.NestedEinsum(1)], ome.EinCode(["mks", "kn"], out))
        y, names = kernel_names(lambda: ome.SlicedEinsum(["s"], node)(x, b))
        assert names.count("k_gemm_packed") == 2, names
        return y

    few = a[:256].permute(2, 1, 0).contiguous().permute(2, 1, 0)
    y = call(few, "mn")
    w = few[:, :, 0].double() @ b.double()
    assert float((y.double() - w).norm() / w.norm()) < 4e-7   # (2.4e-7: BF16x6 products, 8 stages in the accumulator)
    assert torch.equal(y, call(a, "mn")[:256])
    assert torch.equal(y, call(few, "nm").t())
