"""Permutations on extents that divide nothing (k_transpose32: tiles over runs
of one or two modes that are contiguous in x and in y), exact: around the tile
size, with and without a second mode in either run, strided inputs and outputs,
and y <- 3y + 2f."""
import numpy as np
import pytest
import torch

import omeinsum_b200 as ome
from helpers import assert_match, gen, oracle, parse, to_dev, to_np

pytestmark = pytest.mark.gpu

CASES = [
    ("ij->ji", dict(i=5, j=7)),
    ("ij->ji", dict(i=63, j=65)),
    ("ij->ji", dict(i=64, j=129)),
    ("abc->cab", dict(a=31, b=3, c=67)),            # y goes on with x's run
    ("abc->cba", dict(a=5, b=201, c=33)),           # the middle mode could join either run
    ("abcd->dcab", dict(a=7, b=11, c=5, d=13)),     # both runs of two modes
    ("abcde->ecadb", dict(a=31, b=5, c=9, d=3, e=39)),
    ("abcde->ebdca", dict(a=4, b=6, c=1, d=17, e=21)),
    ("abcdef->fbdace", dict(a=3, b=5, c=7, d=2, e=9, f=11)),
]


@pytest.mark.parametrize("dt", ["f32", "f64", "c64", "c128", "i64", "bool", "trop"])
@pytest.mark.parametrize("code,sizes", CASES)
def test_permute(code, sizes, dt):
    rng = np.random.default_rng(sum(sizes.values()))
    (ix,), iy = parse(code)
    x = gen(rng, [sizes[l] for l in ix], dt)
    want = oracle([ix], iy, [x], sizes, dt)
    c = ome.ein(code)
    assert_match(to_np(c(to_dev(x, dt))), want, dt)
    row = torch.from_numpy(np.ascontiguousarray(x)).cuda()
    assert_match(to_np(c(ome.TropicalTensor(row) if dt == "trop" else row)), want, dt)
    if dt in ("trop", "bool"):
        return
    big = torch.zeros([2 * s for s in x.shape], dtype=row.dtype, device="cuda")
    view = big[tuple(slice(1, None, 2) for _ in x.shape)]
    view.copy_(row)
    assert_match(to_np(c(view)), want, dt)
    # into every second element of a larger output, and onto old values
    shape = [sizes[l] for l in iy]
    out = torch.zeros([2 * s for s in shape], dtype=row.dtype, device="cuda").permute(*range(len(shape)))
    y = out[tuple(slice(None, None, 2) for _ in shape)]
    ome.einsum_(c, [to_dev(x, dt)], y, True, False, sizes)
    assert_match(to_np(y), want, dt)
    y0 = gen(rng, shape, dt)
    yd = to_dev(y0, dt)
    ome.einsum_(c, [to_dev(x, dt)], yd, 2, 3, sizes)
    assert_match(to_np(yd), 2 * want + 3 * y0, dt)
