"""The CUDA-core GEMM (k_gemm_simt) and the FP64 matrix-instruction GEMM
(k_gemm_dmma) at the edges of their tiles, K stages and K splits, with several
modes per group, transposed and strided operands.

Tolerances: exact for Int64, Bool and max-plus; FP64 / ComplexF64 within
helpers' 1e-12 (sums of at most 4096 products of normal values, whose
round-off is about sqrt(K) * 2^-53 < 1e-14); FP32 / ComplexF32 on the CUDA
cores within 1e-5.
"""
import numpy as np
import pytest
import torch

import ome_oracle as O
import omeinsum_b200 as ome
from helpers import assert_match, gen, oracle, parse, to_dev, to_np

pytestmark = pytest.mark.gpu


def run(code, sizes, dt, seed, sx=True, sy=False):
    rng = np.random.default_rng(seed)
    ixs, iy = parse(code)
    xs = [gen(rng, [sizes[l] for l in ix], dt) for ix in ixs]
    want = oracle(ixs, iy, xs, sizes, dt)
    c = ome.EinCode(ixs, iy)
    if sx is True and sy is False:
        got = ome.einsum(c, [to_dev(x, dt) for x in xs], sizes)
    else:
        y0 = gen(rng, [sizes[l] for l in iy], dt)
        want = sx * want + sy * y0
        got = to_dev(y0, dt)
        ome.einsum_(c, [to_dev(x, dt) for x in xs], got, sx, sy, sizes)
    ome.device_status()
    assert_match(to_np(got), want, dt)


@pytest.mark.parametrize("dt", ["f64", "c128", "c64", "i64", "bool", "trop"])
@pytest.mark.parametrize("m,k,n", [(16, 8, 16), (17, 9, 33), (31, 64, 65), (64, 65, 63), (127, 15, 129),
                                   (128, 16, 128), (129, 17, 130), (200, 257, 131), (257, 31, 192), (16, 4096, 40)])
def test_tile_edges(m, k, n, dt):
    run("ij,jk->ik", dict(i=m, j=k, k=n), dt, 1000 * m + n)
    run("ji,kj->ki", dict(i=m, j=k, k=n), dt, 1000 * m + n + 1)


@pytest.mark.parametrize("dt", ["f64", "c128", "c64", "i64", "trop"])
@pytest.mark.parametrize("code,sizes", [
    ("acbd,cedf->eabf", dict(a=5, b=27, c=3, d=7, e=9, f=16)),           # two modes in every group
    ("apbqcr,qxpyr->yaxbc", dict(a=2, b=3, c=25, p=2, q=3, r=5, x=8, y=17)),   # three k modes, merged nowhere
    ("lacb,lcd->dabl", dict(a=9, b=15, c=21, d=130, l=3)),               # a batch mode
])
def test_several_modes(code, sizes, dt):
    run(code, sizes, dt, 7)
    if dt in ("f64", "i64"):
        run(code, sizes, dt, 8, sx=2, sy=3)


@pytest.mark.parametrize("dt", ["f64", "c128"])
def test_fp64_views(dt):
    """Operands that are strided views with odd offsets."""
    rng = np.random.default_rng(3)
    a, b = gen(rng, (300, 201), dt), gen(rng, (150, 603), dt)
    ad, bd = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
    got = ome.ein("ij,jk->ki")(ad[1::2, 1:], bd[10:140, ::3].t()[:200].contiguous().t().t())
    want = (a[1::2, 1:] @ b[10:140, ::3].T[:200]).T
    assert_match(to_np(got), want, dt)


@pytest.mark.parametrize("wide", ["none", "a", "b", "both", "edges"])
@pytest.mark.parametrize("m,k,n", [(130, 1000, 70), (40, 37, 300), (64, 20000, 64)])
def test_int64_stages_of_any_size(m, k, n, wide):
    """Int64 products are exact modulo 2^64 whichever stages hold values
    outside [-128, 127]."""
    rng = np.random.default_rng(m + k)
    a = rng.integers(-128, 128, (m, k), dtype=np.int64)
    b = rng.integers(-128, 128, (k, n), dtype=np.int64)
    big = lambda shape: rng.integers(-2 ** 63, 2 ** 63 - 1, shape, dtype=np.int64)
    if wide in ("a", "both"):
        a[:, k // 3:k // 2] = big((m, k // 2 - k // 3))
    if wide in ("b", "both"):
        b[k // 2:, 1::2] = big(b[k // 2:, 1::2].shape)
    if wide == "edges":
        a[0, 0], a[m - 1, k - 1], b[0, 0], b[k - 1, n - 1] = 128, -129, 127, -128
    got = ome.ein("ij,jk->ik")(torch.from_numpy(np.asfortranarray(a)).cuda(), torch.from_numpy(b).cuda())
    assert np.array_equal(to_np(got), a @ b)


@pytest.mark.parametrize("m,k,n", [(16, 8, 16), (33, 9, 40), (128, 77, 129), (130, 4097, 20)])
def test_tropical_f32_special_values(m, k, n):
    """Max-plus on Float32: exact, with infinities, NaN, signed zeros and the
    lowest finite value among the inputs."""
    rng = np.random.default_rng(m * k)
    a = rng.integers(-50, 50, (m, k)).astype(np.float32)
    b = rng.integers(-50, 50, (k, n)).astype(np.float32)
    a[1, :] = -np.inf
    a[2, k // 2] = np.nan
    a[3, 0] = np.inf
    a[4, :] = np.finfo(np.float32).min
    a[5, :], b[:, 0] = -0.0, -0.0
    want = O.einsum([("i", "j"), ("j", "k")], ("i", "k"), [a, b], dict(i=m, j=k, k=n), O.TROPICAL)
    got = ome.ein("ij,jk->ik")(ome.TropicalTensor(torch.from_numpy(np.asfortranarray(a)).cuda()),
                               ome.TropicalTensor(torch.from_numpy(b).cuda()))
    got = to_np(got)
    assert got.dtype == np.float32
    assert np.array_equal(got, want.astype(np.float32), equal_nan=True)


@pytest.mark.parametrize("code,sizes", [
    ("ij,jk->ik", dict(i=16, j=8, k=16)),
    ("ij,jk->ki", dict(i=33, j=31, k=65)),              # one past a tile on each side, K below a stage
    ("ji,kj->ik", dict(i=16, j=256, k=16)),             # one tile, K split over a cluster
    ("ij,jk->ik", dict(i=100, j=2000, k=100)),
    ("ij,jk->ik", dict(i=20, j=30000, k=30)),           # more splits than a cluster holds
    ("apbqc,xpyqc->abxy", dict(a=5, b=8, x=3, y=7, p=3, q=5, c=4)),    # three k modes
    ("apbqc,xpyqc->abxy", dict(a=32, b=32, x=16, y=31, p=8, q=8, c=8)),   # above 2^25 products
])
def test_small_f32_sums_in_double(code, sizes):
    """Small FP32 products are summed in Float64 and rounded once (once per
    split of K beyond a cluster, then their sum): norm-wise below 2e-7."""
    rng = np.random.default_rng(11)
    ixs, iy = parse(code)
    xs = [gen(rng, [sizes[l] for l in ix], "f32") for ix in ixs]
    want = oracle(ixs, iy, xs, sizes, "f32", wide=True)
    c = ome.EinCode(ixs, iy)
    assert_match(to_np(ome.einsum(c, [to_dev(x, "f32") for x in xs], sizes)), want, "f32", 2e-7)
    y0 = gen(rng, [sizes[l] for l in iy], "f32")
    yd = to_dev(y0, "f32")
    ome.einsum_(c, [to_dev(x, "f32") for x in xs], yd, 2, 3, sizes)
    ome.device_status()
    assert_match(to_np(yd), 2 * want + 3 * y0.astype(np.float64), "f32", 3e-7)


@pytest.mark.parametrize("code,sizes", [
    ("ij,jk->ik", dict(i=128, j=4000, k=257)),           # one row tile, a last column tile of one column
    ("ji,kj->ki", dict(i=511, j=513, k=513)),            # transposed operands, C contiguous along the second one
    ("ij,jk->ki", dict(i=1100, j=129, k=900)),
    ("acbd,cedf->eabf", dict(a=9, b=33, c=13, d=21, e=10, f=51)),   # two modes in every group
    ("lij,ljk->lik", dict(l=3, i=300, j=260, k=290)),    # a batch mode
])
def test_large_c32_on_tensor_cores(code, sizes):
    """Large ComplexF32 products run on the packed tensor-core kernel through
    the real embedding: norm-wise below 3e-7 of the ComplexF64 result (BF16x6
    products summed in FP32 over chunks of 128 real k)."""
    rng = np.random.default_rng(17)
    ixs, iy = parse(code)
    xs = [gen(rng, [sizes[l] for l in ix], "c64") for ix in ixs]
    want = oracle(ixs, iy, xs, sizes, "c64", wide=True)
    c = ome.EinCode(ixs, iy)
    for dev in ([to_dev(x, "c64") for x in xs], [torch.from_numpy(x).cuda() for x in xs]):
        assert_match(to_np(ome.einsum(c, dev, sizes)), want, "c64", 3e-7)
        ome.device_status()
    y0 = gen(rng, [sizes[l] for l in iy], "c64")
    yd = to_dev(y0, "c64")
    ome.einsum_(c, [to_dev(x, "c64") for x in xs], yd, 2 + 1j, 3, sizes)   # (general scalars: the CUDA cores)
    assert_match(to_np(yd), (2 + 1j) * want + 3 * y0.astype(np.complex128), "c64")
