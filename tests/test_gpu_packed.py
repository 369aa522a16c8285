"""The packed tensor-core GEMM (k_gemm_packed): rows on 4-byte boundaries, so
that no tensor map describes the operands."""
import os
import subprocess
import sys

import pytest
import torch

import omeinsum_b200 as ome
from test_gpu_parity import kernel_names

pytestmark = pytest.mark.gpu


def test_long_k_running_sums():
    """2050 x 2050 x 65537, whole tiles on most SMs: 256 adds of 8 joined stages
    into a running sum, an add's rounding 0.4 * 2^-24 (rms) of a sum that grows
    as sqrt(i / 256): 2.7e-7, with the accumulators' own 2.4e-7 (norm-wise) 3.6e-7.
    More and smaller adds (4.7e-7 with 4 stages and the cross terms apart) are
    above the limit, 15% higher."""
    g = torch.Generator(device="cuda").manual_seed(5)
    mn, k = 2050, 65537
    a = torch.randn(mn + 1, k, generator=g, device="cuda")[:mn]
    b = torch.randn(k, mn + 1, generator=g, device="cuda")[:, :mn]
    y, names = kernel_names(lambda: ome.ein("ij,jk->ik")(a, b))
    assert "k_gemm_packed" in names, names
    w = a.double() @ b.double()
    assert float((y.double() - w).norm() / w.norm()) < 4.1e-7


@pytest.mark.parametrize("code,shapes", [
    ("ij,jk->ki", [(641, 1030), (1030, 1150)]),                        # 6 and 9 tiles of 128: an odd one on the second side
    ("ij,jk->ik", [(1150, 1030), (1030, 641)]),                        # the same with the operands' roles exchanged
    ("acbd,cedf->eabf", [(11, 33, 61, 23), (33, 20, 23, 55)]),         # two modes that do not merge in every group
    ("lij,ljk->lki", [(3, 390, 517), (3, 517, 970)]),                  # a batch mode
    ("ij,jk->ik", [(2050, 600), (600, 2900)]),                         # 9 x 12 tiles of 256: whole tiles and split ones
])
@pytest.mark.parametrize("prec", [0, 2, 3])
def test_f32(code, shapes, prec):
    """Float32 on rows that start on 4 bytes, with y <- 3 f + 2 y.  Norm-wise:
    three terms 3e-7 (FP32 accumulators of 128 to 256 k), two terms 1e-5 (a
    value's two terms leave 2^-17 of it)."""
    g = torch.Generator(device="cuda").manual_seed(9)
    xs = [torch.randn(*s[:-1], s[-1] + 1, generator=g, device="cuda")[..., 1:] for s in shapes]
    w = torch.einsum(code, *[x.double() for x in xs])
    tol = 1e-5 if prec == 2 else 3e-7
    ome.set_einsum_backend(ome.B200Backend(prec=prec))
    try:
        y, names = kernel_names(lambda: ome.ein(code)(*xs))
        assert "k_gemm_packed" in names, names
        assert float((y - w).norm() / w.norm()) < tol
        for out in (torch.randn(w.shape, generator=g, device="cuda"),
                    torch.randn(w.shape[::-1], generator=g, device="cuda").permute(*range(w.dim() - 1, -1, -1))):
            want = 3 * w + 2 * out.double()
            _, names = kernel_names(lambda: ome.einsum_(ome.ein(code), xs, out, 3, 2))
            assert "k_gemm_packed" in names, names
            assert float((out - want).norm() / want.norm()) < tol
    finally:
        ome.set_einsum_backend(ome.B200Backend())


@pytest.mark.parametrize("m,n,k", [(3072, 3072, 2048), (2304, 5000, 2304)])
def test_f32_aligned(m, n, k):
    """Large square-ish products take the packed kernel although tensor maps
    describe their operands."""
    g = torch.Generator(device="cuda").manual_seed(10)
    a, b = torch.randn(m, k, generator=g, device="cuda"), torch.randn(k, n, generator=g, device="cuda")
    w = a.double() @ b.double()
    for code in ("ij,jk->ik", "ij,jk->ki"):
        y, names = kernel_names(lambda: ome.ein(code)(a, b))
        assert names[0] == "k_gemm_packed", names
        assert float(((y if code[-1] == "k" else y.t()) - w).norm() / w.norm()) < 3e-7


def c32(*shape, g):
    return torch.randn(*shape, dtype=torch.complex64, generator=g, device="cuda")


@pytest.mark.parametrize("code,shapes", [
    ("acbd,cedf->eabf", [(9, 13, 33, 21), (13, 10, 21, 170)]),   # two modes in every group, none contiguous in two tensors
    ("lij,ljk->ikl", [(6, 300, 260), (6, 260, 290)]),            # a batch mode, contiguous in C
    ("ij,jk->ki", [(257, 1004), (1004, 600)]),                   # K in units of 4, rows on 8 bytes, roles exchanged
    ("ji,jk->ik", [(1005, 384), (1005, 384)]),                   # a last unit of one k
])
@pytest.mark.parametrize("prec", [0, 2])
def test_c32(code, shapes, prec):
    """ComplexF32 through the real embedding, on views that start on 8 bytes:
    norm-wise below 3e-7 (BF16x6 products in FP32 accumulators of 128 real k)."""
    g = torch.Generator(device="cuda").manual_seed(6)
    xs = [c32(*s[:-1], s[-1] + 1, g=g)[..., 1:] for s in shapes]
    w = torch.einsum(code, *[x.to(torch.complex128) for x in xs])
    ome.set_einsum_backend(ome.B200Backend(prec=prec))
    try:
        y, names = kernel_names(lambda: ome.ein(code)(*xs))
    finally:
        ome.set_einsum_backend(ome.B200Backend())
    assert "k_gemm_packed" in names, names
    assert float((y.to(w.dtype) - w).norm() / w.norm()) < 3e-7


@pytest.mark.parametrize("value", ["inf", "-inf", "nan", "3.4e38", "1.2e15", "7e-19", "1e-44"])
@pytest.mark.parametrize("side,at", [(0, (0, 0)), (0, (511, 511)), (1, (300, 511))])
def test_c32_out_of_range(value, side, at):
    """A product with a value that BF16 terms do not hold is the CUDA cores'."""
    g = torch.Generator(device="cuda").manual_seed(7)
    xs = [c32(512, 512, g=g), c32(512, 512, g=g)]
    code = ome.ein("ij,jk->ik")
    before = code(*xs)
    torch.view_as_real(xs[side])[at + (1,)] = float(value)
    y = code(*xs)
    again = code(*xs)
    ome.set_einsum_backend(ome.B200Backend(prec=1))
    try:
        w, names = kernel_names(lambda: code(*xs))
    finally:
        ome.set_einsum_backend(ome.B200Backend())
    assert "k_gemm_packed" not in names, names
    for v in (y, again):
        assert torch.equal(torch.nan_to_num(torch.view_as_real(v), nan=123.0), torch.nan_to_num(torch.view_as_real(w), nan=123.0))
    torch.view_as_real(xs[side])[at + (1,)] = 0
    after, names = kernel_names(lambda: code(*xs))
    assert "k_gemm_packed" in names, names
    rows = (slice(None), slice(0, 300)) if side else (slice(1, 511), slice(None))
    assert torch.equal(after[rows].isfinite(), before[rows].isfinite())


def test_c32_out_of_range_in_a_graph():
    """A captured product takes the path of each replay's values."""
    g = torch.Generator(device="cuda").manual_seed(8)
    a, b = c32(512, 512, g=g), c32(512, 512, g=g)
    code = ome.ein("ij,jk->ik")
    plain = code(a, b)
    st = torch.cuda.Stream()
    st.wait_stream(torch.cuda.current_stream())
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.stream(st):
        code(a, b)
        torch.cuda.synchronize()
        with torch.cuda.graph(graph, stream=st):
            y = code(a, b)
    for bad in (False, True, False):
        keep = a[3, 4].clone()
        if bad:
            a[3, 4] = float("inf")
        graph.replay()
        torch.cuda.synchronize()
        if bad:
            assert bool(torch.view_as_real(y)[3].isinf().any())
            assert torch.equal(torch.isfinite(y).all(dim=1), torch.arange(512, device="cuda") != 3)
        else:
            assert torch.equal(y, plain)
        a[3, 4] = keep


FORCED = """
import sys; sys.path[:0] = ["tests", "oracle", "."]
import conftest, torch
import omeinsum_b200 as ome
from test_gpu_parity import kernel_names
for m, n, k in ((3072, 3072, 2048), (64, 64, 64)):
    a, b = torch.randn(m, k, device="cuda"), torch.randn(k, n, device="cuda")
    y, names = kernel_names(lambda: ome.ein("ij,jk->ik")(a, b))
    assert float((y - a.double() @ b.double()).norm() / y.norm()) < 1e-6
    print(*names)
"""


@pytest.mark.parametrize("kernel,names", [
    ("", ["k_gemm_packed", "k_gemm_dmma"]),
    ("tma", ["k_gemm_tma2", "k_gemm_tma2"]),
    ("packed", ["k_gemm_packed", "k_gemm_packed"]),
    ("fused", ["k_gemm_bf16x3", "k_gemm_bf16x3"]),
])
def test_kernel_of_choice(kernel, names):
    """OME_GEMM selects the kernel whatever the size."""
    env = dict(os.environ, OME_GEMM=kernel)
    r = subprocess.run([sys.executable, "-c", FORCED], env=env, capture_output=True, text=True, timeout=300,
                       cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
    assert r.returncode == 0, r.stderr[-2000:]
    got = [line.split()[-1] for line in r.stdout.split("\n") if line.startswith("k_")]
    assert got == names, r.stdout
