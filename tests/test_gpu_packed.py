"""The packed tensor-core GEMM (k_gemm_packed): rows on 4-byte boundaries, so
that no tensor map describes the operands."""
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
