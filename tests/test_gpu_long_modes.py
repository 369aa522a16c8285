"""CUDA-core GEMMs whose modes do not fit 31 or 32 bits (operands expanded with
stride 0 reach such lengths without the memory)."""
import pytest
import torch

import omeinsum_b200 as ome
from test_gpu_parity import kernel_names

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,n", [(torch.int64, 2**30 + 1), (torch.bool, 2**31 + 3), (torch.int64, 2**32 + 3)])
def test_summed_mode(dtype, n):
    """sum over p (2) and q (n, the same value along it) of A[i,p,q] B[p,q,j]."""
    g = torch.Generator(device="cuda").manual_seed(2)
    a, b = (torch.randint(0, 3, (17, 2), generator=g, device="cuda", dtype=torch.int64),
            torch.randint(0, 3, (2, 19), generator=g, device="cuda", dtype=torch.int64))
    if dtype == torch.bool:
        a, b = a > 1, b > 1
    code = ome.ein("ipq,pqj->ij")
    got, names = kernel_names(lambda: code(a[:, :, None].expand(17, 2, n), b[:, None, :].expand(2, n, 19)))
    assert names[0] == "k_gemm_simt", names
    want = (a.long()[:, :, None] * b.long()[None]).sum(1)
    assert torch.equal(got, want > 0 if dtype == torch.bool else want * n)


def test_output_mode():
    """2^32 + 5 rows, all alike, of 16 columns."""
    m = 2**32 + 5
    torch.cuda.empty_cache()
    if torch.cuda.mem_get_info()[0] < 90 << 30:
        pytest.skip("the result takes 64 GiB")
    g = torch.Generator(device="cuda").manual_seed(3)
    a, b = torch.rand(9, generator=g, device="cuda") > 0.6, torch.rand(9, 16, generator=g, device="cuda") > 0.6
    y = ome.ein("ik,kj->ji")(a.expand(m, 9), b)
    row = (a[:, None] & b).any(0)
    assert y.shape == (16, m)
    for lo in range(0, m, 1 << 28):
        assert bool((y[:, lo:lo + (1 << 28)] == row[:, None]).all())
