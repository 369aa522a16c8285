"""Infinities and NaN in CUDA-core and FP64 matrix-instruction GEMMs, at sizes
that leave remainders in every tile: they appear where the sums of products
have them and nowhere else (padding adds none)."""
import numpy as np
import pytest

import omeinsum_b200 as ome
from helpers import gen, to_dev, to_np
from test_gpu_parity import kernel_names

pytestmark = pytest.mark.gpu


def products(a, b):
    """(real part, imaginary part) of a b."""
    with np.errstate(invalid="ignore"):
        if not np.iscomplexobj(a):
            return a @ b, np.zeros((a.shape[0], b.shape[1]))
        return a.real @ b.real - a.imag @ b.imag, a.real @ b.imag + a.imag @ b.real


@pytest.mark.parametrize("dt,kernel", [("f64", "k_gemm_dmma"), ("c128", "k_gemm_dmma"), ("f32", "k_gemm_dmma"),
                                       ("c64", "k_gemm_simt")])
@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
@pytest.mark.parametrize("m,n,k", [(200, 130, 77), (129, 257, 901)])
def test_gemm(dt, kernel, value, m, n, k):
    rng = np.random.default_rng(4)
    a, b = gen(rng, (m, k), dt), gen(rng, (k, n), dt)
    a[m - 1, k - 1] = value
    b[0, n // 2] = value
    b[k - 1, n - 1] = 0
    y, names = kernel_names(lambda: ome.ein("ij,jk->ik")(to_dev(a, dt), to_dev(b, dt)))
    assert names[0] == kernel, names
    wide = np.complex128 if np.iscomplexobj(a) else np.float64
    got = to_np(y).astype(wide)
    for g, w in zip((got.real, got.imag), products(a.astype(wide), b.astype(wide))):
        for kind in (np.isnan, np.isposinf, np.isneginf):
            assert np.array_equal(kind(g), kind(w)), kind.__name__
