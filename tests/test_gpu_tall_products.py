"""FP64 products with more rows than one grid dimension has tiles (GPU required)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

from seemps2_gb300 import core  # noqa: E402


@pytest.mark.parametrize("M, N, K", [(65535 * 16, 2, 2), (65535 * 16 + 1, 2, 2), (65535 * 16 + 1, 16, 3),
                                     (65535 * 32 + 1, 3, 2), (65535 * 32 + 1, 33, 17), (65535 * 64, 2, 3)])
def test_tall_fp64_products(M, N, K):
    """(K + 2) u of |A||B| on every row, up to the last one."""
    g = torch.Generator(device="cuda").manual_seed(M + N)
    A = torch.randn(M, K, dtype=torch.float64, device="cuda", generator=g)
    B = torch.randn(K, N, dtype=torch.float64, device="cuda", generator=g)
    err = ((core._gemm(A, 0, B, 0) - A @ B).abs() / (A.abs() @ B.abs())).max().item()
    assert err <= 2 * (K + 2) * 2.0**-53  # both sides are rounded


def test_tall_two_site_tensor():
    A = torch.randn(1, 2**20, 2, dtype=torch.float64, device="cuda")
    B = torch.randn(2, 2, 1, dtype=torch.float64, device="cuda")
    out = core._contract_last_and_first(A, B)
    assert out.shape == (1, 2**20, 2, 1)
    prod = lambda x, y: torch.einsum("aib,bjc->aijc", x, y)
    assert ((out - prod(A, B)).abs() / prod(A.abs(), B.abs())).max().item() <= 8 * 2.0**-53


def test_beyond_the_row_limit():
    A = torch.ones(65535 * 64 + 1, 2, dtype=torch.float64, device="cuda")
    with pytest.raises(ValueError, match="M too large"):
        core._gemm(A, 0, torch.ones(2, 2, dtype=torch.float64, device="cuda"), 0)


@pytest.mark.parametrize("K", [33, 64, 96, 250, 257, 300])
@pytest.mark.parametrize("M, N", [(1200, 69), (1024, 1024)])
def test_tf32_products_of_few_slabs(M, N, K):
    """One or two CTAs to a tile of a few slabs of K: 2e-6 of the norm, as the others."""
    from tests.test_gpu_tc import _gemm_f32

    rng = np.random.default_rng(M + K)
    A, B = rng.normal(size=(M, K)), rng.normal(size=(K, N))
    ref = A @ B
    assert np.linalg.norm(_gemm_f32("N", "N", A, B, M, N, K) - ref) <= 2e-6 * np.linalg.norm(ref)
