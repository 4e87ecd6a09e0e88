"""A context that has no room for the large clusters (GPU required): the splits take the FP64
kernels that need none, the tensor-core products smaller clusters, and the results stand."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

import seemps2_gb300 as sg  # noqa: E402
from seemps2_gb300 import _lib  # noqa: E402
from tests.test_gpu_edges import check_split, matrix  # noqa: E402


@pytest.fixture(params=[1, 4])
def limit(request):
    set_max = lambda n: _lib.check(_lib.load().sm_ctx_set_max_cluster(_lib.context(), n))
    set_max(request.param)
    yield request.param
    set_max(16)


@pytest.mark.parametrize("cplx", [False, True])
def test_splits_without_the_cluster(limit, cplx):
    rng = np.random.default_rng(11)
    A = matrix(rng, 150, 140, np.geomspace(1.0, 1e-4, 140), cplx)
    check_split(A)
    sg.set_precision("mixed")
    try:
        _lib.stats_reset()
        check_split(A)
        assert _lib.stats_read()["mixed_splits"] == 0
    finally:
        sg.set_precision("fp64")


def test_products_in_smaller_clusters(limit):
    """The bars of the other products: 8 sqrt(K) u of |A||B|, and 2e-6 of the norm."""
    from tests.test_gpu_tc import _gemm_f32, _gemm_f64tc

    rng = np.random.default_rng(12)
    for M, N, K in [(128, 64, 2048), (300, 200, 1000)]:
        A, B = rng.normal(size=(M, K)), rng.normal(size=(K, N))
        err = np.abs(_gemm_f64tc("N", "N", A, B, M, N, K) - A @ B) / (np.abs(A) @ np.abs(B))
        assert err.max() <= 8 * np.sqrt(K) * 2.0**-53
        assert np.linalg.norm(_gemm_f32("N", "N", A, B, M, N, K) - A @ B) <= 2e-6 * np.linalg.norm(A @ B)


def test_limit_is_checked():
    for n in (0, 17):
        with pytest.raises(ValueError):
            _lib.check(_lib.load().sm_ctx_set_max_cluster(_lib.context(), n))
