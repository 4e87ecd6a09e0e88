"""Singular values of FP64 splits through the FP32 start (GPU required): they are those of the
matrix only if the transform that the start applies is unitary to FP64."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

import seemps2_gb300 as sg  # noqa: E402
from seemps2_gb300 import _lib, core  # noqa: E402
from tests.test_gpu_edges import matrix  # noqa: E402


@pytest.mark.parametrize("m, n, decay, cplx", [(512, 512, 1.0, False), (511, 512, 6.0, False), (300, 400, 2.6, False),
                                               (400, 300, 12.0, False), (256, 260, 2.6, True)])
def test_singular_values(m, n, decay, cplx):
    """Within k u of the largest (the backward error of an FP64 SVD of k rows; the products are
    sums of k terms), and their squares sum up to |A|^2 to 4 k u."""
    k = min(m, n)
    A = matrix(np.random.default_rng(m + n), m, n, np.geomspace(1.0, 10.0**-decay, k), cplx)
    _lib.stats_reset()
    with _lib.SplitTrace() as tr:
        core._left_orth_2site(A.reshape(m, 1, 1, n), sg.Strategy(tolerance=1e-14))
    assert _lib.stats_read()["start_finished"] == 1
    s, u = np.asarray(tr.s[0])[:k], 2.0**-53
    assert np.abs(s - np.linalg.svd(A, compute_uv=False)).max() <= k * u * s[0]
    assert abs((s**2).sum() - np.linalg.norm(A) ** 2) <= 4 * k * u * np.linalg.norm(A) ** 2
