"""Splits of few, long rows (GPU required): one CTA takes them up to a length of row, the grid's
kernels beyond; long columns stay with the one CTA."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

import seemps2_gb300 as sg  # noqa: E402
from seemps2_gb300 import _lib, core  # noqa: E402
from tests.test_gpu_edges import check_split, matrix  # noqa: E402


def launches(split, A):
    """of one split: three in the one-CTA form (the split, the isometry, the other factor)"""
    m, n = A.shape
    A = torch.from_numpy(A.reshape(m, 1, 1, n)).cuda()
    split(A, sg.Strategy(tolerance=1e-12))
    _lib.stats_reset()
    split(A, sg.Strategy(tolerance=1e-12))
    return _lib.stats_read()["launches"]


@pytest.mark.parametrize("k, limit, cplx", [(1, 640, False), (2, 384, False), (3, 160, False), (8, 160, False),
                                            (23, 160, False), (1, 320, True), (2, 192, True), (5, 80, True), (23, 80, True)])
def test_routes_and_results_at_the_row_limit(k, limit, cplx):
    rng = np.random.default_rng(k + limit)
    for l, one in [(limit, True), (limit + 1, False), (3 * limit, False)]:
        A = matrix(rng, k, l, np.geomspace(1.0, 1e-3, k), cplx)
        check_split(A)
        check_split(A.T.copy())
        assert (launches(core._right_orth_2site, A) <= 4) == one
        assert (launches(core._left_orth_2site, A.T.copy()) <= 4) == one
        assert launches(core._left_orth_2site, A) <= 4
        assert launches(core._right_orth_2site, A.T.copy()) <= 4
