"""Mixed splits whose tail lies below the FP32 noise (GPU required)."""

import numpy as np
import pytest

from oracle import seemps_oracle as so
from tests.gpu_util import to_np

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

import seemps2_gb300 as sg  # noqa: E402
from seemps2_gb300 import _lib, core  # noqa: E402
from tests.test_gpu_edges import matrix  # noqa: E402


@pytest.mark.parametrize("tail, redone", [(5e-14, True), (1e-16, False)])
def test_weight_left_at_the_noise_level(tail, redone):
    """100 values and a flat tail of 5e-14 of |A|^2, which FP32 cannot tell from its noise: five
    times what the QR may leave outside its rows at this tolerance, so it is run in full; a tail of
    1e-16 is left. The oracle's rank, the product to 2e-6 of its norm."""
    n, k = 256, 100
    s = np.geomspace(1.0, 10.0**-2.6, k)
    s = np.concatenate([s, np.full(n - k, np.sqrt(tail * (s**2).sum() / (n - k)))])
    A = matrix(np.random.default_rng(7), n, n, s, False)
    st, ost = (m.Strategy(tolerance=1e-12, max_bond_dimension=n) for m in (sg, so))
    sg.set_precision("mixed")
    _lib.stats_reset()
    try:
        L, R, e = core._left_orth_2site(A.reshape(n, 1, 1, n), st)
        stats = _lib.stats_read()
    finally:
        sg.set_precision("fp64")
    assert (stats["mixed_cap_redone"] > 0) == redone
    oL, oR, oe = so.left_orth_2site(A.reshape(n, 1, 1, n), ost)
    D = oL.shape[-1]
    assert L.shape[-1] == D
    P = oL.reshape(n, D) @ oR.reshape(D, n)
    assert np.linalg.norm(to_np(L).reshape(n, D) @ to_np(R).reshape(D, n) - P) <= 2e-6 * np.linalg.norm(P)
    assert abs(e - oe) <= 1e-7 * s[0]
