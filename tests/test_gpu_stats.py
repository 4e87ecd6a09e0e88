"""What the timing statistics say of an FP64 split (GPU required)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

import seemps2_gb300 as sg  # noqa: E402
from seemps2_gb300 import _lib, core  # noqa: E402
from tests.test_gpu_edges import matrix  # noqa: E402


def timed_split(A):
    """(statistics, event-timed ms) of one split after two others"""
    m, n = A.shape
    A = torch.from_numpy(A.reshape(m, 1, 1, n)).cuda()
    st = sg.Strategy(tolerance=1e-12)
    for _ in range(2):
        core._left_orth_2site(A, st)
    _lib.stats_reset(timing=True)
    e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
    e[0].record()
    core._left_orth_2site(A, st)
    e[1].record()
    e[1].synchronize()
    s = _lib.stats_read()
    _lib.stats_reset(timing=False)
    return s, e[0].elapsed_time(e[1])


@pytest.mark.parametrize("m, n, values", [(16, 16, "flat"), (200, 220, "flat"), (200, 220, "equal"),
                                          (600, 640, "flat")])
def test_times_of_an_fp64_split(m, n, values):
    """The FP32 start's whole time is its own, an FP64 Jacobi is counted where one ran, and the
    parts do not exceed the call."""
    rng = np.random.default_rng(m)
    s = np.geomspace(1.0, 1e-2, m) if values == "flat" else np.repeat(np.geomspace(1.0, 0.1, m // 8), 8)
    st, ms = timed_split(matrix(rng, m, n, s, False))
    start, finished = (st["start_splits"], st["start_finished"])
    assert start == (1 if m == 200 else 0)
    assert st["jacobi_launches"] == 1 - finished
    assert (st["jacobi_ms"] > 0) == (st["jacobi_flops"] > 0) == (st["jacobi_launches"] == 1)
    flops = 4.0 * n * m**2 + 8.0 * m**3
    assert st["jacobi_flops"] + st["start_flops"] == flops
    assert st["jacobi_ms"] + st["start_ms"] + st["gemm_ms"] <= ms
    # the FP32 QR and Jacobi alone take more than this
    assert (st["start_ms"] > 0.2) if start else (st["start_ms"] == 0)
    if values == "flat":
        assert finished == start
