"""The Lanczos entry's checks and its end at an invariant subspace (GPU required)."""

import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

from seemps2_gb300 import _lib, dmrg  # noqa: E402


def operator(chi, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    r = lambda *s: torch.randn(*s, dtype=torch.float64, device="cuda", generator=g)
    return r(chi, 3, chi), r(3, 2, 2, 2, 2, 3), r(chi, 3, chi)


def lanczos(L, H, R, precision, prepared, m=4):
    a, c, b = L.shape
    g, e, f = R.shape
    n = b * 4 * f
    x0 = torch.ones(n, dtype=torch.float64, device="cuda")
    V = torch.empty((m, n), dtype=torch.float64, device="cuda")
    alpha, beta, steps = (C.c_double * m)(), (C.c_double * m)(), C.c_int()
    _lib.check(_lib.load().sm_two_site_lanczos(
        _lib.context(), _lib.int_array([a, c, b, 2, 2, e, g, f]), _lib.ptr(L), _lib.ptr(H), _lib.ptr(R),
        _lib.ptr(x0), m, dmrg.PRECISIONS[precision], prepared, _lib.ptr(V), alpha, beta, C.byref(steps),
        _lib.stream_handle()))
    return steps.value


def test_prepared_operator_has_to_be_the_one():
    """Another shape, other environments of the same shape, another precision: refused before any
    launch; the right one runs."""
    L, H, R = operator(16)
    op = dmrg.TwoSiteOperator(L, H, R, "bf16")
    assert lanczos(L, H, R, "bf16", 1) == 4
    for other, precision in [(operator(8), "bf16"), (operator(16, seed=1), "bf16"), ((L, H, R), "tf32x3"),
                             ((L, H, R), "fp64")]:
        _lib.stats_reset()
        with pytest.raises(ValueError, match="another prepared operator"):
            lanczos(*other, precision, 1)
        assert _lib.stats_read()["launches"] == 0
    op.ensure_prepared()
    assert lanczos(L, H, R, "bf16", 1) == 4


@pytest.mark.parametrize("precision, spread", [("fp64", False), ("fp64", True), ("fp64tc", True), ("bf16", False)])
def test_run_ends_at_an_invariant_subspace(precision, spread):
    """A diagonal operator of three values: a start that is an eigenvector and one that reaches
    three vectors. Of thirty steps asked for no more are issued than of two beyond those."""
    chi = 24
    eye = torch.eye(chi, dtype=torch.float64, device="cuda").reshape(chi, 1, chi)
    H = np.zeros((1, 2, 2, 2, 2, 1))
    for k, v in enumerate([-1.0, 0.5, 2.0, 2.0]):
        H[0, k // 2, k // 2, k % 2, k % 2, 0] = v
    start, steps = np.random.default_rng(0).normal(size=(chi, 2, 2, chi)), 3
    if not spread:
        start, steps = np.zeros_like(start), 1
        start[3, 0, 0, 5] = 1.0
    launches = []
    for krylov in (steps + 2, 30):
        _lib.stats_reset()
        lam, _, total = dmrg.lanczos_ground_state(eye, H, eye, start, krylov=krylov, precision=precision)
        launches.append(_lib.stats_read()["launches"])
        assert total == steps
        assert abs(lam + 1.0) <= 1e-12
    assert launches[1] <= launches[0]


@pytest.mark.parametrize("precision", ["bf16", "tf32x3"])
def test_mpo_entries_that_vanish_in_fp32(precision):
    """An MPO entry of 1e-60 meets products beyond the FP32 range: nothing is added, no NaN."""
    chi = 160
    L = torch.full((chi, 3, chi), 10.0, dtype=torch.float64, device="cuda")
    H = torch.zeros((3, 2, 2, 2, 2, 3), dtype=torch.float64, device="cuda")
    H[0, 0, 0, 0, 0, 0] = 1e-60
    op = dmrg.TwoSiteOperator(L, H, L, precision)
    out = op.matvec(torch.full((chi, 2, 2, chi), 1e38, dtype=torch.float64, device="cuda"))
    assert (out == 0).all()
