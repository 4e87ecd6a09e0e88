"""Splits of low rank in a cluster sized for many rows (GPU required): a block round is then one
pair, and a CTA's next send follows its last within a few hundred clocks."""

import numpy as np
import pytest

from oracle import seemps_oracle as so
from tests.gpu_util import to_np

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a CUDA GPU", allow_module_level=True)

import seemps2_gb300 as sg  # noqa: E402
from seemps2_gb300 import core  # noqa: E402


@pytest.mark.parametrize("m, n, rank, cplx", [(512, 512, 3, False), (512, 480, 17, False),
                                              (300, 300, 40, False), (256, 256, 9, True)])
def test_mixed_splits_of_low_rank(m, n, rank, cplx):
    """The oracle's rank, an orthogonal factor to 1e-12, the product to 2e-6 of its norm (the
    bars of the other mixed splits), and the same bits each time."""
    rng = np.random.default_rng(m + n + rank)
    normal = lambda r: rng.normal(size=(r, rank)) + (1j * rng.normal(size=(r, rank)) if cplx else 0.0)
    U, V = (np.linalg.qr(normal(r))[0] for r in (m, n))
    A = (U * np.geomspace(1.0, 0.1, rank)) @ V.conj().T
    st = sg.Strategy(tolerance=1e-12, max_bond_dimension=rank)
    oL, oR, _ = so.left_orth_2site(A.reshape(m, 1, 1, n), so.Strategy(tolerance=1e-12, max_bond_dimension=rank))
    first = None
    sg.set_precision("mixed")
    try:
        for _ in range(8):
            L, R, _ = (to_np(x) if hasattr(x, "cpu") else x
                       for x in core._left_orth_2site(A.reshape(m, 1, 1, n), st))
            first = (L, R) if first is None else first
            assert (L == first[0]).all() and (R == first[1]).all()
    finally:
        sg.set_precision("fp64")
    assert L.shape[-1] == oL.shape[-1] == rank
    L, R = L.reshape(m, rank), R.reshape(rank, n)
    assert np.abs(L.conj().T @ L - np.eye(rank)).max() <= 1e-12
    P = oL.reshape(m, rank) @ oR.reshape(rank, n)
    assert np.linalg.norm(L @ R - P) <= 2e-6 * np.linalg.norm(P)


@pytest.mark.parametrize("m, n, cplx", [(33, 190, False), (49, 174, False), (129, 133, False),
                                        (193, 129, True), (1025, 40, False), (1100, 65, False)])
def test_fp64_splits_whose_last_qr_batch_is_one_step(m, n, cplx):
    """4 j + 1 columns to reduce, in registers (the rows to 1024) and streamed, where the sums of
    the last batch follow those of the one before at once: the oracle's rank, the product to
    1e-12 and an orthogonal factor."""
    from tests.test_gpu_edges import check_split, matrix

    rng = np.random.default_rng(m + n)
    k = min(m, n)
    for _ in range(4):
        check_split(matrix(rng, m, n, np.geomspace(1.0, 1e-3, k), cplx))


@pytest.mark.parametrize("m, n, rank, cplx", [(512, 512, 430, False), (512, 500, 470, False), (512, 512, 490, False),
                                              (512, 512, 200, True), (512, 512, 300, True), (300, 512, 296, False)])
def test_mixed_splits_of_many_rows(m, n, rank, cplx):
    """Where shared memory has no room to send a round's rows from buffers apart (beyond 448 real
    rows of 512, 224 complex ones), with and without a warp to spare, and just below."""
    test_mixed_splits_of_low_rank(m, n, rank, cplx)
