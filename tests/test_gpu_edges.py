"""Splits, products and steps at the sizes where a kernel's tiles or the choice between
two kernels change (GPU required): one short and one long of each boundary, remainders,
the smallest and the largest."""

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


def gaussian(rng, shape, cplx):
    x = rng.normal(size=shape)
    return x + 1j * rng.normal(size=shape) if cplx else x


def matrix(rng, m, n, s, cplx):
    """m x n with the singular values s"""
    q = [np.linalg.qr(gaussian(rng, (r, len(s)), cplx))[0] for r in (m, n)]
    return (q[0] * s) @ q[1].conj().T


def check_split(A, tol=1e-12, maxb=10**6, atol=1e-12):
    """Both two-site splits of the m x n matrix A against the oracle's: the kept rank, the
    product, the discarded weight, and the orthogonal factor.  An FP64 split of k rows is
    some 10 k rotations of each element, 4 roundings each: below 1e-12 for k < 250."""
    m, n = A.shape
    st = sg.Strategy(tolerance=tol, max_bond_dimension=maxb)
    ost = so.Strategy(tolerance=tol, max_bond_dimension=maxb)
    scale = max(np.linalg.norm(A, 2), 1e-300)
    for fn, ofn, left in [(core._left_orth_2site, so.left_orth_2site, True),
                          (core._right_orth_2site, so.right_orth_2site, False)]:
        L, R, e = fn(A.reshape(m, 1, 1, n), st)
        oL, oR, oe = ofn(A.reshape(m, 1, 1, n), ost)
        assert L.shape == oL.shape and R.shape == oR.shape
        D = L.shape[-1]
        L, R = to_np(L).reshape(m, D), to_np(R).reshape(D, n)
        assert np.abs(L @ R - oL.reshape(m, D) @ oR.reshape(D, n)).max() <= atol * scale
        Q = L.conj().T @ L if left else R @ R.conj().T
        assert np.abs(Q - np.eye(D)).max() <= atol
        assert abs(e - oe) <= 1e-9 * max(1e-2 * scale, oe)


@pytest.mark.parametrize("m, n, cplx", [
    (1, 1, False), (1, 1, True), (1, 7, False), (2, 2, True), (3, 2, False), (5, 4, True),
    (8, 9, False), (31, 33, False), (32, 32, True), (33, 31, False), (47, 64, False),
    # the last that one CTA takes, and the first that it does not: the work of 23^2 378
    # and, where the FP32 start takes over, 36^3 and 24^2 86 (complex 23^2 94, 27^3), the
    # shared memory of 9 x 2275
    (23, 378, False), (379, 23, False), (36, 36, False), (37, 37, False), (24, 86, False), (87, 24, False),
    (23, 94, True), (95, 23, True), (27, 27, True), (28, 28, True), (9, 2275, False), (2277, 9, False),
    (48, 86, False), (87, 48, False), (36, 38, True), (39, 36, True), (49, 49, False),
])
def test_small_fp64_splits(m, n, cplx):
    rng = np.random.default_rng(100 * m + n)
    k = min(m, n)
    check_split(matrix(rng, m, n, np.geomspace(1.0, 1e-3, k), cplx))
    # rows down to 1e-9 of the largest, half of them cut
    check_split(matrix(rng, m, n, np.geomspace(1.0, 1e-9, k), cplx), maxb=max(1, k // 2))


@pytest.mark.parametrize("cplx", [False, True])
def test_small_fp64_splits_of_odd_matrices(cplx):
    """Pairs of rows whose norms differ by far more than the FP32 range, equal rows,
    a zero row, and entries that are not finite."""
    rng = np.random.default_rng(5)
    A = gaussian(rng, (6, 20), cplx)
    graded = A * np.array([[1.0], [1e-30], [1e-60], [1.0], [0.0], [1e-5]])
    check_split(graded, tol=1e-25)
    check_split(np.vstack([A[:3], A[:3]]))
    A[2] = 0
    check_split(A)
    A[2, 3] = np.nan
    with pytest.raises(Exception):
        core._left_orth_2site(A.reshape(6, 1, 1, 20), sg.Strategy(tolerance=1e-12))


@pytest.mark.parametrize("M, N, K", [
    # tiles of 128 x 32 and 128 x 64 and their remainders, one slab of K and ragged ones,
    # clusters of 1, 2, 4 and 8 ranges, ranges left empty, several clusters to a tile
    (32, 32, 2048), (33, 65, 1000), (127, 33, 512), (129, 64, 300), (256, 257, 32), (257, 2080, 33),
    (1100, 1100, 64), (640, 640, 96), (300, 500, 288), (128, 32, 4097), (40, 48, 9001),
])
def test_sliced_gemm_tiles(M, N, K):
    """Against numpy's FP64 product, normalised by |A||B|: 8 sqrt(K) u; a row with a NaN or an
    infinity gives NaN, and only there."""
    from tests.test_gpu_tc import _gemm_f64tc

    rng = np.random.default_rng(M + N + K)
    A = rng.normal(size=(M, K)) * np.exp(rng.uniform(-18, 18, size=(M, 1)))
    B = rng.normal(size=(K, N)) * np.exp(rng.uniform(-18, 18, size=(1, N)))
    B[:, N // 2] = 0.0
    ref, scale = A @ B, np.abs(A) @ np.abs(B)
    scale[:, N // 2] = 1.0
    for opA, opB in [("N", "N"), ("T", "T")]:
        a, b = (A, B) if opA == "N" else (A.T.copy(), B.T.copy())
        assert np.max(np.abs(_gemm_f64tc(opA, opB, a, b, M, N, K) - ref) / scale) <= 8 * np.sqrt(K) * 2.0**-53
    A[1, 0], A[M - 1, K - 1] = np.nan, np.inf
    out = _gemm_f64tc("N", "N", A, B, M, N, K)
    assert np.isnan(out[[1, M - 1]]).all()
    rest = np.delete(np.arange(M), [1, M - 1])
    assert np.max((np.abs(out - ref) / scale)[rest]) <= 8 * np.sqrt(K) * 2.0**-53


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("chi, D, dense", [(33, 3, False), (31, 12, False), (65, 4, True), (1, 17, True)])
def test_mpo_scprod_lists(chi, D, dense, cplx):
    """<O a|O b> with tiles of 32 x 32 bonds left ragged and more than 256 inputs to an output
    (2 x 12^2), mostly zero and dense MPO tensors; sums of about chi^2 D^2 terms."""
    rng = np.random.default_rng(chi + D)
    n, d = 4, 2
    bond = [1] + [chi] * (n - 1) + [1]
    ob = [1] + [D] * (n - 1) + [1]
    a, b = ([gaussian(rng, (bond[i], d, bond[i + 1]), cplx) for i in range(n)] for _ in range(2))
    O = [gaussian(rng, (ob[i], d, d, ob[i + 1]), cplx) for i in range(n)]
    if not dense:
        O = [t * (rng.random(t.shape) < 0.2) for t in O]
    prod = lambda x: [np.einsum("aijb,cjd->acibd", o, t).reshape(o.shape[0] * t.shape[0], d, -1)
                      for o, t in zip(O, x)]
    ref = so.scprod(prod(a), prod(b))
    got = sg.mpo_scprod(sg.MPO(O), sg.MPS(a), sg.MPS(b))
    norm = np.sqrt(abs(so.scprod(prod(a), prod(a)) * so.scprod(prod(b), prod(b))))
    assert abs(got - ref) <= 1e-12 * norm


@pytest.mark.parametrize("M, N, K", [(32, 32, 600), (65, 33, 257), (129, 130, 96), (400, 300, 200), (48, 40, 5000)])
def test_sliced_complex_gemm_tiles(M, N, K):
    """The three real products of a complex one: 16 sqrt(K) u of |A||B| (the sum of three
    bounds of 8 sqrt(K) u, each of at most half of |A||B| in the part it enters)."""
    from tests.test_gpu_tc import _cplx_case, _gemm_c

    for opA, opB in [("N", "N"), ("T", "C"), ("C", "T")]:
        Aop, Bop, A, B = _cplx_case(M, N, K, opA, opB, M + N + K, scaled=True)
        out = _gemm_c("sm_gemm_f64tc", opA, opB, A, B, M, N, K)
        err = np.max(np.abs(out - Aop @ Bop) / (np.abs(Aop) @ np.abs(Bop)))
        assert err <= 16 * np.sqrt(K) * 2.0**-53


@pytest.mark.parametrize("M, N, K", [(64, 64, 1024), (65, 129, 1100), (127, 300, 250), (257, 128, 129), (128, 65, 17000)])
def test_tf32_gemm_tiles(M, N, K):
    """Tiles of 128 x 128 left ragged, clusters of 1 to 8 ranges of K and several clusters to a
    tile: 2e-6 of the norm (three products of 11-bit parts); a row of
    zeros stays one, and one with an infinity is not finite."""
    from tests.test_gpu_tc import _gemm_f32

    rng = np.random.default_rng(M + N + K)
    A, B = rng.normal(size=(M, K)), rng.normal(size=(K, N))
    A[3] = 0.0
    ref = A @ B
    out = _gemm_f32("N", "T", A, B.T.copy(), M, N, K)
    assert np.linalg.norm(out - ref) <= 2e-6 * np.linalg.norm(ref)
    assert (out[3] == 0.0).all()
    A[3, 5] = np.inf
    out = _gemm_f32("T", "N", A.T.copy(), B, M, N, K)
    assert not np.isfinite(out[3]).any()
    rest = np.delete(np.arange(M), 3)
    assert np.linalg.norm((out - ref)[rest]) <= 2e-6 * np.linalg.norm(ref)
