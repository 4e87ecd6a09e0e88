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


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("M, N, K", [(1, 1, 1), (15, 17, 16), (16, 33, 17), (31, 32, 129), (33, 200, 31),
                                     (174, 174, 190), (300, 7, 2000), (600, 600, 40)])
def test_fp64_gemm_tiles(M, N, K, cplx):
    """Tiles of 16 and 32 and one to eight ranges of K, every operand rule: (K + 2) u of |A||B|,
    twice that for complex products."""
    rng = np.random.default_rng(M + N + K)
    A, B = gaussian(rng, (M, K), cplx), gaussian(rng, (K, N), cplx)
    ref, scale = A @ B, np.abs(A) @ np.abs(B)
    op = {0: lambda x: x, 1: lambda x: x.T.copy(), 2: lambda x: x.conj().T.copy()}
    for opA, opB in [(0, 0), (1, 2), (2, 1), (0, 2)]:
        out = to_np(core._gemm(op[opA](A), opA, op[opB](B), opB))
        assert np.max(np.abs(out - ref) / scale) <= (2 + 2 * cplx) * (K + 2) * 2.0**-53


@pytest.mark.parametrize("m, n, kind, cplx", [
    (24, 300, "flat", False), (49, 64, "flat", True), (64, 65, "graded", False), (100, 200, "flat", False),
    (200, 100, "graded", False), (129, 130, "groups", False), (96, 128, "groups", True),
    (120, 150, "rank", False), (128, 100, "rank", True), (33, 257, "graded", True),
])
def test_fp64_splits_through_the_fp32_start(m, n, kind, cplx):
    """Flat spectra, spectra that span 1e-12 (several FP32 levels), groups of equal values (left
    to the Jacobi) and rank-deficient matrices, square, wide and tall."""
    rng = np.random.default_rng(m + n)
    k = min(m, n)
    s = {"flat": np.geomspace(1.0, 0.03, k), "graded": np.geomspace(1.0, 1e-12, k),
         "groups": np.repeat(np.geomspace(1.0, 0.01, k // 8 + 1), 8)[:k],
         "rank": np.geomspace(1.0, 1e-3, k // 3)}[kind]
    check_split(matrix(rng, m, n, s, cplx))


@pytest.mark.parametrize("m, n, cplx", [
    (24, 24, False), (64, 65, False), (129, 128, False), (257, 300, False), (96, 700, False), (512, 514, False),
    (25, 24, True), (128, 129, True), (256, 200, True), (300, 310, True),
])
def test_mixed_splits_at_the_cluster_sizes(m, n, cplx):
    """Where the FP32 stage changes its cluster or its registers: the oracle's rank (a gap of
    1e-8), an orthogonal factor to 1e-12, and the kept part to 2e-6 (the coupling of a kept and
    a dropped row that the split accepts is 1e-6)."""
    rng = np.random.default_rng(m + n)
    k = min(m, n) // 2
    A = matrix(rng, m, n, np.concatenate([np.geomspace(1.0, 0.1, k), np.full(k // 2, 1e-9)]), cplx)
    st = sg.Strategy(tolerance=1e-12, max_bond_dimension=k)
    ost = so.Strategy(tolerance=1e-12, max_bond_dimension=k)
    sg.set_precision("mixed")
    try:
        L, R, _ = core._left_orth_2site(A.reshape(m, 1, 1, n), st)
    finally:
        sg.set_precision("fp64")
    oL, oR, _ = so.left_orth_2site(A.reshape(m, 1, 1, n), ost)
    assert L.shape[-1] == oL.shape[-1] == k
    L, R = to_np(L).reshape(m, k), to_np(R).reshape(k, n)
    assert np.abs(L.conj().T @ L - np.eye(k)).max() <= 1e-12
    P = oL.reshape(m, k) @ oR.reshape(k, n)
    assert np.linalg.norm(L @ R - P) <= 2e-6 * np.linalg.norm(P)


@pytest.mark.parametrize("a, g, c, e", [(1, 1, 3, 3), (9, 33, 4, 9), (33, 8, 70, 5), (31, 40, 5, 17)])
def test_two_site_matvec_lists(a, g, c, e):
    """More than 8 output bonds, more than 256 inputs to an output (2 x 2 x 70), rectangular
    environments, sparse MPO tensors: sums of a c p1 p2 e terms, 1e-12 of the largest entry."""
    from oracle import dmrg_oracle as do
    from seemps2_gb300 import dmrg

    rng = np.random.default_rng(a + g + c + e)
    b, f = a + 2, g + 1
    L, R = rng.normal(size=(a, c, b)), rng.normal(size=(g, e, f))
    H = rng.normal(size=(c, 2, 2, 2, 2, e)) * (rng.random((c, 2, 2, 2, 2, e)) < 0.3)
    v = rng.normal(size=(b, 2, 2, f))
    ref = do.two_site_matvec(L, H, R, v)
    scale = do.two_site_matvec(abs(L), abs(H), abs(R), abs(v)).max()
    out = to_np(dmrg.two_site_matvec(L, H, R, v, "fp64"))
    assert np.abs(out - ref).max() <= 1e-12 * scale


def test_lanczos_of_tiny_operators():
    """Four unknowns and a run of thirty steps (it breaks down at four), and an eigenvector as
    the start (it breaks down at one): the lowest eigenvalue to 1e-12 of the norm."""
    from seemps2_gb300 import dmrg

    rng = np.random.default_rng(2)
    h = rng.normal(size=(4, 4))
    h = h + h.T
    H = h.reshape(2, 2, 2, 2).transpose(0, 2, 1, 3).reshape(1, 2, 2, 2, 2, 1)
    one = np.ones((1, 1, 1))
    w, u = np.linalg.eigh(h)
    for start in (rng.normal(size=4), u[:, 0]):
        ev, vec, _ = dmrg.lanczos_ground_state(one, H, one, start.reshape(1, 2, 2, 1), krylov=30)
        assert abs(ev - w[0]) <= 1e-12 * np.abs(w).max()
        assert abs(abs(to_np(vec).ravel() @ u[:, 0]) - 1.0) <= 1e-12


@pytest.mark.parametrize("batch", [1, 31, 33, 257])
def test_mlp_gradients_of_ragged_batches(batch):
    """One row, and a row short of and beyond the 32 x 32 tiles: the bars of the other gradient
    tests (1e-4 of the largest entry)."""
    from tests.test_gpu_learned import test_gradients_match_oracle

    test_gradients_match_oracle(batch)
