"""What is timed: the calls that users of seemps2_gb300 make, over the sizes they make them at.

A case is one of six kinds of call:

* ``apply``   ``MPO.apply`` with its variational ``simplify``: the framework's main path, in the
  plain FP64 form (the default) and in the mixed forms (``set_precision``), from short chains of
  small bond (latency) to the n=30, chi=256 benchmark workload;
* ``euler``   ``simplify`` of an ``MPSSum``: one explicit Euler step x + dt L x;
* ``split``   one two-site split of the kernel table (``_left_orth_2site`` and its relatives);
* ``batch``   ``apply_batch`` of many independent, uneven MPS in complex64 storage;
* ``matvec`` / ``lanczos``  the two-site eigenproblem of DMRG: the prepared operator applied to a
  few vectors, and one Lanczos run;
* ``train``   loss and gradients of the rank predictor on a batch of truncations.

The factors of a split and the sites of an MPS are fixed only up to signs and rotations of the bond
bases, so a program never compares them; what it reads is what they stand for.  A split therefore
returns the product of its factors, and a simplified state its dense vector where that is short,
else its two-site overlap tensor with the input state (``AntilinearForm.tensor2site``: every site of
both states enters, nothing depends on the bond bases of the result).  The forms whose contractions
run at FP32 accuracy normalise their states (as ``SIMPLIFICATION_STRATEGY`` does) and keep their
results in 32 bits, like the complex64 storage of the batches.  The error bounds of a result are left
out: where nothing is discarded they are the square root of a rounding error.
"""

import math

import numpy as np
import torch

import seemps2_gb300 as sg
from seemps2_gb300 import batch, core, dmrg, learned

VECTOR_SITES = 16  # states up to this length are read as dense vectors


def listed():
    return [
        # the shortest call: a few sites, small bonds, all launches and host work
        dict(name="apply_small_fp64", kind="apply", operator="random", n=10, chi=8, D=3, cplx=False,
             form="fp64", tol=1e-10, maxb=16),
        # a random complex operator on a random state, compressed to twice the bond
        dict(name="apply_random_c128", kind="apply", operator="random", n=20, chi=32, D=4, cplx=True,
             form="fp64", tol=1e-10, maxb=64),
        # a finite-difference step on a 2^24-point grid in the default precision
        dict(name="apply_qtt_fp64", kind="apply", operator="laplacian", n=24, chi=64, D=3, cplx=False,
             form="fp64", tol=1e-12, maxb=64),
        # the same on 2^30 points at bond 128, still in plain FP64: the largest plain call
        dict(name="apply_qtt_fp64_large", kind="apply", operator="laplacian", n=30, chi=128, D=3,
             cplx=False, form="fp64", tol=1e-12, maxb=128),
        # the benchmark workload in its default form
        dict(name="apply_qtt_mixed", kind="apply", operator="laplacian", n=30, chi=256, D=3,
             cplx=False, form="mixed+learned", tol=1e-12, maxb=256),
        # one explicit Euler step of a diffusion equation, mixed precision
        dict(name="euler_mixed", kind="euler", n=30, chi=128, form="mixed", tol=1e-12, maxb=256),
        # one split of a TEBD or DMRG step, plain FP64, odd sizes, exponentially decaying values
        dict(name="split_fp64_odd", kind="split", op="left", a=87, b=95, cplx=False, form="fp64",
             decay=12.0, rank=174, tol=1e-12, maxb=128),
        # the mixed split at the benchmark's size and spectrum
        dict(name="split_mixed_512", kind="split", op="left", a=256, b=256, cplx=False, form="mixed",
             decay=2.6, rank=258, tol=1e-12, maxb=256),
        # many small independent compressions at once
        dict(name="batch_c64", kind="batch", count=12, nmin=10, nmax=40, chimin=8, chimax=64,
             streams=12, tol=1e-8),
        # DMRG at bond 256: the operator of a Lanczos run prepared, then applied
        dict(name="matvec_bf16_256", kind="matvec", chi=256, chir=256, precision="bf16", vectors=8),
        # one Lanczos run at the bond an L=100 Heisenberg chain reaches
        dict(name="lanczos_fp64_108", kind="lanczos", chi=108, chir=108, precision="fp64", krylov=30),
        # one training step of the rank predictor
        dict(name="train_512", kind="train", rows=512),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["apply"] * 6 + ["mixed"] * 3 + ["euler"] + ["split"] * 4 + ["batch"] +
                      ["matvec", "lanczos", "train"])
    if kind == "apply":
        if rng.random() < 0.5:
            n, chi = rng.randint(10, 26), _log_int(rng, 6, 96)
            return dict(kind="apply", operator="laplacian", n=n, chi=chi, D=3, cplx=False, form="fp64",
                        tol=1e-12, maxb=chi)
        cplx = rng.random() < 0.5
        n, chi, D = rng.randint(8, 22), _log_int(rng, 4, 32), rng.randint(2, 4)
        return dict(kind="apply", operator="random", n=n, chi=chi, D=D, cplx=cplx, form="fp64",
                    tol=rng.choice([1e-8, 1e-10]), maxb=2 * chi)
    if kind == "mixed":
        n, chi = rng.randint(16, 30), _log_int(rng, 32, 256)
        return dict(kind="apply", operator="laplacian", n=n, chi=chi, D=3, cplx=False,
                    form=rng.choice(["mixed", "mixed+learned"]), tol=1e-12, maxb=chi)
    if kind == "euler":
        chi = _log_int(rng, 16, 128)
        return dict(kind="euler", n=rng.randint(16, 30), chi=chi, form="mixed", tol=1e-12, maxb=2 * chi)
    if kind == "split":
        form = rng.choice(["fp64", "fp64", "mixed"])
        cplx = rng.random() < 0.3
        hi = 256 if form == "mixed" else 160
        a, b = _log_int(rng, 6, hi), _log_int(rng, 6, hi)
        if cplx:
            a, b = min(a, 120), min(b, 120)
        k = 2 * min(a, b)
        return dict(kind="split", op=rng.choice(["left", "right", "left", "svd"]) if form == "fp64" else
                    rng.choice(["left", "right"]), a=a, b=b, cplx=cplx, form=form,
                    decay=rng.choice([2.6, 4.0, 12.0]) if form == "fp64" else 2.6,
                    rank=max(1, int(k * rng.uniform(0.4, 1.0))), tol=1e-12,
                    maxb=max(1, int(k * rng.uniform(0.4, 0.8))))
    if kind == "batch":
        return dict(kind="batch", count=rng.randint(4, 12), nmin=10, nmax=rng.randint(12, 40), chimin=8,
                    chimax=rng.choice([16, 32, 64]), streams=rng.choice([4, 8, 12]), tol=1e-8)
    if kind == "matvec":
        return dict(kind="matvec", chi=_log_int(rng, 32, 256), chir=_log_int(rng, 32, 256),
                    precision=rng.choice(["fp64", "fp64tc", "tf32x3", "bf16"]),
                    vectors=rng.randint(2, 8))
    if kind == "lanczos":
        return dict(kind="lanczos", chi=_log_int(rng, 8, 160), chir=_log_int(rng, 8, 160),
                    precision=rng.choice(["fp64", "fp64tc"]), krylov=30)
    return dict(kind="train", rows=_log_int(rng, 48, 4096))


# --- inputs (numpy, from the seed alone) ------------------------------------------------------


def _normal(rng, shape, cplx=False):
    x = rng.normal(size=shape)
    return x + 1j * rng.normal(size=shape) if cplx else x


def _bonds(n, chi):
    return [min(chi, 2 ** min(i, n - i)) if min(i, n - i) < 30 else chi for i in range(n + 1)]


def _random_mps(rng, n, chi, cplx):
    """i.i.d. normal sites, normalised as a state."""
    b = _bonds(n, chi)
    sites = [_normal(rng, (b[i], 2, b[i + 1]), cplx) for i in range(n)]
    rho = np.eye(1)
    for k, A in enumerate(sites):
        rho = np.tensordot(A.conj(), np.tensordot(rho, A, axes=1), axes=([0, 1], [0, 1]))
        s = math.sqrt(abs(np.trace(rho)))
        sites[k], rho = A / s, rho / s**2
    sites[-1] = sites[-1] / math.sqrt(abs(rho[0, 0]))
    return sites


def _orthonormal_mps(rng, n, chi):
    """i.i.d. normal sites made left-orthonormal by QR, normalised."""
    b = _bonds(n, chi)
    sites, carry = [], np.eye(1)
    for i in range(n):
        A = np.tensordot(carry, rng.normal(size=(b[i], 2, b[i + 1])), axes=1)
        l, d, r = A.shape
        if i < n - 1:
            Q, carry = np.linalg.qr(A.reshape(l * d, r))
            sites.append(np.ascontiguousarray(Q.reshape(l, d, -1)))
        else:
            sites.append(A / np.linalg.norm(A))
    return sites


def _random_mpo(rng, n, D, cplx):
    return [_normal(rng, (1 if i == 0 else D, 2, 2, 1 if i == n - 1 else D), cplx) / math.sqrt(2 * D)
            for i in range(n)]


def _apply_inputs(case, rng):
    n, chi = case["n"], case["chi"]
    if case.get("operator", "laplacian") == "random":
        return _random_mps(rng, n, chi, case["cplx"]), _random_mpo(rng, n, case["D"], case["cplx"])
    h2 = 4.0**n
    return _orthonormal_mps(rng, n, chi), learned.tridiagonal_mpo(n, -2.0 * h2, h2, h2)


def _split_matrix(case, rng):
    m, n, r = 2 * case["a"], 2 * case["b"], case["rank"]
    r = min(r, m, n)
    U = np.linalg.qr(_normal(rng, (m, r), case["cplx"]))[0]
    V = np.linalg.qr(_normal(rng, (n, r), case["cplx"]))[0]
    return (U * np.geomspace(1.0, 10.0 ** -case["decay"], r)) @ V.conj().T


def _batch_inputs(case, rng):
    out = []
    # the sizes of a batch are spread evenly over its ranges, so that every seed costs the same
    lo, hi = case["chimin"], case["chimax"]
    chis = [c for c in (8, 16, 32, 64, 128) if lo <= c <= hi]
    for k in range(case["count"]):
        n = case["nmin"] + (k * 7) % (case["nmax"] - case["nmin"] + 1)
        chi = chis[k % len(chis)]
        mps = [t.astype(np.complex64) for t in _random_mps(rng, n, chi, True)]
        mpo = [t.astype(np.complex64) for t in _random_mpo(rng, n, 2 + 2 * (k % 2), True)]
        out.append((mps, mpo, chi))
    return out


def _heisenberg_pair():
    """The two-site bulk operator of the spin-1/2 Heisenberg chain, [c, i, j, k, l, d]."""
    Sp = np.array([[0.0, 1.0], [0.0, 0.0]])
    Sz, I2 = np.diag([0.5, -0.5]), np.eye(2)
    W = np.zeros((5, 2, 2, 5))
    W[0, :, :, 0] = W[4, :, :, 4] = I2
    W[0, :, :, 1], W[0, :, :, 2], W[0, :, :, 3] = Sp, Sp.T, Sz
    W[1, :, :, 4], W[2, :, :, 4], W[3, :, :, 4] = 0.5 * Sp.T, 0.5 * Sp, Sz
    return np.tensordot(W, W, axes=1)


def _dmrg_inputs(case, rng, vectors):
    a, g = case["chi"], case["chir"]
    L, R = rng.normal(size=(a, 5, a)), rng.normal(size=(g, 5, g))
    L, R = 0.5 * (L + L.transpose(2, 1, 0)), 0.5 * (R + R.transpose(2, 1, 0))
    H = _heisenberg_pair()
    H = 0.5 * (H + H.transpose(0, 2, 1, 4, 3, 5))
    return L, H, R, [rng.normal(size=(a, 2, 2, g)) for _ in range(vectors)]


def _train_inputs(case, rng):
    dims = learned.DIMS
    X = rng.normal(size=(case["rows"], dims[0])).astype(np.float32)
    y = rng.uniform(1.0, 8.0, size=case["rows"]).astype(np.float32)
    return X, y


def _strategy(case, maxb=None):
    return sg.DEFAULT_STRATEGY.replace(tolerance=case["tol"], max_sweeps=2, simplification_tolerance=0.0,
                                       max_bond_dimension=case["maxb"] if maxb is None else maxb,
                                       normalize=case.get("form", "fp64") != "fp64")


def _cuda(x):
    return torch.from_numpy(np.ascontiguousarray(x)).cuda()


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    state = dict(case=case)
    if case.get("form") == "mixed+learned":
        learned.RankModel.load(learned.PACKAGED_MODEL).install()
    if kind in ("apply", "euler"):
        mps, mpo = _apply_inputs(case, rng)
        state.update(psi=sg.MPS(mps), mpo=sg.MPO(mpo, _strategy(case)), strategy=_strategy(case))
    elif kind == "split":
        A = _split_matrix(case, rng)
        state.update(A=_cuda(A.reshape(case["a"], 2, 2, case["b"])),
                     strategy=sg.Strategy(tolerance=case["tol"], max_bond_dimension=case["maxb"]))
    elif kind == "batch":
        inst = _batch_inputs(case, rng)
        state.update(mpos=[sg.MPO(o, _strategy(case, chi)) for _, o, chi in inst],
                     states=[sg.MPS(s) for s, _, _ in inst])
    elif kind in ("matvec", "lanczos"):
        L, H, R, vs = _dmrg_inputs(case, rng, case.get("vectors", 1))
        state.update(L=_cuda(L), H=_cuda(H), R=_cuda(R), vs=[_cuda(v) for v in vs])
    else:
        X, y = _train_inputs(case, rng)
        state.update(model=learned.RankModel.initial(seed=seed % 2**31), X=_cuda(X), y=_cuda(y))
    return state


# --- one pass ----------------------------------------------------------------------------------


def _set_form(case):
    form = case.get("form", "fp64")
    sg.set_precision(form, contractions="fp64" if form == "fp64" else "fp32")


def _read(psi, out):
    """What a program reads of a simplified state (see the module's text)."""
    if psi.size <= VECTOR_SITES:
        return out.to_vector()
    return sg.AntilinearForm(psi, out, center=psi.size // 2).tensor2site(+1)


def _kept(case, x):
    """Results of the FP32-accurate forms are kept in 32 bits."""
    return x if case.get("form", "fp64") == "fp64" else x.to(torch.complex64 if x.is_complex() else
                                                             torch.float32)


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "apply":
        _set_form(case)
        out = state["mpo"].apply(state["psi"])
        return _kept(case, _read(state["psi"], out))
    if kind == "euler":
        _set_form(case)
        psi = state["psi"]
        dt = 0.1 * 0.25 ** case["n"]  # a stable explicit step, dt = 0.1 h^2
        step = psi + dt * state["mpo"].apply(psi, simplify=False)
        out = sg.simplify(step, strategy=state["strategy"])
        return _kept(case, _read(psi, out))
    if kind == "split":
        _set_form(case)
        A, st = state["A"], state["strategy"]
        if case["op"] == "svd":
            U, s, V = core._destructive_svd(A.reshape(2 * case["a"], 2 * case["b"]))
            return {"s": s, "product": core._contract_last_and_first(U * s, V)}
        fn = core._left_orth_2site if case["op"] == "left" else core._right_orth_2site
        L, R, _ = fn(A, st)
        return {"product": _kept(case, core._contract_last_and_first(L, R))}
    if kind == "batch":
        sg.set_precision("fp64")
        outs, _ = batch.apply_batch(state["mpos"], state["states"], streams=case["streams"],
                                    precision="mixed")
        return [_read(p, o).to(torch.complex64) for p, o in zip(state["states"], outs)]
    if kind == "matvec":
        sg.set_precision("fp64")
        L, H, R, prec = state["L"], state["H"], state["R"], case["precision"]
        if prec in ("fp64", "fp64tc"):
            return [dmrg.two_site_matvec(L, H, R, v, prec) for v in state["vs"]]
        op = dmrg.TwoSiteOperator(L, H, R, prec)
        return [op.matvec(v).float() for v in state["vs"]]
    if kind == "lanczos":
        sg.set_precision("fp64")
        v = state["vs"][0]
        lam, x, _ = dmrg.lanczos_ground_state(state["L"], state["H"], state["R"], v,
                                              krylov=case["krylov"], precision=case["precision"])
        # the eigenvector's sign: towards the start vector
        return {"energy": torch.tensor(lam, dtype=torch.float64), "vector": x * torch.sign((x * v).sum())}
    loss, grads = state["model"].loss_and_grad(state["X"], state["y"])
    return {"loss": loss, "grads": grads}


# --- the least work of a pass --------------------------------------------------------------------


def _sweep_work(n, chi, ket, maxb, cplx, sweeps):
    """Flops of the canonical form, the norm and the sweeps at the bonds' upper limits (splits as
    4 m n^2 + 8 n^3 of the canonical form's one-site and the sweeps' two-site matrices)."""
    cf = 4.0 if cplx else 1.0
    K, B = _bonds(n, ket), _bonds(n, maxb)
    fl = 0.0
    for i in range(n):
        m, k = min(K[i], 2 * B[i + 1]), max(K[i], 2 * B[i + 1])
        fl += 4.0 * k * m * m + 8.0 * m**3 + 2.0 * 2 * K[i] * K[i + 1] * B[i + 1]
        fl += (1 + sweeps) * 2.0 * 2 * (B[i] * K[i] * K[i + 1] + B[i] * K[i + 1] * B[i + 1])
    for i in range(n - 1):
        p, q = 2 * B[i], 2 * B[i + 2]
        m, k = min(p, q), max(p, q)
        fl += sweeps * (4.0 * k * m * m + 8.0 * m**3 + 2.0 * p * q * K[i + 1])
    size = sum(2 * B[i] * B[i + 1] for i in range(n)) + sum(2 * _bonds(n, chi)[i] * _bonds(n, chi)[i + 1]
                                                           for i in range(n))
    return {"bytes": (16.0 if cplx else 8.0) * size, "flops": cf * fl}


def work(case):
    kind = case["kind"]
    if kind == "apply":
        return _sweep_work(case["n"], case["chi"], case["chi"] * case["D"], case["maxb"], case["cplx"], 2)
    if kind == "euler":
        return _sweep_work(case["n"], case["chi"], 4 * case["chi"], case["maxb"], False, 2)
    if kind == "split":
        m, n = 2 * case["a"], 2 * case["b"]
        lo, hi = min(m, n), max(m, n)
        e, cf = (16.0, 4.0) if case["cplx"] else (8.0, 1.0)
        return {"bytes": e * 2 * m * n, "flops": cf * (4.0 * hi * lo * lo + 8.0 * lo**3)}
    if kind == "batch":
        tot = {"bytes": 0.0, "flops": 0.0}
        chis = [c for c in (8, 16, 32, 64, 128) if case["chimin"] <= c <= case["chimax"]]
        for k in range(case["count"]):
            n, chi = case["nmin"] + (k * 7) % (case["nmax"] - case["nmin"] + 1), chis[k % len(chis)]
            w = _sweep_work(n, chi, chi * (2 + 2 * (k % 2)), chi, True, 2)
            tot = {key: tot[key] + w[key] for key in tot}
        return tot
    if kind in ("matvec", "lanczos"):
        a, g = case["chi"], case["chir"]
        times = case["vectors"] if kind == "matvec" else case["krylov"]
        one = 2.0 * 5 * 4 * a * g * (a + g) + 2.0 * a * g * 4 * 16
        vec = 4.0 * a * g
        extra = 4.0 * vec * times * times if kind == "lanczos" else 0.0
        return {"bytes": 8.0 * (5 * a * a + 5 * g * g + 2 * vec * (times if kind == "matvec" else 1)),
                "flops": times * one + extra}
    d = learned.DIMS
    par = sum(d[k] * d[k + 1] for k in range(len(d) - 1))
    return {"bytes": 4.0 * (case["rows"] * (d[0] + 1) + 2 * par), "flops": 6.0 * case["rows"] * par}


# --- the same in 64 bits, plain numpy ------------------------------------------------------------


def _rank(s, tol, maxb):
    tail = np.concatenate([[0.0], np.cumsum(s[::-1] ** 2)])  # tail[j]: the j smallest dropped
    over = np.nonzero(tail[:len(s)] > tail[-1] * tol)[0]
    drop = int(over[0]) - 1 if len(over) else len(s) - 1
    return min(len(s) - drop, maxb)


def _split(A, tol, maxb):
    U, s, V = np.linalg.svd(A, full_matrices=False)
    D = _rank(s, tol, maxb)
    return U[:, :D], s[:D], V[:D]


def _env_left(B, A, rho):
    return np.tensordot(B.conj(), np.tensordot(rho, A, axes=1), axes=([0, 1], [0, 1]))


def _env_right(B, A, rho):
    return np.tensordot(np.tensordot(A, rho, axes=1), B.conj(), axes=([1, 2], [1, 2]))


def _overlap(a, b):
    rho = np.eye(1)
    for A, B in zip(a, b):
        rho = _env_left(A, B, rho)
    return rho[0, 0]


def _join(weights, kets):
    n = len(kets[0])
    out = []
    for i in range(n):
        As = [k[i] for k in kets]
        if i == 0:
            out.append(np.concatenate([w * A for w, A in zip(weights, As)], axis=2))
        elif i == n - 1:
            out.append(np.concatenate(As, axis=0))
        else:
            B = np.zeros((sum(A.shape[0] for A in As), 2, sum(A.shape[2] for A in As)), As[0].dtype)
            l = r = 0
            for A in As:
                B[l:l + A.shape[0], :, r:r + A.shape[2]] = A
                l, r = l + A.shape[0], r + A.shape[2]
            out.append(B)
    return out


def _simplified(weights, kets, tol, maxb, normalize=False, sweeps=2):
    """The sites of the two-site variational simplification, canonical start at site 0."""
    n, nt = len(kets[0]), len(kets)
    bra = _join(weights, kets) if nt > 1 or weights[0] != 1 else list(kets[0])
    norm2 = abs(sum(np.conj(weights[i]) * weights[j] * _overlap(kets[i], kets[j])
                    for i in range(nt) for j in range(nt)))
    for i in range(n - 1, 0, -1):
        a, d, b = bra[i].shape
        U, s, V = _split(bra[i].reshape(a, d * b), tol, maxb)
        bra[i] = V.reshape(-1, d, b)
        bra[i - 1] = np.tensordot(bra[i - 1], U * s, axes=1)
    L = [[np.eye(1)] * n for _ in range(nt)]
    R = [[np.eye(1)] * n for _ in range(nt)]
    for t in range(nt):
        for i in range(n - 1, 0, -1):
            R[t][i - 1] = _env_right(bra[i], kets[t][i], R[t][i])
    right, err = True, 2.0
    for _ in range(sweeps):
        for i in range(n - 1) if right else range(n - 2, -1, -1):
            AA = sum(w * np.tensordot(np.tensordot(L[t][i], kets[t][i], axes=1),
                                      np.tensordot(kets[t][i + 1], R[t][i + 1], axes=1), axes=1)
                     for t, w in enumerate(weights))
            a, d, e, b = AA.shape
            U, s, V = _split(AA.reshape(a * d, e * b), tol, maxb)
            U, V = (U, s[:, None] * V) if right else (U * s, V)
            bra[i], bra[i + 1] = U.reshape(a, d, -1), V.reshape(-1, e, b)
            for t in range(nt):
                if right and i + 1 < n:
                    L[t][i + 1] = _env_left(bra[i], kets[t][i], L[t][i])
                elif not right:
                    R[t][i] = _env_right(bra[i + 1], kets[t][i + 1], R[t][i + 1])
        c = n - 1 if right else 0
        one = sum(w * np.tensordot(L[t][c], np.tensordot(kets[t][c], R[t][c], axes=1), axes=1)
                  for t, w in enumerate(weights))
        nm = np.vdot(bra[c], bra[c]).real
        old, err = err, 2.0 * abs(1.0 - np.vdot(bra[c], one).real / math.sqrt(nm * norm2))
        if err > old:
            break
        right = not right
    if normalize:
        bra[c] = bra[c] / math.sqrt(nm)
    return bra


def _read_exact(psi, out):
    n = len(psi)
    if n <= VECTOR_SITES:
        v = np.ones((1, 1))
        for A in out:
            v = np.tensordot(v, A, axes=1).reshape(-1, A.shape[2])
        return v.reshape(-1)
    c = n // 2
    L, R = np.eye(1), np.eye(1)
    for i in range(c):
        L = _env_left(psi[i], out[i], L)
    for i in range(n - 1, c + 1, -1):
        R = _env_right(psi[i], out[i], R)
    return np.tensordot(np.tensordot(L, out[c], axes=1), np.tensordot(out[c + 1], R, axes=1), axes=1)


def _product(mpo, mps):
    return [np.einsum("aijb,cjd->caidb", O, A, optimize=True).reshape(O.shape[0] * A.shape[0], O.shape[1], -1)
            for O, A in zip(mpo, mps)]


def _double(ts):
    return [t.astype(np.complex128 if np.iscomplexobj(t) else np.float64) for t in ts]


def exact(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind in ("apply", "euler"):
        mps, mpo = _apply_inputs(case, rng)
        prod = _product(mpo, mps)
        if kind == "euler":
            weights, kets = [1.0, 1.0], [mps, [0.1 * 0.25 ** case["n"] * prod[0]] + prod[1:]]
        else:
            weights, kets = [1.0], [prod]
        return _read_exact(mps, _simplified(weights, kets, case["tol"], case["maxb"],
                                            case.get("form", "fp64") != "fp64"))
    if kind == "split":
        A = _split_matrix(case, rng)
        if case["op"] == "svd":
            return {"s": np.linalg.svd(A, compute_uv=False), "product": A}
        U, s, V = _split(A, case["tol"], case["maxb"])
        return {"product": ((U * s) @ V).reshape(case["a"], 2, 2, case["b"])}
    if kind == "batch":
        inst = [(_double(mps), _double(mpo), chi) for mps, mpo, chi in _batch_inputs(case, rng)]
        return [_read_exact(mps, _simplified([1.0], [_product(mpo, mps)], case["tol"], chi))
                for mps, mpo, chi in inst]
    if kind in ("matvec", "lanczos"):
        L, H, R, vs = _dmrg_inputs(case, rng, case.get("vectors", 1))

        def matvec(v):
            x = np.tensordot(L, v, axes=([2], [0]))  # a c k l f
            x = np.tensordot(x, H, axes=([1, 2, 3], [0, 2, 4]))  # a f i j d
            return np.tensordot(x, R, axes=([4, 1], [1, 2]))  # a i j g

        if kind == "matvec":
            return [matvec(v) for v in vs]
        v = vs[0]
        Q, T = [v.reshape(-1) / np.linalg.norm(v)], np.zeros((case["krylov"],) * 2)
        m = min(case["krylov"], v.size)
        for j in range(m):
            w = matvec(Q[j].reshape(v.shape)).reshape(-1)
            T[j, j] = Q[j] @ w
            for _ in range(2):
                M = np.array(Q)
                w = w - M.T @ (M @ w)
            if j + 1 < m:
                T[j, j + 1] = T[j + 1, j] = np.linalg.norm(w)
                Q.append(w / T[j, j + 1])
        lam, Y = np.linalg.eigh(T[:m, :m])
        x = (Y[:, 0] @ np.array(Q)).reshape(v.shape)
        return {"energy": lam[:1].reshape(()), "vector": x * np.sign(np.sum(x * v))}
    X, y = _train_inputs(case, rng)
    d = learned.DIMS
    gen = np.random.default_rng(seed % 2**31)  # the initial parameters, drawn layer by layer
    par = []
    for k in range(len(d) - 1):
        bound = 1.0 / np.sqrt(d[k])
        par.append([gen.uniform(-bound, bound, size=sz).astype(np.float32).astype(np.float64)
                    for sz in (d[k + 1] * d[k], d[k + 1])])
    z, a = [], [X.astype(np.float64)]
    c = math.sqrt(2.0 / math.pi)
    for k, (W, b) in enumerate(par):
        z.append(a[-1] @ W.reshape(d[k + 1], d[k]).T + b)
        t = np.tanh(c * (z[-1] + 0.044715 * z[-1] ** 3))
        a.append(0.5 * z[-1] * (1.0 + t) if k + 1 < len(par) else z[-1])
    r = a[-1][:, 0] - y.astype(np.float64)
    g, grads = (2.0 * r / len(r))[:, None], []
    for k in range(len(par) - 1, -1, -1):
        grads = [(g.T @ a[k]).reshape(-1), g.sum(axis=0)] + grads
        if k:
            x = z[k - 1]
            t = np.tanh(c * (x + 0.044715 * x**3))
            dx = 0.5 * (1.0 + t) + 0.5 * x * (1.0 - t * t) * c * (1.0 + 3.0 * 0.044715 * x * x)
            g = (g @ par[k][0].reshape(d[k + 1], d[k])) * dx
    return {"loss": np.array([np.mean(r * r)]), "grads": np.concatenate(grads)}
