"""Signs of the eigenvectors that the Davidson step takes from a symmetric Ritz matrix.  An eigenvector is fixed up to
its sign; cyclic Jacobi decides it by the order of its rotations, and programs that keep vectors rely on it.  The
reference here restates that order: rounds r = 0, 1, .. of the pairs {r, m - 1} and {r + k, r - k} modulo m - 1
(m = n rounded up to even), each rotation of lower index p and higher index q by the smaller root of t^2 + 2 tau t - 1
= 0, tau = (a_qq - a_pp) / (2 a_pq), t = 1 at tau = 0.
"""
import numpy as np
import pytest

from cpsd_b200 import api, synth

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def jacobi(A):
    """eigenvalues and eigenvector columns, unsorted"""
    n = len(A)
    m = n + (n & 1)
    S, V = np.zeros((m, m)), np.eye(m)
    S[:n, :n] = A
    for rnd in range(50 * (m - 1)):
        a = np.abs(S[:n, :n])
        if not np.any(np.triu(a > 1e-17 * np.sqrt(np.outer(a.diagonal(), a.diagonal())), 1)):
            break
        r = rnd % (m - 1)
        J, U = np.eye(m), V.copy()
        pairs = [sorted((r, m - 1))] + [sorted(((r + k) % (m - 1), (r - k) % (m - 1))) for k in range(1, m // 2)]
        for p, q in pairs:
            if abs(S[p, q]) <= 1e-17 * np.sqrt(abs(S[p, p] * S[q, q])):
                continue
            d, b = S[q, q] - S[p, p], 2.0 * S[p, q]
            t = abs(b) / (abs(d) + np.hypot(d, b))
            if d != 0.0 and (d > 0.0) != (b > 0.0):
                t = -t
            c = float(1.0 / np.sqrt(1.0 + np.longdouble(t) ** 2))
            J[p, p] = J[q, q] = c
            J[p, q], J[q, p] = t * c, -t * c
            U[:, p], U[:, q] = c * V[:, p] - t * c * V[:, q], t * c * V[:, p] + c * V[:, q]
        S, V = J.T @ S @ J, U
        for p, q in pairs:
            S[p, q] = S[q, p] = 0.0
    return S.diagonal()[:n], V[:n, :n]


def davidson(A, diag, guess, D, cyc, conv):
    """lowest roots of the symmetric A (rows of the returned vectors), with the steps of mod_davidson.f90:40-728"""
    nroot, B, AB = len(guess), guess, guess @ A
    H, full, free = AB @ B.T, False, D - len(guess)
    for _ in range(cyc):
        w, V = jacobi(0.5 * (H + H.T))
        order = np.argsort(w, kind="stable")
        ev = w[order[:nroot]]
        C = V[:, order[:nroot + 5 if full else nroot]]
        if full:
            Q, R = np.linalg.qr(C)
            C = Q * np.sign(R.diagonal())
            B, AB = C.T @ B, C.T @ AB
            H, free = AB @ B.T, D - len(B)
            X, AX = B[:nroot], AB[:nroot]
        else:
            X, AX = C.T @ B, C.T @ AB
        X, AX = X / np.linalg.norm(X, axis=1)[:, None], AX / np.linalg.norm(X, axis=1)[:, None]
        res = AX - ev[:, None] * X
        open_ = [k for k in range(nroot) if np.abs(res[k]).max() >= conv]
        if not open_:
            break
        n0 = len(B)
        for k in open_[:free]:
            d = ev[k] - diag
            d = np.where(np.abs(d) < 1e-4, np.where(d < 0.0, -1e-4, 1e-4), d)
            q = res[k] / d
            q /= np.linalg.norm(q)
            for _ in range(2):
                q = q - B.T @ (B @ q)
            B = np.vstack([B, q / np.linalg.norm(q)])
            free -= 1
        full = free == 0
        AB = np.vstack([AB, B[n0:] @ A])
        H = B @ AB.T
    return ev, X


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 8, 15, 19, 20, 31, 32])
def test_eigenvector_signs(n):
    """Values and vectors (sign included) of matrices as Ritz matrices look, full ones, ones of equal diagonal elements
    (rotations of exactly 45 degrees) and ones with zeros.  Rounding of a rotation is 2 eps, and a column takes part in
    one rotation of each of up to about 110 rounds: values within 220 eps |A|, vectors within that over the gap."""
    rng = np.random.default_rng(n)
    for kind in range(4):
        A = rng.standard_normal((n, n))
        A = A + A.T
        if kind == 0:
            A = np.diag(rng.uniform(0.0, 3.0, n)) + 0.05 * A
        elif kind == 2:
            np.fill_diagonal(A, 1.0)
        elif kind == 3:
            A[np.abs(A) < 0.7] = 0.0
        w, V = api.syev(A)
        wr, Vr = jacobi(A)
        scale = np.linalg.norm(A, 2)
        assert np.max(np.abs(w - wr)) < 5e-14 * scale
        gap = np.array([min([abs(wr[k] - wr[j]) for j in range(n) if j != k], default=scale) for k in range(n)])
        err = np.linalg.norm(V - Vr, axis=0)
        assert np.all(err < 5e-14 * scale / gap + 1e-13), (kind, err, gap)


@pytest.mark.parametrize("nmo,nocc_a,roots,seed", [(20, 4, 3, 7), (20, 4, 5, 6), (31, 5, 4, 3), (31, 5, 6, 4),
                                                      (44, 6, 5, 4), (48, 9, 2, 4)])
def test_cis_vectors_keep_their_sign(nmo, nocc_a, roots, seed):
    s = synth.System(nmo=nmo, nocc_a=nocc_a, nocc_b=nocc_a - 2, nirrep=1, seed=seed, roots=roots, skip_abcd=True,
                     run_opts=dict(lowest=1, davidson_conv=8, davidson_cyc=100))
    api.use_torch_stream()
    om, R, _ = api.cis_run(s, api.make_system(s), api.DeviceIntegrals(s), api.make_params(s))
    o, v = int(s.popo.sum()), int(s.popv.sum())
    e1 = (s.eorb[o:][None, :] - s.eorb[:o][:, None]).reshape(-1)
    A = s.ints["iabj"].reshape(o * v, o * v) + np.diag(e1)
    a, i = (x.reshape(-1) for x in np.meshgrid(np.arange(v), np.arange(o)))
    flip = np.nonzero((a >= s.vrta[0]) & (i < s.popa[0]))[0]  # alpha occupied to beta virtual
    low = flip[np.argsort(e1[flip], kind="stable")[:roots]]
    ev, X = davidson(0.5 * (A + A.T), e1, np.eye(o * v)[low], 20, 100, 1e-8)
    assert np.max(np.abs(om - ev)) < 1e-11
    R = R.cpu().numpy().reshape(roots, o * v)
    # converged to 1e-8: the vectors agree to about that over the gap; a flipped sign is a difference of 2
    assert np.max(np.linalg.norm(R - X, axis=1)) < 1e-5, np.sum(R * X, axis=1)


def test_rotations_are_orthogonal_to_rounding():
    """The mean defect |V^T V - 1| over 60 matrices is that of rotations with a correctly rounded c = 1 / sqrt(1 + t^2) and
    s = t c, or less.  (A defect of the rotations stays in the columns and adds up over the steps of a Davidson loop;
    where c and s take the rounding of one reciprocal root apart it is 1.5 times the reference's, restated on the CPU,
    with their correction 0.9 times.  A tenth is left for the reciprocal root of the device.)"""
    rng = np.random.default_rng(0)
    defect = np.zeros(2)
    for _ in range(60):
        A = 0.1 * rng.standard_normal((20, 20)) + np.diag(rng.uniform(0.0, 3.0, 20))
        A = A + A.T
        defect += [np.abs(V.T @ V - np.eye(20)).max() / 60 for V in (api.syev(A)[1], jacobi(A)[1])]
    assert defect[0] <= 1.1 * defect[1], defect
