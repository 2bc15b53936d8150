"""The sweep of the device eigensolver in NumPy (molgw_b200/csrc/eigh_jacobi.cu): every entry
inside a block is rotated in the first round of a sweep only, the other rounds rotate the
entries between the two blocks of a pair.  It converges to LAPACK's eigenpairs, no further from
them than rotating everything in every round, in up to two sweeps more; matrices of low rank, which
contour deformation meets when there are fewer transitions than auxiliary functions, take up to
four more (15 to 19 at n = 512, rank 240), each of about half the work."""
import numpy as np
import pytest

from tests.test_block_jacobi_model import KB, KS, block_jacobi, inner_sweep, rr_pair


def cross_sweep(S, tau):
    Q = np.eye(KS)
    for r in range(KB):
        a = np.arange(KB)
        b = KB + ((a + r) & (KB - 1))
        apq = S[a, b]
        rot = np.abs(apq) > tau
        d, p2 = S[b, b] - S[a, a], 2.0 * apq
        t = np.where(rot, p2 / np.where(rot, d + np.copysign(np.sqrt(d * d + p2 * p2), d), 1.0), 0.0)
        c = np.where(rot, 1.0 / np.sqrt(t * t + 1.0), 1.0)
        G = np.eye(KS)
        G[a, a], G[a, b], G[b, a], G[b, b] = c, t * c, -t * c, c
        S = G.T @ S @ G
        S = 0.5 * (S + S.T)
        Q = Q @ G
    return Q


def block_jacobi_cross(A, max_sweeps=60):
    n = A.shape[0]
    nb, A, V = n // KB, A.copy(), np.eye(n)
    tau = 1e-14 * np.linalg.norm(A)
    for sweep in range(1, max_sweeps + 1):
        rotated = False
        for r in range(nb - 1):
            J = np.eye(n)
            for k in range(nb // 2):
                I, Jb = rr_pair(r, k, nb)
                idx = np.r_[I * KB:(I + 1) * KB, Jb * KB:(Jb + 1) * KB]
                S = A[np.ix_(idx, idx)]
                off = S - np.diag(np.diag(S)) if r == 0 else S[:KB, KB:]
                if np.abs(off).max() <= tau:
                    continue
                rotated = True
                J[np.ix_(idx, idx)] = inner_sweep(S, 0.25 * tau)[1] if r == 0 else cross_sweep(S, 0.25 * tau)
            A = J.T @ A @ J
            A = 0.5 * (A + A.T)
            V = V @ J
        if not rotated:
            return np.diag(A).copy(), V, sweep
    raise RuntimeError("no convergence")


@pytest.mark.parametrize("n", [64, 128, 256])
@pytest.mark.parametrize("decades", [0.0, 4.0])
@pytest.mark.parametrize("rank", [3.0, 0.8, 0.24])
def test_cross_sweeps_converge(n, decades, rank):
    rng = np.random.default_rng(n)
    k = int(rank * n)
    X = rng.standard_normal((n, k)) * 10.0 ** (-decades * rng.random((n, 1)))
    A = -(X @ X.T) / k
    lam, V, sweeps = block_jacobi_cross(A)
    ref = np.linalg.eigvalsh(A)
    scale = np.abs(ref).max()
    # rounding of the rotations: about sweeps x n of them act on every entry, 2^-53 sqrt(2 n sweeps)
    tol = 20 * 2.0 ** -53 * np.sqrt(2.0 * n * sweeps)
    assert np.abs(np.sort(lam) - ref).max() < tol * scale
    assert np.abs(V.T @ V - np.eye(n)).max() < tol
    assert np.abs(A @ V - V * lam).max() < 2e-12 * scale
    lam_all, V_all, sweeps_all = block_jacobi(A)
    assert sweeps <= sweeps_all + (2 if rank > 1.0 else 4)
    for err, err_all in ((np.sort(lam) - ref, np.sort(lam_all) - ref),
                         (V.T @ V - np.eye(n), V_all.T @ V_all - np.eye(n))):
        assert np.linalg.norm(err) <= 1.2 * np.linalg.norm(err_all) + 1e-15
