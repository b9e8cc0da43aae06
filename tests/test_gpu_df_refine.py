"""The finish's whole-matrix steps: rows that are nearly orthogonal (the state the
single-precision stage leaves), with an isolated pair of nearly equal norms (rotated
by itself), a cluster of three (left to the Jacobi), discarded rows, on both sides of
the smallest row count, at ragged sizes and the longest rows.

Bounds: W = Q A with Q unitary to the finish's 48 bits (sums of n terms: n 2^-46),
every pair orthogonal to the tolerance 1e-7 (a step accepted without a look leaves
less), separated values to the same n 2^-46 of the largest."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
TOL = 1e-7


def _near(seed, m, n, cplx, kind):
    rng = np.random.default_rng(seed)
    dt = np.complex64 if cplx else np.float32

    def rnd(*s):
        a = rng.standard_normal(s)
        return a + 1j * rng.standard_normal(s) if cplx else a
    v = np.linalg.qr(rnd(n, m))[0].conj().T
    s = np.exp(-3.0 * np.arange(m) / m)
    if kind == "pair":
        s[5] = s[4] * (1 + 1e-6)
    if kind == "three":
        s[5], s[6] = s[4] * (1 + 1e-6), s[4] * (1 - 2e-6)
    mix = np.eye(m) + 2e-6 * rnd(m, m)
    return (s[:, None] * (mix @ v)).astype(dt)


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("kind", ["plain", "pair", "three"])
@pytest.mark.parametrize("m,n", [(23, 40), (24, 24), (33, 65), (100, 301), (256, 256), (257, 512)])
def test_finish(gpu, cplx, kind, m, n):
    from tncontract_gb300 import _ops
    A = _near(m, m, n, cplx, kind)
    W, S, order, info = _ops.svd_rows_df(torch.from_numpy(A).cuda(), tol=TOL)
    assert info.cpu().tolist()[0] == 0
    W, S = W.cpu().numpy(), S.cpu().numpy()
    A = A.astype(W.dtype)
    bound = n * 2.0 ** -46
    assert np.linalg.norm(W.conj().T @ W - A.conj().T @ A) <= 4 * bound * np.linalg.norm(A) ** 2
    nrm = np.linalg.norm(W, axis=1)
    G = np.abs(W @ W.conj().T) / np.outer(nrm, nrm)
    np.fill_diagonal(G, 0.0)
    assert G.max() <= TOL
    if kind == "plain":  # what is left of a pair counts to second order over the gap, so not in a cluster
        s0 = np.linalg.svd(A, compute_uv=False)
        assert np.max(np.abs(S - s0)) <= (4 * bound + m * TOL ** 2) * s0[0]
    assert np.all(np.diff(S) <= 0) and np.allclose(S, nrm[order.cpu().numpy()], rtol=1e-12)


@pytest.mark.parametrize("cplx,m,n", [(True, 768, 800), (True, 770, 800), (False, 1024, 1100), (False, 1030, 1100)])
def test_longest(gpu, cplx, m, n):
    test_finish(gpu, cplx, "plain", m, n)


@pytest.mark.parametrize("cplx,n", [(False, 1024), (True, 512)])
def test_keep(gpu, cplx, n):
    """Rows from nkeep on are orthogonal to the kept ones; equal norms among them are no concern."""
    from tncontract_gb300 import _ops
    m, keep = 60, 40
    A = _near(1, m, n, cplx, "plain")
    A[keep:] = A[keep:] / np.linalg.norm(A[keep:], axis=1)[:, None] * np.linalg.norm(A[keep])
    W, S, order, info = _ops.svd_rows_df(torch.from_numpy(A).cuda(), tol=TOL, nkeep=keep)
    assert info.cpu().tolist()[0] == 0
    W = W.cpu().numpy()
    nrm = np.linalg.norm(W, axis=1)
    G = np.abs(W @ W.conj().T) / np.outer(nrm, nrm)
    np.fill_diagonal(G, 0.0)
    G[keep:, keep:] = 0.0
    assert G.max() <= TOL
    A = A.astype(W.dtype)
    assert np.linalg.norm(W.conj().T @ W - A.conj().T @ A) <= 4 * n * 2.0 ** -46 * np.linalg.norm(A) ** 2
