"""Clustered spectra in the refined FP64 SVD (24 to 512 rows): what its steps leave to the FP64 Jacobi starts from a
unitary J, and pairs that already meet the tolerance are not left to it."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _matrix(n, s, dt, seed):
    rng = np.random.default_rng(seed)

    def unitary():
        a = rng.standard_normal((n, n))
        if np.issubdtype(dt, np.complexfloating):
            a = a + 1j * rng.standard_normal((n, n))
        return np.linalg.qr(a)[0]
    return ((unitary() * s) @ unitary().conj().T).astype(dt)


@pytest.mark.parametrize("dt", [np.float64, np.complex128])
@pytest.mark.parametrize("n,size,gap", [(40, 5, 1e-4), (64, 16, 1e-6), (97, 30, 1e-5), (130, 130, 1e-6), (64, 64, 1e-12)])
def test_cluster(gpu, dt, n, size, gap):
    """`size` values within `gap` of one another beside generic ones.  Bounds: 8 n eps, as for other spectra."""
    from tncontract_gb300 import _ops
    s = np.sort(np.concatenate([1.0 + gap * np.linspace(0, 1, size), np.linspace(0.2, 0.9, n - size)]))[::-1]
    A = _matrix(n, s, dt, n)
    U, S, V = (t.cpu().numpy() for t in _ops.svd(torch.from_numpy(A).cuda()))
    tol = 8 * n * np.finfo(dt).eps
    assert np.max(np.abs(S - np.linalg.svd(A, compute_uv=False))) <= tol
    assert np.max(np.abs(U.conj().T @ U - np.eye(n))) <= tol
    assert np.max(np.abs(V @ V.conj().T - np.eye(n))) <= tol
    assert np.linalg.norm((U * S) @ V - A) <= tol * np.linalg.norm(A)


@pytest.mark.parametrize("dt", [np.float64, np.complex128])
@pytest.mark.parametrize("tol", [1e-8, 3e-8, 1e-7])
def test_equal_pair_below_the_tolerance(gpu, dt, tol):
    """Two equal values whose rows meet a caller's tolerance while others do not: their angle is large but nothing has to
    be rotated, so the steps finish the work.  info[1] counts the sweeps of the Jacobi that ended it: the
    single-precision one's (five or more from a random matrix), not the FP64 one's (one or two after the steps)."""
    from tncontract_gb300 import _ops
    n = 48
    s = np.linspace(0.1, 2.0, n)[::-1].copy()
    s[1] = s[0]
    for seed in range(12):
        infos = []
        A = _matrix(n, s, dt, 100 + seed)
        _ops.svd(torch.from_numpy(A).cuda(), tol=tol, info_out=infos)
        assert infos[0].cpu().tolist()[0] == 0
        assert infos[0].cpu().tolist()[1] >= 4, (seed, infos[0].cpu().tolist())


@pytest.mark.parametrize("dt", [np.float64, np.complex128])
@pytest.mark.parametrize("tol", [1e-10, 1e-8, 3e-8, 1e-7])
@pytest.mark.parametrize("n", [24, 48, 100])
def test_loose_tolerance(gpu, dt, tol, n):
    """A caller's loose tolerance is one on the rows' orthogonality: the accumulated factor stays unitary to rounding, and
    the singular values are second order in the tolerance (8 n tol^2 beside the usual 8 n eps)."""
    from tncontract_gb300 import _ops
    s = np.linspace(0.1, 2.0, n)[::-1].copy()
    s[1] = s[0]
    for shape in ("square", "tall"):
        A = _matrix(n, s, dt, n)
        if shape == "tall":
            A = np.linalg.qr(_matrix(2 * n, np.ones(2 * n), dt, 1)[:, :n])[0] @ A
        U, S, V = (t.cpu().numpy() for t in _ops.svd(torch.from_numpy(A).cuda(), tol=tol))
        assert np.max(np.abs(S - s)) <= 8 * n * (np.finfo(dt).eps + tol * tol)
        # the accumulated side: VH of a tall or square matrix is normalised rows or J, U the other
        both = [np.max(np.abs(U.conj().T @ U - np.eye(n))), np.max(np.abs(V @ V.conj().T - np.eye(n)))]
        assert min(both) <= 8 * n * np.finfo(dt).eps, both
        assert max(both) <= 2 * tol + 8 * n * np.finfo(dt).eps, both
        assert np.linalg.norm((U * S) @ V - A) <= 16 * n * np.finfo(dt).eps * np.linalg.norm(A)


@pytest.mark.parametrize("dt", [np.float64, np.complex128])
@pytest.mark.parametrize("tol", [1.5e-9, 3e-9])
def test_rule_of_the_steps(gpu, dt, tol):
    """A triangular matrix (its QR changes nothing) with one pair of rows of equal norm just below the tolerance, whose angle
    is large, and a dozen rows of nearly equal norms above it, whose angles (up to 8.5e-4) take a second step; all too
    nearly orthogonal for the single-precision Jacobi to rotate.  The steps end the work, and info[1] is that Jacobi's one
    sweep; the FP64 Jacobi would have counted two, one that rotates and one that finds nothing."""
    from tncontract_gb300 import _ops
    n, m, below = 40, 12, 0.9
    phase = np.exp(0.7j) if np.issubdtype(dt, np.complexfloating) else 1.0
    R = np.diag(np.linspace(2.0, 0.5, n)).astype(dt)
    R[0, 1] = phase * below * tol * abs(R[0, 0])
    R[1, 1] = np.sqrt(abs(R[0, 0]) ** 2 + abs(R[0, 1]) ** 2)
    size, g, t = abs(R[2, 2]), 2.772e-6, 8.5e-4
    for i in range(m):
        R[2 + i, 2 + i] = size * np.sqrt(1 - g / t * i)
        R[2 + i, 3 + i:2 + m] = phase * g * R[2 + i, 2 + i]
    infos = []
    U, S, V = (t.cpu().numpy() for t in _ops.svd(torch.from_numpy(np.ascontiguousarray(R.conj().T)).cuda(), tol=tol,
                                                 info_out=infos))
    assert infos[0].cpu().tolist()[:3] == [0, 1, 0]
    assert np.max(np.abs(S - np.linalg.svd(R, compute_uv=False))) <= 8 * n * np.finfo(dt).eps + 2 * below * tol
    assert np.linalg.norm((U * S) @ V - R.conj().T) <= 16 * n * np.finfo(dt).eps * np.linalg.norm(R)
