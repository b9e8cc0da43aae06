"""tnc_svd where its route changes: row counts on both sides of the refinement's
smallest and largest, odd and unaligned ones, and of the single-precision Jacobi's
row widths; wide and tall; generic, graded, repeated and vanishing singular values;
norms near the ends of FP64's squares.

Bounds: the factors come from products of n terms (n eps, worst case) on rows
orthogonal to sqrt(n) eps (4 sqrt(n) eps in single precision): 8 n eps covers
both.  Singular vectors of vanishing values are not determined and not checked."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _matrix(m, n, dt, kind):
    rng = np.random.default_rng(m * 1000 + n)
    k = min(m, n)

    def rnd(*s):
        a = rng.standard_normal(s)
        return a + 1j * rng.standard_normal(s) if np.issubdtype(dt, np.complexfloating) else a
    if kind == "random":
        return rnd(m, n).astype(dt)
    j = np.arange(k)
    s = {"graded": np.exp(-10.0 * j / k), "steep": np.exp(-33.0 * j / k), "repeated": 3.0 - j * 4 // k * 0.5,
         "deficient": np.where(j < k // 2, 2.0 - j / k, 0.0), "large": 1e150 * np.exp(-5.0 * j / k),
         "small": 1e-140 * np.exp(-5.0 * j / k)}[kind]
    return ((np.linalg.qr(rnd(m, k))[0] * s) @ np.linalg.qr(rnd(n, k))[0].conj().T).astype(dt)


def _check(A):
    from tncontract_gb300 import _ops
    U, S, V = (t.cpu().numpy() for t in _ops.svd(torch.from_numpy(A).cuda()))
    wide = np.complex128 if np.iscomplexobj(A) else np.float64
    A, U, S, V = A.astype(wide), U.astype(wide), S.astype(np.float64), V.astype(wide)
    s0 = np.linalg.svd(A, compute_uv=False)
    return A, U, S, V, s0


@pytest.mark.parametrize("dt", [np.float32, np.complex64, np.float64, np.complex128])
@pytest.mark.parametrize("m,n", [(23, 23), (24, 24), (25, 31), (48, 33), (63, 64), (65, 65), (128, 130), (129, 129), (200, 257),
                                 (257, 256), (511, 513), (513, 520)])
def test_sizes(gpu, dt, m, n):
    A, U, S, V, s0 = _check(_matrix(m, n, dt, "random"))
    tol = 8 * max(m, n) * np.finfo(dt).eps
    k = min(m, n)
    assert np.max(np.abs(S - s0)) <= tol * s0[0]
    assert np.linalg.norm((U * S) @ V - A) <= tol * np.linalg.norm(A)
    assert np.max(np.abs(U.conj().T @ U - np.eye(k))) <= tol and np.max(np.abs(V @ V.conj().T - np.eye(k))) <= tol


@pytest.mark.parametrize("dt", [np.float64, np.complex128])
@pytest.mark.parametrize("m,n", [(24, 24), (64, 70), (97, 60), (160, 160)])
@pytest.mark.parametrize("kind", ["graded", "steep", "repeated", "deficient", "large", "small"])
def test_spectra(gpu, dt, m, n, kind):
    A, U, S, V, s0 = _check(_matrix(m, n, dt, kind))
    tol = 8 * max(m, n) * np.finfo(dt).eps
    k = min(m, n) // 2 if kind == "deficient" else min(m, n)
    scale = s0[0]
    assert np.max(np.abs(S - s0)) <= tol * scale
    assert np.linalg.norm((U * (S / scale)) @ V - A / scale) <= tol * np.linalg.norm(A / scale)
    if kind != "steep":  # its last values are at the noise floor
        assert np.max(np.abs(U[:, :k].conj().T @ U[:, :k] - np.eye(k))) <= tol
        assert np.max(np.abs(V[:k] @ V[:k].conj().T - np.eye(k))) <= tol


@pytest.mark.parametrize("bad", [np.nan, np.inf])
def test_nonfinite(gpu, bad):
    from tncontract_gb300 import _ops
    A = _matrix(40, 40, np.float64, "random")
    A[3, 5] = bad
    with pytest.raises(ValueError):
        _ops.svd(torch.from_numpy(A).cuda())


def test_cap(gpu):
    """A caller's small sweep cap is still reported when it is reached, in every precision."""
    from tncontract_gb300 import _ops
    for dt in (np.float32, np.float64):
        infos = []
        with pytest.raises(np.linalg.LinAlgError):
            _ops.svd(torch.from_numpy(_matrix(40, 40, dt, "random")).cuda(), max_sweeps=2, info_out=infos)
        assert infos[0].cpu().tolist()[:2] == [2, 2]
