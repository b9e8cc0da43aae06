"""The single-precision Jacobi's rotation is unitary to rounding and without a bias: one pair of rows at a time."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", [np.float32, np.complex64])
def test_rotation_keeps_the_norm(gpu, dt):
    """Bound, in u = eps / 2: c is an ulp off (2 u), s and its product with the rows 5 u more, an entry of the result is
    two products and a sum (3 u), and squared norms double that: 20 u.  The mean of 500 such errors, were they uniform,
    has a deviation of 20 u / sqrt(3 * 500); four of them."""
    from tncontract_gb300 import _ops
    rng = np.random.default_rng(5)
    drift = []
    for _ in range(500):
        a = rng.standard_normal((2, 24)) + (1j * rng.standard_normal((2, 24)) if np.issubdtype(dt, np.complexfloating) else 0)
        a[1] = a[1] * 10.0 ** rng.uniform(-1.5, 0.2) + a[0] * rng.uniform(-1, 1)
        a = a.astype(dt)
        W, S, _o, info = _ops.svd_rows(torch.from_numpy(a).cuda(), block_rows=8)
        assert info.cpu().tolist()[0] == 0
        W = W.cpu().numpy().astype(np.complex128)
        n0 = np.linalg.norm(a.astype(np.complex128)) ** 2
        drift.append((np.linalg.norm(W) ** 2 - n0) / n0 / (np.finfo(dt).eps / 2))
        assert abs(np.vdot(W[0], W[1])) <= 64 * np.finfo(dt).eps * np.linalg.norm(W[0]) * np.linalg.norm(W[1])
        ref = np.linalg.svd(a.astype(np.complex128), compute_uv=False)
        assert np.max(np.abs(S.cpu().numpy() - ref)) <= 16 * np.finfo(dt).eps * ref[0]
    assert np.max(np.abs(drift)) <= 20, np.max(np.abs(drift))
    assert abs(np.mean(drift)) <= 4 * 20 / np.sqrt(3 * 500), np.mean(drift)
