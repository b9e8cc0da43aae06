"""The panelled QR at the edges of its panels (16, 32 or 64 columns by type),
register tiles (32 rows a CTA and multiples), cluster sizes and row loops, and
past its 4096 rows, against LAPACK in double precision."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

DTYPES = [np.float32, np.float64, np.complex64, np.complex128]
SHAPES = [(1, 1), (1, 40), (15, 16), (17, 16), (31, 33), (33, 31), (64, 64), (65, 65), (129, 15), (257, 80), (512, 17), (513, 65),
          (700, 130), (1025, 33), (1537, 96), (2049, 40), (4096, 20), (4097, 20), (40, 600), (130, 2000)]


def rnd(rng, shape, dt):
    a = rng.standard_normal(shape)
    if np.issubdtype(dt, np.complexfloating):
        a = a + 1j * rng.standard_normal(shape)
    return a.astype(dt)


@pytest.mark.parametrize("dt", DTYPES)
@pytest.mark.parametrize("shape", SHAPES)
def test_qr_panel_edges(gpu, dt, shape):
    """A = Q R with orthonormal Q to a few roundings per step; R with LAPACK's signs (a real diagonal of the sign opposite to
    the column's leading entry); R from tnc_qr_r the same bits."""
    from tncontract_gb300 import _ops
    m, n = shape
    k = min(m, n)
    A = rnd(np.random.default_rng(m + 7 * n), shape, dt)
    x = torch.from_numpy(A).cuda()
    Q, R = _ops.qr(x)
    R2 = _ops.qr_r(x)
    assert torch.equal(R, R2)
    Q, R = Q.cpu().numpy(), R.cpu().numpy()
    wide = A.astype(np.complex128 if np.issubdtype(dt, np.complexfloating) else np.float64)
    eps = np.finfo(dt).eps
    bound = 4 * eps * np.sqrt(m) * np.sqrt(k)
    assert np.linalg.norm(Q @ R - wide) <= bound * np.linalg.norm(wide)
    assert np.linalg.norm(np.conj(Q).T @ Q - np.eye(k)) <= bound * np.sqrt(k)
    assert np.all(np.tril(R, -1) == 0)
    _, Rl = np.linalg.qr(wide)
    # R is determined up to the conditioning of A's columns
    cond = np.linalg.cond(wide[:, :k])
    assert np.linalg.norm(R - Rl) <= bound * 10 * cond * np.linalg.norm(Rl)


@pytest.mark.parametrize("dt", DTYPES)
def test_qr_panel_reduced_columns(gpu, dt):
    """Columns that need no reflector (already reduced, zero), a repeated column and scales over 200 decades (double) or 20
    (single), at panel edges."""
    from tncontract_gb300 import _ops
    A = rnd(np.random.default_rng(8), (300, 90), dt)
    for c in (0, 16, 31, 32, 64):
        A[:, c] = 0
    A[0, 0] = 2
    A[:, 63] = A[:, 5]
    A[:, 70:80] *= 1e-100 if np.finfo(dt).eps < 1e-10 else 1e-10
    Q, R = (t.cpu().numpy() for t in _ops.qr(torch.from_numpy(A).cuda()))
    bound = 4 * np.finfo(dt).eps * np.sqrt(300 * 90)
    assert np.linalg.norm(np.conj(Q).T @ Q - np.eye(90)) <= bound * np.sqrt(90)
    wide = A.astype(np.complex128 if np.issubdtype(dt, np.complexfloating) else np.float64)
    err = np.linalg.norm(Q @ R.astype(wide.dtype) - wide, axis=0)
    assert np.all(err <= bound * np.linalg.norm(wide, axis=0))
