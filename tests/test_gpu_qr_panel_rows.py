"""QR at the row counts where the panel's rows a lane and its CTAs change (single precision)."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

EDGES = [128, 129, 256, 257, 384, 385, 512, 513, 768, 769, 1024, 1025, 1280, 1281, 1536, 1537, 1792, 1793]


@pytest.mark.parametrize("dt", [np.float32, np.complex64])
@pytest.mark.parametrize("m", EDGES)
def test_qr_panel_rows(gpu, dt, m):
    """Two panels, the second of 64 rows less: A = Q R and orthonormal Q to a few roundings per step, R from tnc_qr_r the
    same bits."""
    from tncontract_gb300 import _ops
    n = 70
    rng = np.random.default_rng(m)
    A = rng.standard_normal((m, n))
    if np.issubdtype(dt, np.complexfloating):
        A = A + 1j * rng.standard_normal((m, n))
    A = A.astype(dt)
    x = torch.from_numpy(A).cuda()
    Q, R = _ops.qr(x)
    assert torch.equal(R, _ops.qr_r(x))
    Q, R = Q.cpu().numpy(), R.cpu().numpy()
    wide = A.astype(np.complex128 if np.issubdtype(dt, np.complexfloating) else np.float64)
    bound = 4 * np.finfo(dt).eps * np.sqrt(m * n)
    assert np.linalg.norm(Q.astype(wide.dtype) @ R - wide) <= bound * np.linalg.norm(wide)
    assert np.linalg.norm(np.conj(Q).T @ Q - np.eye(n)) <= bound * np.sqrt(n)
    assert np.all(np.tril(R, -1) == 0)
