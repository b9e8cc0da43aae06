"""The QR of more rows than the panels take (4096): its blocked form (128 columns or more: panels by the dataflow kernel,
products split over the rows, triangular solves against V^H V), at and beyond its first sizes, ragged blocks, and the R
factor alone of an adjoint."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DTYPES = [np.float32, np.float64, np.complex64, np.complex128]


def rnd(shape, dt):
    rng = np.random.default_rng(shape[0] + 7 * shape[1])
    a = rng.standard_normal(shape)
    if np.issubdtype(dt, np.complexfloating):
        a = a + 1j * rng.standard_normal(shape)
    return a.astype(dt)


@pytest.mark.parametrize("dt", DTYPES)
@pytest.mark.parametrize("shape", [(4097, 128), (4200, 200), (4500, 129), (5000, 64)])
def test_long(gpu, dt, shape):
    """Bounds as for the panels (test_gpu_qr_panels.py): a few roundings a step."""
    from tncontract_gb300 import _ops
    m, k = shape
    A = rnd(shape, dt)
    A[:, 7] = 0  # a column that needs no reflector
    x = torch.from_numpy(A).cuda()
    Q, R = _ops.qr(x)
    assert torch.equal(R, _ops.qr_r(x))
    Q, R = Q.cpu().numpy(), R.cpu().numpy()
    wide = A.astype(np.complex128 if np.issubdtype(dt, np.complexfloating) else np.float64)
    bound = 4 * np.finfo(dt).eps * np.sqrt(m) * np.sqrt(k)
    assert np.linalg.norm(Q @ R.astype(wide.dtype) - wide) <= bound * np.linalg.norm(wide)
    assert np.linalg.norm(np.conj(Q).T @ Q - np.eye(k)) <= bound * np.sqrt(k)
    assert np.all(np.tril(R, -1) == 0)


@pytest.mark.parametrize("dt", DTYPES)
def test_long_adjoint(gpu, dt):
    from tncontract_gb300 import _ops
    x = torch.from_numpy(rnd((200, 4300), dt)).cuda()
    R = _ops.qr_r(x, adjoint=True)
    _, R2 = _ops.qr(x.conj().resolve_conj().T.contiguous())
    assert torch.equal(R, R2)
