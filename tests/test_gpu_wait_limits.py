"""The bounded waits of the single-precision Jacobi (a row's step counter) and of the QR's panels (a step's bytes): one that nothing completes gives up after the
limit and reports it, its own kernel's limit being the one that counts; factorisations right after are correct."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _check():
    from tncontract_gb300 import _ops
    rng = np.random.default_rng(0)
    for dt in (np.float32, np.float64):
        A = rng.standard_normal((70, 50)).astype(dt)
        x = torch.from_numpy(A).cuda()
        ref = np.linalg.svd(A.astype(np.float64), compute_uv=False)
        assert np.allclose(_ops.svd(x)[1].cpu().numpy(), ref, rtol=0, atol=800 * np.finfo(dt).eps * ref[0])
        Q, R = (t.cpu().numpy().astype(np.float64) for t in _ops.qr(x))
        assert np.linalg.norm(Q @ R - A) <= 400 * np.finfo(dt).eps * np.linalg.norm(A)


@pytest.mark.parametrize("kind", [3, 4])
def test_wait_runs_out(gpu, kind):
    from tncontract_gb300 import _lib as L
    from tncontract_gb300 import _ops
    try:
        _ops.set_spin_limit(1 << 12)
        assert _ops.wait_selftest(kind) == L.ERR_TIMEOUT
    finally:
        _ops.set_spin_limit(0)
    _check()
