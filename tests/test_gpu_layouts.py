"""Data movement at the sizes where its kernels change shape: the MPO site
product's column split, one short sum per element, checked to a few
roundings."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

DTYPES = [np.float32, np.float64, np.complex64, np.complex128]


def rnd(rng, shape, dt):
    a = rng.standard_normal(shape)
    if np.issubdtype(dt, np.complexfloating):
        a = a + 1j * rng.standard_normal(shape)
    return a.astype(dt)


@pytest.mark.parametrize("dt", DTYPES)
@pytest.mark.parametrize("din,dout,chl,chr_,Dl,Dr", [(2, 2, 1, 9, 1, 3), (2, 2, 127, 43, 3, 3), (3, 2, 5, 129, 5, 1),
                                                     (4, 3, 2, 64, 2, 2), (5, 2, 3, 50, 3, 5), (2, 2, 3, 5, 48, 48)])
def test_mps_mpo_site_shapes(gpu, dt, din, dout, chl, chr_, Dl, Dr):
    from tncontract_gb300 import _ops
    rng = np.random.default_rng(5)
    A, W = rnd(rng, (din, chl, chr_), dt), rnd(rng, (dout, din, Dl, Dr), dt)
    wide = np.complex128 if np.issubdtype(dt, np.complexfloating) else np.float64
    t = np.einsum("plr,opab->olarb", A.astype(wide), W.astype(wide))
    ref = t.reshape(dout, chl * Dl, chr_ * Dr)
    bound = 8 * din * np.finfo(dt).eps * np.max(np.abs(A)) * np.max(np.abs(W))
    for layout in (0, 1):
        out = _ops.mps_mpo_site(torch.from_numpy(A).cuda(), torch.from_numpy(W).cuda(), layout).cpu().numpy()
        assert np.max(np.abs(out - (ref if layout else ref.transpose(1, 0, 2)))) <= bound
