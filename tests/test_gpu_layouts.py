"""Data movement at the sizes where its kernels change shape: the permute's
boxes (short and kept inner axes, cut boxes, every rank), and the MPO site
product's column split.  Moves are exact; the site product is one short sum per
element, checked to a few roundings."""
import itertools

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


SHAPES = [(2,), (1025,), (3, 17), (16, 33), (17, 16), (31, 3, 31), (2, 2, 2, 2, 2, 2, 2, 2), (40, 2, 3, 50), (65, 3, 2, 33),
          (5, 64, 3), (3, 5, 31), (1, 7, 1, 129), (257, 2, 130), (33, 2, 33, 2), (2, 1000, 2)]


@pytest.mark.parametrize("dt", DTYPES)
@pytest.mark.parametrize("shape", SHAPES)
def test_permute_boxes(gpu, dt, shape):
    from tncontract_gb300 import _ops
    a = rnd(np.random.default_rng(3), shape, dt)
    perms = list(itertools.permutations(range(len(shape))))
    if len(perms) > 24:
        perms = [perms[i] for i in np.random.default_rng(4).integers(0, len(perms), 12)]
    x = torch.from_numpy(a).cuda()
    for perm in perms:
        for conj in (False, True):
            out = _ops.permute(x, perm, conj=conj).cpu().numpy()
            ref = np.transpose(a, perm)
            assert np.array_equal(out, np.conj(ref) if conj else ref), (shape, perm, conj)


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
