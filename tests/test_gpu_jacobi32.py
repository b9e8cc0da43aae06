"""The single-precision block Jacobi at the edges of its half-blocks (ragged and
missing rows, an odd number of half-blocks, one half-block) and row lengths
(lane pieces, unaligned rows, each register width), every half-block height, and
with rows beyond nkeep left alone among themselves.

Bounds: a row takes part in about nr rotations a sweep and ten sweeps, each
leaving an error of about 4 eps of the pair: sqrt(12 nr) 4 eps |A|_F on the
singular values (random signs).  Converged pairs meet the tolerance 4 sqrt(L) eps
up to the rounding of the inner product itself, taken as as much again."""
import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -23


def _rows(seed, m, n, dt):
    rng = np.random.default_rng(seed)
    a = rng.standard_normal((m, n))
    if np.issubdtype(dt, np.complexfloating):
        a = a + 1j * rng.standard_normal((m, n))
    return (a * np.exp(-3.0 * np.arange(m) / m)[:, None]).astype(dt)


def _check(A, W, S, keep=None):
    m, n = A.shape
    wide = np.complex128 if np.iscomplexobj(A) else np.float64
    W = W.astype(wide)
    s0 = np.linalg.svd(A.astype(wide), compute_uv=False)
    tol = 2 * 4 * np.sqrt(max(n, 8)) * EPS
    nrm = np.linalg.norm(W, axis=1)
    G = np.abs(W @ W.conj().T) / np.maximum(np.outer(nrm, nrm), 1e-30)
    np.fill_diagonal(G, 0.0)
    if keep is not None:
        G[keep:, keep:] = 0.0
    else:
        assert np.max(np.abs(np.sort(S)[::-1] - s0)) <= np.sqrt(12 * m) * 4 * EPS * np.linalg.norm(A)
    assert np.max(G) <= tol


SHAPES = [(1, 1), (2, 2), (3, 7), (5, 5), (8, 8), (9, 33), (16, 127), (17, 128), (24, 129), (33, 256), (40, 257), (63, 63),
          (65, 511), (130, 512), (20, 513), (18, 1024)]


@pytest.mark.parametrize("dt", [np.float32, np.complex64])
@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("block_rows", [2, 4, 8, 16])
def test_rows(gpu, dt, shape, block_rows):
    from tncontract_gb300 import _ops
    A = _rows(sum(shape), *shape, dt)
    W, S, order, info = _ops.svd_rows(torch.from_numpy(A).cuda(), block_rows=block_rows)
    assert info.cpu().tolist()[0] == 0
    _check(A, W.cpu().numpy(), S.cpu().numpy())


@pytest.mark.parametrize("dt", [np.float32, np.complex64])
@pytest.mark.parametrize("nkeep", [1, 8, 13])
def test_rows_keep(gpu, dt, nkeep):
    from tncontract_gb300 import _ops
    m, n, h = 37, 50, 4
    A = torch.from_numpy(_rows(nkeep, m, n, dt)).cuda()
    W, S = torch.empty_like(A), torch.empty(m, dtype=torch.float32, device="cuda")
    order, info = torch.empty(m, dtype=torch.int64, device="cuda"), torch.empty(4, dtype=torch.int32, device="cuda")
    sz = C.c_size_t()
    _ops._call("tnc_svd_rows_workspace_size", _ops.code(A.dtype), m, n, C.byref(sz))
    ws = _ops.workspace(sz.value)
    _ops._call("tnc_svd_rows_keep", _ops.code(A.dtype), m, n, _ops._p(A), _ops._p(W), _ops._p(S), _ops._p(order), 0, 0.0, h,
               nkeep, _ops._p(ws), sz.value, _ops._p(info), _ops._stream())
    assert info.cpu().tolist()[0] == 0
    keep = -(-nkeep // h) * h
    _check(A.cpu().numpy(), W.cpu().numpy(), S.cpu().numpy(), keep)
