"""The FP64 GEMM's tile shapes: sizes at the edges of the 8 x 16, 16 x 16 and
32 x 32 tiles and on both sides of the lines between them, ragged K, every
operand layout, batches.  Bound: (k + 2) roundings of |A| |B| per term of a real
sum, twice that in complex."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SIZES = [(1, 1, 1), (7, 15, 3), (8, 16, 16), (9, 17, 17), (32, 32, 16), (33, 31, 15), (100, 97, 33), (208, 192, 40), (513, 291, 18),
         (700, 660, 5)]


@pytest.mark.parametrize("dt", [np.float64, np.complex128])
@pytest.mark.parametrize("m,n,k", SIZES)
def test_wide_gemm_tiles(gpu, dt, m, n, k):
    from tncontract_gb300 import _lib as L
    from tncontract_gb300 import _ops
    rng = np.random.default_rng(7)
    cplx = dt is np.complex128

    def rnd(*shape):
        a = rng.standard_normal(shape)
        return (a + 1j * rng.standard_normal(shape) if cplx else a).astype(dt)
    ops = {L.OP_N: lambda x: x, L.OP_T: lambda x: x.T, L.OP_C: lambda x: np.conj(x).T, L.OP_R: np.conj}
    batch = 3 if m * n < 20000 else 1
    for opA, opB in [(L.OP_N, L.OP_N), (L.OP_T, L.OP_N), (L.OP_N, L.OP_C), (L.OP_C, L.OP_T), (L.OP_R, L.OP_R)]:
        A = rnd(batch, *((k, m) if opA in (L.OP_T, L.OP_C) else (m, k)))
        B = rnd(batch, *((n, k) if opB in (L.OP_T, L.OP_C) else (k, n)))
        C0 = rnd(batch, m, n)
        Cd = torch.from_numpy(C0.copy()).cuda()
        _ops.gemm(opA, opB, m, n, k, torch.from_numpy(A).cuda(), A.shape[2], torch.from_numpy(B).cuda(), B.shape[2], Cd, n,
                  alpha=0.5, beta=2.0, batch=batch, sA=A[0].size, sB=B[0].size, sC=m * n)
        got = Cd.cpu().numpy()
        for b in range(batch):
            a, bm = ops[opA](A[b]), ops[opB](B[b])
            want = 0.5 * (a @ bm) + 2.0 * C0[b]
            bound = (4 * k + 8) * 2.0 ** -52 * (0.5 * np.abs(a) @ np.abs(bm) + 2.0 * np.abs(C0[b]))
            assert np.all(np.abs(got[b] - want) <= bound), (opA, opB, b)
