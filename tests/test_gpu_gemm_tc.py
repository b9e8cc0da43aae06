"""The tensor-core GEMM over the edges of its K slices and of the groups of three that
it sums in tensor memory, ragged rows, every operand layout (contiguous rows in pairs
and alone, strided rows), batches, digits at their largest, and rows of very
different size.

Bound: cutting at the third digit and dropping the products below it leaves at most
2^-23 of 2^(ea + eb) a term, 2^e at most twice the row's largest component (four
times that sum in complex); the FP32 sums round (k / 192 + 3) times."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SHAPES = [(64, 64, 33), (65, 130, 64), (128, 128, 65), (100, 70, 191), (129, 65, 192), (70, 200, 193), (64, 64, 385), (200, 64, 577),
          (300, 129, 128)]


@pytest.mark.parametrize("dt", [np.float32, np.complex64])
@pytest.mark.parametrize("m,n,k", SHAPES)
def test_tc(gpu, dt, m, n, k):
    from tncontract_gb300 import _lib as L
    from tncontract_gb300 import _ops
    rng = np.random.default_rng(m + n + k)
    cplx = dt is np.complex64
    wide = np.complex128 if cplx else np.float64

    def rnd(*shape):
        a = rng.standard_normal(shape)
        if cplx:
            a = a + 1j * rng.standard_normal(shape)
        a *= np.exp(8 * rng.standard_normal((shape[0], shape[1], 1)))  # rows of very different size
        if k % 2:  # digits at their largest
            a = np.sign(a.real) * 0.99999994 * (1 + 1j if cplx else 1)
        return a.astype(dt)
    ops = {L.OP_N: lambda x: x, L.OP_T: lambda x: x.T, L.OP_C: lambda x: np.conj(x).T, L.OP_R: np.conj}
    batch = 2
    for opA, opB in [(L.OP_N, L.OP_N), (L.OP_T, L.OP_C), (L.OP_C, L.OP_T), (L.OP_R, L.OP_R)]:
        A = rnd(batch, *((k, m) if opA in (L.OP_T, L.OP_C) else (m, k)))
        B = rnd(batch, *((n, k) if opB in (L.OP_T, L.OP_C) else (k, n)))
        C0 = rnd(batch, m, n)
        Cd = torch.from_numpy(C0.copy()).cuda()
        _ops.gemm(opA, opB, m, n, k, torch.from_numpy(A).cuda(), A.shape[2], torch.from_numpy(B).cuda(), B.shape[2], Cd, n,
                  alpha=2.0, beta=0.5, batch=batch, sA=A[0].size, sB=B[0].size, sC=m * n, tc=True)
        got = Cd.cpu().numpy()
        for b in range(batch):
            a, bm = ops[opA](A[b]).astype(wide), ops[opB](B[b]).astype(wide)
            want = 2.0 * (a @ bm) + 0.5 * C0[b]
            big = np.outer(np.max(np.maximum(np.abs(a.real), np.abs(a.imag)), axis=1),
                           np.max(np.maximum(np.abs(bm.real), np.abs(bm.imag)), axis=0))
            bound = 2.0 * (4 if cplx else 1) * 4 * k * 2.0 ** -23 * big \
                + (2 * k / 192 + 8) * 2.0 ** -23 * (2.0 * np.abs(a) @ np.abs(bm) + 0.5 * np.abs(C0[b]))
            assert np.all(np.abs(got[b] - want) <= bound), (opA, opB, b)
    assert L.lib().tnc_gemm_tc_error() == 0
