"""The GEMM's tile shapes: sizes at the edges of the FP64 tiles (8 x 16, 16 x 16,
32 x 32) and of the FP32 ones (64 x 64 and 32 x 32, with K split over a cluster) and on
both sides of the lines between them, ragged K, every operand layout, batches, and
groups.  Bound: (k + 2) roundings of |A| |B| per term of a real sum, twice that
in complex."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SIZES = [(1, 1, 1), (7, 15, 3), (8, 16, 16), (9, 17, 17), (32, 32, 16), (33, 31, 15), (100, 97, 33), (208, 192, 40), (513, 291, 18),
         (700, 660, 5)]
SINGLE = [(1, 1, 1), (1, 1, 1537), (1, 33, 255), (31, 32, 17), (33, 32, 64), (65, 31, 128), (64, 70, 511), (300, 200, 129),
          (769, 31, 90), (832, 768, 33), (800, 830, 20)]


@pytest.mark.parametrize("m,n,k,dt", [s + (t,) for s in SIZES for t in (np.float64, np.complex128)]
                         + [s + (t,) for s in SINGLE for t in (np.float32, np.complex64)])
def test_gemm_tiles(gpu, dt, m, n, k):
    from tncontract_gb300 import _lib as L
    from tncontract_gb300 import _ops
    rng = np.random.default_rng(7)
    cplx = dt in (np.complex64, np.complex128)
    wide = np.complex128 if cplx else np.float64

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
                  alpha=0.5, beta=2.0, batch=batch, sA=A[0].size, sB=B[0].size, sC=m * n, tc=False)
        got = Cd.cpu().numpy()
        for b in range(batch):
            a, bm = ops[opA](A[b]).astype(wide), ops[opB](B[b]).astype(wide)
            want = 0.5 * (a @ bm) + 2.0 * C0[b]
            bound = (4 * k + 8) * np.finfo(dt).eps * (0.5 * np.abs(a) @ np.abs(bm) + 2.0 * np.abs(C0[b]))
            assert np.all(np.abs(got[b] - want) <= bound), (opA, opB, b)


@pytest.mark.parametrize("dt", [np.float32, np.complex64, np.float64, np.complex128])
def test_grouped_split(gpu, dt):
    """Problems of very different K and size in one launch: some CTAs of a split have no slice."""
    from tncontract_gb300 import _lib as L
    from tncontract_gb300 import _ops
    rng = np.random.default_rng(8)
    cplx = dt in (np.complex64, np.complex128)
    wide = np.complex128 if cplx else np.float64

    def rnd(*shape):
        a = rng.standard_normal(shape)
        return (a + 1j * rng.standard_normal(shape) if cplx else a).astype(dt)
    probs, want = [], []
    for m, n, k in [(1, 1, 900), (40, 33, 7), (64, 100, 300), (5, 70, 16), (130, 2, 17)]:
        A, B = rnd(m, k), rnd(k, n)
        Cd = torch.empty((m, n), dtype=torch.from_numpy(A).dtype, device="cuda")
        probs.append((L.OP_N, L.OP_N, m, n, k, torch.from_numpy(A).cuda(), k, torch.from_numpy(B).cuda(), n, Cd, n))
        want.append((A.astype(wide) @ B.astype(wide), (4 * k + 8) * np.finfo(dt).eps * (np.abs(A) @ np.abs(B))))
    _ops.gemm_grouped(probs)
    for p, (ref, bound) in zip(probs, want):
        assert np.all(np.abs(p[9].cpu().numpy() - ref) <= bound)
