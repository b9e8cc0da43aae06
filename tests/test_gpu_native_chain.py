"""The native compression and overlap against their op-by-op forms and NumPy: uneven
bonds, both row lengths' sides, every dtype, the call's own results (bonds and
discarded weights from the right, log norm, fold), sites far from unit norm, a
non-contiguous site, and what is refused.

Bounds: both forms make the same decisions; a bond's values carry about
sqrt(n) eps of the largest, a chain of N sites N times that."""
import math

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DTYPES = [np.float32, np.float64, np.complex64, np.complex128]


def _chain(seed, N, d, chi, dt, scale=1.0):
    rng = np.random.default_rng(seed)
    out = []
    for i in range(N):
        s = (d, chi[i], chi[i + 1])
        a = rng.standard_normal(s)
        if np.issubdtype(dt, np.complexfloating):
            a = a + 1j * rng.standard_normal(s)
        out.append((scale * a / np.sqrt(a.size)).astype(dt))
    return out


def _dense(sites):
    v = np.ones((1, 1))
    for a in sites:
        a = np.asarray(a).astype(np.complex128)
        v = np.tensordot(v, a, (-1, 1)).reshape(-1, a.shape[2])
    return v.reshape(-1)


@pytest.mark.parametrize("dt", DTYPES)
@pytest.mark.parametrize("N,d,bond", [(2, 2, [1, 2, 1]), (3, 3, [1, 7, 5, 1]), (7, 2, [1, 3, 9, 20, 33, 11, 6, 1]),
                                      (5, 4, [1, 24, 40, 37, 3, 1])])
def test_compress_matches_op_by_op(gpu, monkeypatch, dt, N, d, bond):
    from tncontract_gb300 import engine
    sites = _chain(N, N, d, bond, dt, 0.3)
    dev = [torch.from_numpy(a).cuda() for a in sites]
    dev[0] = dev[0].permute(2, 1, 0).contiguous().permute(2, 1, 0)  # not contiguous
    chi = max(2, max(bond) // 2)
    got = {}
    for native in (True, False):
        if not native:
            monkeypatch.setattr(engine, "_native_chain", lambda P: False)
        st = engine.SweepStats()
        out, log_norm = engine.compress(dev, chi, stats=st, fold_norm=False, log_norm_in=0.25)
        folded, rest = engine.compress(dev, chi)
        assert rest == 0.0
        got[native] = (st.bonds, st.discarded, math.exp(log_norm - 0.25) * _dense([o.cpu() for o in out]),
                       _dense([o.cpu() for o in folded]))
    a, b = got[True], got[False]
    tol = 40 * N * math.sqrt(d * max(bond)) * np.finfo(dt).eps
    assert a[0] == b[0]
    assert np.allclose(a[1], b[1], rtol=0, atol=tol)
    assert np.linalg.norm(a[2] - b[2]) <= tol * np.linalg.norm(b[2])
    assert np.linalg.norm(a[3] - a[2]) <= tol * np.linalg.norm(b[2])


@pytest.mark.parametrize("dt", DTYPES)
@pytest.mark.parametrize("scale", [1.0, 1e25, 1e-25])
def test_overlap(gpu, dt, scale):
    from tncontract_gb300 import engine
    for N, d, ba, bb in [(1, 3, [1, 4], [1, 5]), (2, 2, [1, 3, 1], [1, 70, 1]), (6, 3, [1, 5, 17, 33, 9, 2, 1], [1, 3, 8, 80, 7, 4, 1])]:
        bra, ket = _chain(1, N, d, ba, dt, scale), _chain(2, N, d, bb, dt, scale)
        db, dk = ([torch.from_numpy(a).cuda() for a in P] for P in (bra, ket))
        for conj in (True, False):
            # per-site factors out of the reference, which overflows as the state does
            x, y = (_dense([a.astype(np.complex128) / scale for a in P]) for P in (bra, ket))
            if N == 1:
                x, y = x.reshape(d, -1)[:, 0], y.reshape(d, -1)[:, 0]
            ref = np.vdot(x, y) if conj else np.dot(x, y)
            tol = 40 * N * math.sqrt(d * 80) * np.finfo(dt).eps * np.linalg.norm(x) * np.linalg.norm(y)
            m, log = engine.inner_product(db, dk, conj_bra=conj, log_scale=True)
            assert abs(m * math.exp(log - 2 * N * math.log(scale)) - ref) <= tol
            if scale == 1.0:
                assert abs(engine.inner_product(db, dk, conj_bra=conj) - ref) <= tol


def test_refused(gpu):
    from tncontract_gb300 import engine
    z = [torch.zeros(2, 1, 3, device="cuda"), torch.zeros(2, 3, 1, device="cuda")]
    with pytest.raises(ValueError):
        engine.compress(z, 2)
