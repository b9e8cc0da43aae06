"""Log-scaled overlaps and fidelities of states whose sites are far from unit norm: norms whose
squares leave the type's range (FP64 above 1.3e154 and below 1e-162, single precision where products
of site and environment do), largest entries next to the ends of the range, and one site of e^600
beside ordinary ones, as the double-precision sweep leaves its first site.

Bound: as for states of unit norm (a sum of d b terms a site, N sites), the factors being powers of
two; a site written near the small end of its type is rounded there before either side reads it."""
import math

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
BONDS = ([1, 5, 17, 33, 9, 2, 1], [1, 3, 8, 80, 7, 4, 1])
CASES = [(np.float64, 1e-200), (np.float64, 1e160), (np.float64, math.exp(600)), (np.float64, 1e-300), (np.float64, 1e307),
         (np.complex128, 1e-200), (np.complex128, 1e160), (np.complex128, math.exp(600)), (np.complex128, 1e-300),
         (np.complex128, 1e307), (np.float32, 1e-34), (np.float32, 1e37), (np.complex64, 1e-34), (np.complex64, 1e37)]


def _chain(seed, bonds, dt, scales):
    rng = np.random.default_rng(seed)
    out = []
    for i, c in enumerate(scales):
        s = (3, bonds[i], bonds[i + 1])
        a = rng.standard_normal(s)
        if np.issubdtype(dt, np.complexfloating):
            a = a + 1j * rng.standard_normal(s)
        out.append((a / np.sqrt(a.size) * c).astype(dt))
    return out


def _dense(sites, scales):
    v = np.ones((1, 1))
    for a, c in zip(sites, scales):
        # scaled back in two steps that stay inside the double range
        a = a.astype(np.complex128) / math.sqrt(c) / math.sqrt(c)
        v = np.tensordot(v, a, (-1, 1)).reshape(-1, a.shape[2])
    return v.reshape(-1)


@pytest.mark.parametrize("first_only", [False, True])
@pytest.mark.parametrize("dt,scale", CASES)
def test_overlap_range(gpu, dt, scale, first_only):
    from tncontract_gb300 import engine
    N = 6
    scales = [scale] + [1.0 if first_only else scale] * (N - 1)
    bra, ket = _chain(1, BONDS[0], dt, scales), _chain(2, BONDS[1], dt, scales)
    x, y = _dense(bra, scales), _dense(ket, scales)
    db, dk = ([torch.from_numpy(a).cuda() for a in P] for P in (bra, ket))
    tol = 40 * N * math.sqrt(3 * 80) * np.finfo(dt).eps
    size = np.linalg.norm(x) * np.linalg.norm(y)
    for conj in (True, False):
        ref = np.vdot(x, y) if conj else np.dot(x, y)
        m, log = engine.inner_product(db, dk, conj_bra=conj, log_scale=True)
        got = m * math.exp(log - 2 * sum(math.log(c) for c in scales))
        assert abs(got - ref) <= tol * size
    f = abs(np.vdot(x, y)) ** 2 / (np.linalg.norm(x) * np.linalg.norm(y)) ** 2
    assert abs(engine.fidelity(db, dk) - f) <= 4 * tol


@pytest.mark.parametrize("dt", [np.float64, np.complex128])
def test_fidelity_of_a_folded_sweep(gpu, dt):
    """The double-precision sweep folds log norms up to 600 into its first site."""
    from tncontract_gb300 import engine
    sites = [torch.from_numpy(a).cuda() for a in _chain(3, BONDS[0], dt, [1.0] * 6)]
    mpo = [torch.eye(3, dtype=sites[0].dtype, device="cuda").reshape(3, 3, 1, 1) for _ in sites]
    st = engine.SweepStats()
    out = engine.apply_compress_native(sites, mpo, 64, log_norm_in=400.0, stats=st)
    assert st.norm_folded and float(out[0].abs().max()) > 1e160
    assert abs(engine.fidelity(sites, out) - 1.0) <= 1e-12
