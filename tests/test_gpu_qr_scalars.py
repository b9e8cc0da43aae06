"""The scalars of a Householder reflector (beta, tau and the factor of its vector) through the QR."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _qr(A):
    from tncontract_gb300 import _ops
    return [t.cpu().numpy() for t in _ops.qr(torch.from_numpy(A).cuda())]


@pytest.mark.parametrize("dt,tiny", [(np.complex64, 1.2e-20), (np.float32, 1.2e-20), (np.complex128, 1.5e-155), (np.float64, 1.5e-155)])
@pytest.mark.parametrize("lead", [True, False])
def test_tiny_columns(gpu, dt, tiny, lead):
    """Columns beside ordinary ones whose squared norm is a subnormal number.

    Bound: a square x^2 of a subnormal result is off by half a step u (2^-149, 2^-1074), so the squared norm of the
    column by rows u / tiny^2 of itself at most and the reflector's scalars by as much (the factor of the vector twice),
    beside the usual 4 eps sqrt(m k)."""
    cplx = np.issubdtype(dt, np.complexfloating)
    rng = np.random.default_rng(3)
    A = rng.standard_normal((40, 12)) + (1j * rng.standard_normal((40, 12)) if cplx else 0)
    A[:, 5] = 0
    A[:, 9] = 0
    if lead:  # the first column: nothing has been projected out of it
        A[:, 0] = 0
        A[:4, 0] = tiny * np.array([1 + 0.5j, 0.3, -0.7j, 0.9]) if cplx else tiny * np.array([1, 0.3, -0.7, 0.9])
    # and the last: its rows above the diagonal are ordinary, what is left below them is tiny
    A[:, 11] = 0
    A[20:24, 11] = tiny
    A = A.astype(dt)
    step = float(np.nextafter(np.zeros(1, np.finfo(dt).dtype), np.ones(1, np.finfo(dt).dtype))[0])
    tol = 4 * np.finfo(dt).eps * np.sqrt(40 * 12) + 4 * 40 * step / tiny / tiny
    Q, R = _qr(A)
    wide = A.astype(np.complex128 if cplx else np.float64)
    assert np.isfinite(Q).all() and np.isfinite(R).all()
    assert np.linalg.norm(Q @ R.astype(wide.dtype) - wide) <= tol * np.linalg.norm(wide)
    if lead:
        err = np.linalg.norm(Q[:, :1] @ R[:1, :1].astype(wide.dtype) / tiny - wide[:, :1] / tiny)
        assert err <= tol * 4
    assert np.linalg.norm(Q.conj().T @ Q - np.eye(12)) <= tol * np.sqrt(12)


@pytest.mark.parametrize("dt", [np.float32, np.float64, np.complex64, np.complex128])
def test_two_rows(gpu, dt):
    """One reflector at a time: a column of two entries over the whole range of ratios and (double precision) of
    exponents, against extended precision.

    Bound, in u = eps / 2: the norm's square takes 2 u (complex 4 u: four squares, three sums), its root half of that and
    2 u of its own (an ulp); so R is off by 3 u (4 u).  alpha - beta then carries 4 u (5 u), its reciprocal 5 u (complex,
    over the squared modulus, 14 u), tau 9 u (10 u) at up to 2, the vector one u more than its factor; Q's entries are
    1 - tau and tau v, and three products of one term each make them: 16 u (real) and 32 u (complex) cover both."""
    rng = np.random.default_rng(11)
    info = np.finfo(dt)
    cplx = np.issubdtype(dt, np.complexfloating)
    big = np.float64 if info.eps > 1e-10 else np.longdouble
    worst_r = worst_q = 0.0
    mean = []
    for _ in range(400):
        e = rng.integers(-40, 41) if info.eps > 1e-10 else rng.integers(-480, 481)
        a = rng.standard_normal(2) + (1j * rng.standard_normal(2) if cplx else 0)
        a = (a * np.array([1.0, 2.0 ** rng.integers(-12, 13)])).astype(dt)
        a = np.ldexp(a.view(info.dtype), e).astype(info.dtype).view(dt)
        Q, R = _qr(a.reshape(2, 1))
        parts = np.ldexp(a.view(info.dtype).astype(big), -int(e))
        n = np.sqrt((parts * parts).sum())
        r = np.ldexp(big(R[0, 0].real), -int(e))
        rel = float((abs(r) - n) / n / info.eps)
        mean.append(rel)
        worst_r = max(worst_r, abs(rel))
        ref = -np.sign(parts[0]) * parts / n
        worst_q = max(worst_q, float(np.max(np.abs(Q[:, 0].copy().view(info.dtype).astype(big) - ref)) / info.eps))
    assert worst_r <= 2 and worst_q <= (16 if cplx else 8), (worst_r, worst_q)
    # unbiased: the mean of 400 errors of at most 2 eps, uniform or better, stays within 4 deviations
    assert abs(np.mean(mean)) <= 4 * 2 / np.sqrt(3) / np.sqrt(400), np.mean(mean)


@pytest.mark.parametrize("dt", [np.float32, np.float64])
def test_real_norm_is_rounded_once_a_step(gpu, dt):
    """R of one real column of two entries.  Bound, in u = eps / 2: two squares and their sum, 2 u, halved by the root,
    which is rounded correctly: 2 u of the result, that is u of 2^k where the result lies in [2^k, 2^(k+1))."""
    rng = np.random.default_rng(12)
    eps = np.finfo(dt).eps
    for _ in range(1500):
        a = (rng.standard_normal(2) * np.array([1.0, 2.0 ** rng.integers(-3, 4)])).astype(dt)
        _, R = _qr(a.reshape(2, 1))
        x = a.astype(np.float64 if dt == np.float32 else np.longdouble)
        n = np.sqrt((x * x).sum())
        assert abs(abs(x.dtype.type(R[0, 0])) - n) <= eps * n * 1.0001, a
