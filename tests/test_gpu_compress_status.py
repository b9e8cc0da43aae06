"""What engine.compress and the native sweep say of a state they cannot compress: non-finite values
and zero states are told apart, alike in the native and the op-by-op form."""
import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _state(dt):
    rng = np.random.default_rng(0)
    return [torch.from_numpy(rng.standard_normal(s)).to(dt).cuda() for s in ((2, 1, 4), (2, 4, 6), (2, 6, 1))]


@pytest.mark.parametrize("native", [True, False])
@pytest.mark.parametrize("site", [0, 1, 2])
@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
@pytest.mark.parametrize("dt", [torch.float32, torch.float64, torch.complex64, torch.complex128])
def test_nonfinite(gpu, monkeypatch, dt, bad, site, native):
    from tncontract_gb300 import engine
    if not native:
        monkeypatch.setattr(engine, "_native_chain", lambda P: False)
    P = _state(dt)
    P[site][1, 0, 0] = bad
    with pytest.raises(ValueError, match="infs or NaNs"):
        engine.compress(P, 3)


@pytest.mark.parametrize("native", [True, False])
@pytest.mark.parametrize("dt", [torch.float32, torch.complex128])
def test_zero(gpu, monkeypatch, dt, native):
    from tncontract_gb300 import engine
    if not native:
        monkeypatch.setattr(engine, "_native_chain", lambda P: False)
    P = _state(dt)
    P[1].zero_()
    with pytest.raises(ValueError, match="zero state"):
        engine.compress(P, 3)


def test_codes(gpu):
    """The C entry: a zero state, a non-finite one and a bad argument have a code each."""
    from tncontract_gb300 import _lib as L
    from tncontract_gb300 import _ops

    def call(P, chi):
        N = len(P)
        bonds = (C.c_int64 * (N + 1))(1, *[int(s.shape[2]) for s in P])
        ones = (C.c_int64 * (N + 1))(*[1] * (N + 1))
        sz = C.c_size_t()
        assert L.lib().tnc_sweep_workspace_size(L.F64, N, 2, bonds, ones, 0, C.byref(sz)) == L.OK
        ws = torch.empty(sz.value, dtype=torch.uint8, device="cuda")
        ptrs = (C.c_void_p * N)(*[s.data_ptr() for s in P])
        ob, oo, od, ln = (C.c_int64 * (N + 1))(), (C.c_int64 * N)(), (C.c_double * (N - 1))(), C.c_double(0.0)
        return L.lib().tnc_sweep_compress(L.F64, N, 2, ptrs, bonds, chi, 1e-15, _ops._p(ws), sz.value, ob, oo, od,
                                          C.byref(ln), _ops._stream())
    P = _state(torch.float64)
    assert call(P, 3) == L.OK
    assert call(P, -1) == L.ERR_ARG
    Z = [p.clone() for p in P]
    Z[2].zero_()
    assert call(Z, 3) == L.ERR_ZERO_STATE
    Z[2][0, 0, 0] = float("nan")
    assert call(Z, 3) == L.ERR_NONFINITE
    assert "zero state" in L.lib().tnc_status_string(L.ERR_ZERO_STATE).decode()
