"""The operations a profiled sweep reports for its double-float finish: those of the whole-matrix steps that ran."""
import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt,gram,rotation", [(torch.complex64, 24, 48), (torch.float32, 6, 12)])
@pytest.mark.parametrize("d", [24, 40, 130])
def test_steps_are_counted(gpu, dt, gram, rotation, d):
    """Two sites, one bond of d rows of d elements: a Gram matrix a step, and as many rotations or one fewer."""
    from tncontract_gb300 import engine
    g = torch.Generator().manual_seed(d)
    sites = [torch.randn(s, generator=g, dtype=dt).cuda() for s in ((d, 1, d + 5), (d, d + 5, 1))]
    mpo = [torch.eye(d, dtype=dt, device="cuda").reshape(d, d, 1, 1) for _ in sites]
    prof = (C.c_double * 12)()
    engine.apply_compress_native(sites, mpo, d, profile=prof, core="df")
    assert prof[10] == 1.0  # one finish
    per = prof[11] / float(d) ** 3
    assert per in {gram * n + rotation * (n - last) for n in (1, 2, 3, 4) for last in (0, 1) if n - last <= 3}, per
