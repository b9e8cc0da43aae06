"""con works on its arguments' own data: what it returns never shares it, and the
arguments keep theirs (over the CPU stand-in of the device ops)."""
import numpy as np
import pytest

import host_fake


@pytest.mark.parametrize("order", ["cost", "argument"])
def test_con_shares_nothing(order):
    with host_fake.cpu_ops():
        import tncontract_gb300 as tn
        rng = np.random.default_rng(0)
        a = tn.Tensor(rng.standard_normal((2, 3)), ["a", "b"])
        b = tn.Tensor(rng.standard_normal((3, 1, 4)), ["c", "u", "d"])
        c = tn.Tensor(rng.standard_normal((4, 2)), ["e", "f"])
        t = tn.Tensor(rng.standard_normal((2, 5, 2)), ["x", "y", "z"])
        held = [x.data.clone() for x in (a, b, c, t)]
        for args in ((a,), (b,), (t, ("x", "z")), (a, b, ("b", "c")), (a, b, c, ("b", "c"), ("d", "e"))):
            r = tn.con(*args, order=order)
            for x in (a, b, c, t):
                assert r.data.untyped_storage().data_ptr() != x.data.untyped_storage().data_ptr()
            r.data.zero_()
        for x, h, labels in zip((a, b, c, t), held, (["a", "b"], ["c", "u", "d"], ["e", "f"], ["x", "y", "z"])):
            assert np.array_equal(x.data.numpy(), h.numpy()) and x.labels == labels
