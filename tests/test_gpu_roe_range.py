"""The function-level Roe flux and Jacobian against the oracle, bit for bit,
with velocities up to the largest whose kinetic energy is a number."""
import numpy as np
import pytest

from pointwise_inputs import faces

pytestmark = pytest.mark.gpu


# density 1.5: from 1.1e154 on rho (u u + v v) overflows for some faces, half of it not
@pytest.mark.parametrize("scale", [1e-150, 1.0, 1e150, 1e153, 1.2e154, 1.4e154])
def test_roe_of_any_velocity(oracle_lib, native_lib, scale):
    import torch
    from hamstr_oop_gb300 import native
    nxy, ql, qr = faces(2000, 11)
    for q in (ql, qr):
        q[:, 0] = 1.5
        q[:, 1:3] *= scale
        with np.errstate(over="ignore"):
            q[:, 3] = np.minimum(q[:, 3] * scale * scale, 1.7e308)
    t = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (nxy, ql, qr)]
    got = [x.cpu().numpy() for x in (*native.flux_roe2d(*t), *native.jacobian_roe2d(*t))]
    with np.errstate(all="ignore"):
        want = (*oracle_lib.flux_roe2d(nxy, ql, qr), *oracle_lib.jacobian_roe2d(nxy, ql, qr))
    assert np.array_equal(got[1], want[1], equal_nan=True)
    there = ~np.isnan(want[1])               # the reference stops at a face whose speeds are not numbers
    for g, w in zip(got, want):
        assert np.array_equal(g[there], w[there], equal_nan=True)
