"""FP32 line kernels at the chain lengths where their row rings turn over."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# open chains of nj rows and loops of ni, about the rings' four and eight rows
@pytest.mark.parametrize("ni,nj", [(4, 2), (6, 3), (8, 4), (10, 5), (14, 7), (16, 8), (18, 9), (30, 15), (34, 17)])
def test_short_chains_take_the_fp64_step(make_case, native_lib, ni, nj):
    """One step is the FP64 step to FP32 rounding (the change of a step is under
    a tenth of q, a row's solve is a few dozen roundings of 6e-8, and there are
    under a hundred rows and a few sweeps: well within 1e-4), and the same bits
    with either block assembly and any block size."""
    from hamstr_oop_gb300 import native
    host = native.Case(make_case(ni, nj, order=1, CFL=5.0, msweep=2))
    plain, mixed = native.GpuSolver(host), native.GpuSolver(host)
    q0 = plain.get("q")
    plain.step()
    want = plain.get("q")
    mixed.set_precision(True)
    got = []
    for fused in (0, 1):
        for block in (32, 64, 128):
            mixed.set_shape(mx_fused=fused, mx_block=block)
            mixed.set("q", q0)
            mixed.step()
            got.append(mixed.get("q"))
    assert np.max(np.abs(want - q0)) > 1e-4 * np.max(np.abs(q0))     # the step moves q
    assert np.max(np.abs(got[0] - want)) < 1e-4 * np.max(np.abs(want))
    for g in got[1:]:
        assert np.array_equal(g, got[0])
