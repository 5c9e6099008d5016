"""The sums over a cell's faces on meshes to either side of one block per SM,
where the linear residual's products change pipes, and on cells with three
faces: bit-identical to the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ni,nj,split", [(8, 3, 0.0), (302, 128, 0.0), (304, 128, 0.0), (250, 121, 0.5)])
def test_cell_sums_are_the_oracles(make_case, oracle_lib, native_lib, ni, nj, split):
    from hamstr_oop_gb300 import native
    case = make_case(ni, nj, split=split, seed=3, order=1, CFL=5.0, msweep=2)
    orc, host = oracle_lib.OracleCase(case, "port"), native.Case(case)
    if split:
        for c in (orc, host):
            c.set_option("chain_end_rule", 1)
    gpu = native.GpuSolver(host)
    want, got = orc.step(), gpu.step()
    for name in ("r", "dq", "q"):
        assert np.array_equal(np.asarray(gpu.get(name)), np.asarray(orc.get(name))), name
    # the maximum norms are those of the same values, the others tree sums
    assert got[1] == want[1] and got[3] == want[3]
    assert abs(got[0] - want[0]) <= 1e-13 * want[0] and abs(got[2] - want[2]) <= 1e-13 * want[2]
