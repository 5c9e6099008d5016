"""The launch shapes a handle starts with, on both sides of the rules that
choose them from the mesh (csrc/api.cu default_line_packing and
default_mx_fused): whatever the default is, states are those of every shape
set explicitly."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _batch(make_case, n, ni, nj, split):
    from hamstr_oop_gb300 import native
    base = native.Case(make_case(ni, nj, split=split, seed=1, order=1, CFL=2.0, msweep=2))
    if split:
        base.set_option("chain_end_rule", 1)
    cases = []
    for k in range(n):
        c = base.clone()
        c.set_flow(0.3 + 0.3 * k / n, 1.0)
        cases.append(c)
    return native.GpuSolver.batch(cases)


# rows of open chains per pair of them a sub-partition can hold, over the longest chain's: 1.6 and 1.7 by
# the first two; more than 24 open chains to a sub-partition on split meshes by the last two (the others have
# 16 rows to a chain); more than 2^15 chains on the fourth
@pytest.mark.parametrize("n,ni,nj,split,lanes,bundle,fused", [(31, 64, 16, 0.0, 16, 0, 0), (33, 64, 16, 0.0, 4, 0, 0),
                                                             (2, 64, 16, 0.5, 16, 0, 0), (420, 64, 16, 0.0, 4, 0, 1),
                                                             (70, 64, 16, 0.5, None, 8, 0)])
def test_defaults_by_the_mesh_change_no_state(make_case, native_lib, n, ni, nj, split, lanes, bundle, fused):
    g = _batch(make_case, n, ni, nj, split)
    start = g.shape()
    assert start["adi_bundle_rows"] == bundle and start["mx_fused"] == fused
    assert lanes is None or start["adi_open_lanes"] == lanes
    q0 = g.get("q")
    for mixed, shapes in ((False, [dict(adi_open_lanes=ln, adi_bundle_rows=bu) for ln in (32, 16, 4) for bu in (0, 8)]),
                          (True, [dict(mx_fused=f, mx_block=b) for f in (0, 1) for b in (32, 64)])):
        g.set_precision(mixed)
        g.set_shape(**start)
        g.set("q", q0)
        g.march(2, 0.0)
        want = g.get("q")
        assert not np.array_equal(want, q0)
        for shape in shapes:
            g.set_shape(**shape)
            g.set("q", q0)
            g.march(2, 0.0)
            assert np.array_equal(g.get("q"), want), (mixed, shape)


def test_blocks_that_do_not_fit_are_assembled_inside(make_case, native_lib):
    """The FP32 blocks (192 bytes a row) are allocated last; where memory has run
    out before them, a handle whose default is to keep them goes without, with
    the same states."""
    import torch
    from hamstr_oop_gb300 import native
    host = native.Case(make_case(512, 256, order=1, CFL=2.0, msweep=2))
    free = lambda: torch.cuda.mem_get_info()[0]
    a, b = native.GpuSolver(host), native.GpuSolver(host)
    assert a.shape()["mx_fused"] == b.shape()["mx_fused"] == 0
    torch.cuda.synchronize()
    before = free()
    a.set_precision(True)
    took = before - free()
    blocks = 192 * a.layout()["nRow"]
    assert took > blocks > 40 << 20
    room = took - blocks // 2              # half of the blocks would fit
    hog = []
    while free() - room >= 16 << 20:           # (smaller pieces may take a larger segment)
        hog.append(torch.empty(min(8 << 30, (free() - room) >> 21 << 21), dtype=torch.uint8, device="cuda"))
    b.set_precision(True)
    assert b.shape()["mx_fused"] == 1
    del hog
    torch.cuda.empty_cache()
    a.march(3, 0.0)
    b.march(3, 0.0)
    assert np.array_equal(a.get("q"), b.get("q"))
