"""block_tridag5's six lanes per line against the oracle, bit for bit: line
counts around the five lines of a warp, the shortest lines, and degenerate
pivots (the reference divides regardless)."""
import numpy as np
import pytest

from pointwise_inputs import blocks5

pytestmark = pytest.mark.gpu


def _check(oracle_lib, a, b, c, f, periodic):
    import torch
    from hamstr_oop_gb300 import native
    t = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (a, b, c, f)]
    native.block_tridag5(*t, periodic)
    got = [x.cpu().numpy() for x in t]
    for k in range(a.shape[0]):
        with np.errstate(all="ignore"):
            want = oracle_lib.block_tridag5(a[k], b[k], c[k], f[k], periodic)
        for g, w, what in zip(got, want, "abcf"):
            assert np.array_equal(g[k], w, equal_nan=True), (k, what)


@pytest.mark.parametrize("periodic", [False, True])
@pytest.mark.parametrize("nlines,n", [(1, 2), (4, 3), (5, 5), (6, 4), (11, 9), (1, 40)])
def test_lines_bitexact(oracle_lib, native_lib, nlines, n, periodic):
    _check(oracle_lib, *blocks5(nlines, n, 7 * nlines + n), periodic)


def test_open_lines_of_one_row(oracle_lib, native_lib):
    _check(oracle_lib, *blocks5(7, 1, 3), False)


@pytest.mark.parametrize("periodic", [False, True])
@pytest.mark.parametrize("value", [0.0, np.inf, np.nan])
def test_degenerate_pivots(oracle_lib, native_lib, value, periodic):
    a, b, c, f = blocks5(6, 8, 21)
    b[2, 0, 0, 0] = value
    _check(oracle_lib, a, b, c, f, periodic)


# the line counts from which a thread takes a whole line (csrc/strand5.cu one_thread_a_line)
@pytest.mark.parametrize("periodic,n,first", [(False, 1, 6000), (False, 2, 60000), (True, 2, 130000), (True, 3, 130000),
                                              (True, 4, 250000)])
def test_many_lines_as_few_lines(native_lib, periodic, n, first):
    """One more and one fewer line than the rule's count, against the same
    lines in smaller calls: solution and scratch, bit for bit."""
    import torch
    from hamstr_oop_gb300 import native
    few = 1000
    host = [torch.from_numpy(x).cuda() for x in blocks5(few, n, 17 * n)]
    want = [x.clone() for x in host]
    native.block_tridag5(*want, periodic)
    for nlines in (first - 1, first, first + 1):
        got = [x.repeat((nlines // few + 1,) + (1,) * (x.dim() - 1))[:nlines].contiguous() for x in host]
        native.block_tridag5(*got, periodic)
        for g, w in zip(got, want):
            whole = nlines // few * few
            assert torch.equal(g[:whole].view(-1, few, *w.shape[1:]), w.expand(whole // few, *w.shape))
            assert torch.equal(g[whole:], w[:nlines - whole])
