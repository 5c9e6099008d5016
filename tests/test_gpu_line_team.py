"""block_tridag4's two-warp lines (csrc/line_solve.cuh factor_line_team) against the oracle, bit for bit.

Lengths around the shared ring of 16 rows, the shortest lines, more lines
than the GPU has SMs, and lines whose pivots are zero, infinite or NaN: the
reference divides regardless, and the values that do not depend on them stay
exact.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _systems(seed, nlines, n):
    rng = np.random.default_rng(seed)
    a, c = (rng.standard_normal((nlines, n, 4, 4)) for _ in range(2))
    b = rng.standard_normal((nlines, n, 4, 4)) + 6.0 * np.eye(4)
    return a, b, c, rng.standard_normal((nlines, n, 4))


def _solve(native, a, b, c, f, periodic):
    import torch
    ta, tb, tc, tf = (torch.from_numpy(x).cuda() for x in (a, b, c, f))
    native.block_tridag4(ta, tb, tc, tf, periodic)
    return tf.cpu().numpy()


@pytest.mark.parametrize("periodic", [False, True])
@pytest.mark.parametrize("nlines,n", [(1, 2), (2, 4), (3, 15), (3, 16), (3, 17), (2, 33), (1, 400), (700, 6)])
def test_lines_bitexact(oracle_lib, native_lib, nlines, n, periodic):
    from hamstr_oop_gb300 import native
    a, b, c, f = _systems(nlines + 31 * n + int(periodic), nlines, n)
    got = _solve(native, a, b, c, f, periodic)
    for k in range(nlines):
        assert np.array_equal(got[k], oracle_lib.block_tridag4(a[k], b[k], c[k], f[k], periodic)), k


def test_open_line_of_one_row(oracle_lib, native_lib):
    from hamstr_oop_gb300 import native
    a, b, c, f = _systems(5, 4, 1)
    got = _solve(native, a, b, c, f, False)
    for k in range(4):
        assert np.array_equal(got[k], oracle_lib.block_tridag4(a[k], b[k], c[k], f[k], False))


@pytest.mark.parametrize("periodic", [False, True])
@pytest.mark.parametrize("value", [0.0, np.inf, np.nan, 5e-324, 1e308])
def test_degenerate_pivots(oracle_lib, native_lib, value, periodic):
    """Such a row's first pivot in one line of three; the others are unaffected."""
    from hamstr_oop_gb300 import native
    a, b, c, f = _systems(9, 3, 20)
    b[1, 0, 0, 0] = value
    got = _solve(native, a, b, c, f, periodic)
    for k in range(3):
        with np.errstate(all="ignore"):
            want = oracle_lib.block_tridag4(a[k], b[k], c[k], f[k], periodic)
        assert np.array_equal(got[k], want, equal_nan=True), k
