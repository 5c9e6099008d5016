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


@pytest.mark.parametrize("periodic", [False, True])
@pytest.mark.parametrize("fn", ["block_tridag4", "block_tridag4_noalloc"])
@pytest.mark.parametrize("odd", ["a", "b", "c", "f", "abcf"])
def test_operands_on_any_8_byte_boundary(oracle_lib, native_lib, fn, odd, periodic):
    """An operand may start an odd number of doubles into its storage."""
    import torch
    from hamstr_oop_gb300 import native
    host = dict(zip("abcf", _systems(77, 3, 21)))
    dev = {}
    for name, x in host.items():
        room = torch.empty(x.size + 1, dtype=torch.float64, device="cuda")
        view = (room[1:] if name in odd else room[:-1]).view(x.shape)
        view.copy_(torch.from_numpy(x))
        assert view.data_ptr() % 16 == (8 if name in odd else 0)
        dev[name] = view
    getattr(native, fn)(dev["a"], dev["b"], dev["c"], dev["f"], periodic)
    torch.cuda.synchronize()
    got = dev["f"].cpu().numpy()
    for k in range(3):
        want = oracle_lib.block_tridag4(host["a"][k], host["b"][k], host["c"][k], host["f"][k], periodic)
        assert np.array_equal(got[k], want), k


@pytest.mark.parametrize("periodic", [False, True])
@pytest.mark.parametrize("nlines", [4700, 4800])
def test_scratch_from_the_pool_and_beyond_it(native_lib, nlines, periodic):
    """Calls whose scratch (2,656 doubles a line) is just below and above what
    the pool serves, 96 MiB, give what smaller calls give on the same lines."""
    from hamstr_oop_gb300 import native
    assert (nlines * 2656 * 8 <= 96 << 20) == (nlines == 4700)
    a, b, c, f = _systems(nlines, 300, 33)
    want = _solve(native, a, b, c, f, periodic)
    a, b, c, f = (np.tile(x, (nlines // 300 + 1,) + (1,) * (x.ndim - 1))[:nlines] for x in (a, b, c, f))
    got = _solve(native, a, b, c, f, periodic)
    for k in range(0, nlines, 300):
        assert np.array_equal(got[k:k + 300], want[:min(300, nlines - k)]), k


@pytest.mark.parametrize("periodic,n", [(False, 1), (False, 20), (True, 2), (True, 20)])
@pytest.mark.parametrize("operand", ["a", "b"])
def test_any_nan_may_stand_in_a_block(oracle_lib, native_lib, operand, periodic, n):
    """Also the one that marks an empty word of the two warps' ring: the solve
    ends as for any other NaN, and not by a wait that gives up, which would
    fill the line with the NaN of all bits set."""
    from hamstr_oop_gb300 import native
    a, b, c, f = _systems(13, 3, n)
    {"a": a, "b": b}[operand].view(np.uint64)[1, 0, 2, 0] = 0xFFF4C3A59B7D6E21
    got = _solve(native, a, b, c, f, periodic)
    assert not np.any(got.view(np.uint64) == 0xFFFFFFFFFFFFFFFF)
    for k in range(3):
        with np.errstate(all="ignore"):
            want = oracle_lib.block_tridag4(a[k], b[k], c[k], f[k], periodic)
        assert np.array_equal(got[k], want, equal_nan=True), k


def test_a_large_call_gets_what_the_pool_kept(native_lib):
    """Scratch beyond the pool's share that fits only with what the pool kept
    from a smaller call, which the driver takes back for it."""
    import torch
    from hamstr_oop_gb300 import native
    need = 9000 * 2656 * 8
    systems = [torch.from_numpy(np.tile(x, (9000 // 300,) + (1,) * (x.ndim - 1))).cuda() for x in _systems(2, 300, 33)]
    small = [x[:2900].clone() for x in systems]
    native.block_tridag4(*small, True)     # 59 MiB of scratch, which the pool keeps
    torch.cuda.synchronize()
    free = lambda: torch.cuda.mem_get_info()[0]
    hog, room = [], need - (24 << 20)
    while free() - room >= 16 << 20:           # (smaller pieces may take a larger segment)
        hog.append(torch.empty(min(8 << 30, (free() - room) >> 21 << 21), dtype=torch.uint8, device="cuda"))
    native.block_tridag4(*systems, True)
    del hog
    torch.cuda.empty_cache()
    assert torch.equal(systems[3][:2900], small[3])


def test_threads_and_streams_share_the_scratch_pool(native_lib):
    """Eight host threads on streams of their own, each with its own systems."""
    import threading
    import torch
    from hamstr_oop_gb300 import native
    work, bad = [], []
    for k in range(8):
        sysk = _systems(40 + k, 30 + k, 20 + 7 * k)
        work.append((sysk, _solve(native, *sysk, bool(k % 2)), torch.cuda.Stream()))

    def solve(k):
        (a, b, c, f), want, stream = work[k]
        with torch.cuda.stream(stream):
            ta, tb, tc, f0 = (torch.from_numpy(x).cuda() for x in (a, b, c, f))
            for _ in range(20):
                tf = f0.clone()
                native.block_tridag4(ta, tb, tc, tf, bool(k % 2), stream=stream.cuda_stream)
                if not np.array_equal(tf.cpu().numpy(), want):
                    bad.append(k)
    threads = [threading.Thread(target=solve, args=(k,)) for k in range(8)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad


AFTER_RESET = r"""
import ctypes, sys
import numpy as np
sys.path.insert(0, sys.argv[1])
from hamstr_oop_gb300 import native
lib = native.load()
rt = ctypes.CDLL("libcudart.so.13")   # the runtime the library is linked with

def solve(fn, a, b, c, f, periodic):
    dev = []
    for x in (a, b, c, f):
        p = ctypes.c_void_p()
        assert rt.cudaMalloc(ctypes.byref(p), ctypes.c_size_t(x.nbytes)) == 0
        assert rt.cudaMemcpy(p, x.ctypes.data_as(ctypes.c_void_p), ctypes.c_size_t(x.nbytes), 1) == 0
        dev.append(p)
    assert fn(f.shape[0], f.shape[1], periodic, *[p.value for p in dev], None) == 0
    out = np.empty_like(f)
    assert rt.cudaMemcpy(out.ctypes.data_as(ctypes.c_void_p), dev[3], ctypes.c_size_t(f.nbytes), 2) == 0
    return out

rng = np.random.default_rng(3)
a, c = (rng.standard_normal((5, 12, 4, 4)) for _ in range(2))
b = rng.standard_normal((5, 12, 4, 4)) + 6.0 * np.eye(4)
f = rng.standard_normal((5, 12, 4))
both = lib.hamstr_gpu_block_tridag4, lib.hamstr_gpu_block_tridag4_noalloc
first = [solve(fn, a, b, c, f, 1) for fn in both]
assert np.array_equal(*first)
for _ in range(2):
    assert rt.cudaDeviceReset() == 0
    for fn in both:
        assert np.array_equal(solve(fn, a, b, c, f, 1), first[0])
print("same after a reset")
"""


def test_scratch_does_not_outlive_its_context():
    """After cudaDeviceReset, which ends the process's own context, the next
    call makes a pool in the new one, and the allocation-free one looks its
    scratch up again.  In a process of its own."""
    import os
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-c", AFTER_RESET, root], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "same after a reset" in r.stdout, r.stdout + r.stderr
