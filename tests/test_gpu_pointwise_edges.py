"""Line reconstructions over every size and component count the kernels
index by, and with smoothness eps down to zero, against the oracle, bit for
bit.  Data of order one and of order 1e-40, where the weights' derivatives
with a tiny eps come near the subnormal range."""
import numpy as np
import pytest

from pointwise_inputs import lines

pytestmark = pytest.mark.gpu


def _check(oracle_lib, name, nlines, imax, nq, is_, ie, eps, scale=1.0, qt=0.25):
    import torch
    from hamstr_oop_gb300 import native
    f, dq, prior = lines(nlines, imax, nq, 3 * imax + nq)
    f, dq = f * scale, dq * scale
    t = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (f, dq, prior[0], prior[1], prior[2])]
    native.reconstruct(name, t[0], t[2], t[3], is_, ie, dq=t[1], f2=t[4], qt=qt, eps=eps)
    got = [x.cpu().numpy() for x in t[2:]]
    for k in range(nlines):
        with np.errstate(all="ignore"):
            want = oracle_lib.recon_line(name, f[k], is_, ie, dq=dq[k], qt=qt, eps=eps, ql=prior[0, k], qr=prior[1, k],
                                         f2=prior[2, k])
        for g, w, what in zip(got, want, ("ql", "qr", "f2")):
            assert np.array_equal(g[k], w, equal_nan=True), (k, what)


@pytest.mark.parametrize("name", ["muscl", "muscl_deriv", "weno", "weno_deriv"])
@pytest.mark.parametrize("nlines,imax", [(1, 5), (1, 6), (3, 64), (5, 67)])
def test_sizes(oracle_lib, native_lib, name, nlines, imax):
    muscl = name.startswith("muscl")
    _check(oracle_lib, name, nlines, imax, 4, 1 if muscl else 2, imax - 2 if muscl else imax - 1, 1e-10)


@pytest.mark.parametrize("name,is_,off", [("muscl", 2, 4), ("muscl_deriv", 3, 5), ("muscl", 3, 8)])
def test_part_of_a_line(oracle_lib, native_lib, name, is_, off):
    """f2 is written on the whole line, ql and qr on is .. ie (none in the last case)."""
    _check(oracle_lib, name, 4, 10, 4, is_, 10 - off, 1e-10)


@pytest.mark.parametrize("eps", [1e-10, 1e-59, 1e-61, 1e-100, 0.0])
@pytest.mark.parametrize("scale", [1.0, 1e-40])
def test_weno_deriv_with_any_eps(oracle_lib, native_lib, eps, scale):
    _check(oracle_lib, "weno_deriv", 3, 40, 4, 2, 39, eps, scale)
