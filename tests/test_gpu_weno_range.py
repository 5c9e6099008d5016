"""The function-level WENO reconstructions against the oracle, bit for bit, on
values over most of the range of a double: differences whose squares come near
the largest number."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _check(oracle_lib, name, f, dq, eps=1e-10):
    import torch
    from hamstr_oop_gb300 import native
    t = [torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (f, dq, np.zeros_like(f), np.zeros_like(f))]
    native.reconstruct(name, t[0], t[2], t[3], 2, f.shape[1] - 1, dq=t[1], eps=eps)
    ql, qr = t[2].cpu().numpy(), t[3].cpu().numpy()
    z = np.zeros_like(f[0])
    for k in range(f.shape[0]):
        with np.errstate(all="ignore"):
            want = oracle_lib.recon_line(name, f[k], 2, f.shape[1] - 1, dq=dq[k], eps=eps, ql=z, qr=z, f2=z)
        assert np.array_equal(ql[k], want[0], equal_nan=True) and np.array_equal(qr[k], want[1], equal_nan=True), k
    return ql


def test_weno_up_to_the_largest_smoothness_sum(oracle_lib, native_lib):
    """Evenly rising values: second differences vanish, first differences e up
    to 2.6e154, whose 0.25 e e is finite and e e not."""
    step = np.linspace(0.5e154, 1.3e154, 6)[:, None, None]
    f = np.arange(1.0, 21.0)[None, :, None] * step + np.zeros((1, 1, 4))
    assert np.all(np.isfinite(_check(oracle_lib, "weno", f, np.zeros_like(f))))
