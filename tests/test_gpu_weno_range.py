"""The function-level WENO reconstructions against the oracle, bit for bit, on
values and increments over most of the range of a double: increments down to
the subnormal numbers, where a factor moved out of a product would round
differently, and differences whose squares come near the largest number."""
import numpy as np
import pytest

from pointwise_inputs import lines

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


@pytest.mark.parametrize("eps", [1e-10, 1e-15, 1e-40, 0.0])
@pytest.mark.parametrize("size", [1.0, 1e-150, 1e-230, 1e-250, 1e-265, 1e-272, 1e-280, 1e-290, 1e-300, 1e-308, 1e-315])
def test_weno_deriv_of_any_increment(oracle_lib, native_lib, size, eps):
    f, dq, _ = lines(4, 60, 4, 5)
    f[:2] = 1.0 + 1e-5 * (f[:2] - 1.0)                  # smooth flow, and one with a jump
    dq *= size
    dq[:, 20:30] = 0.0                                  # undisturbed cells
    assert np.any(_check(oracle_lib, "weno_deriv", f, dq, eps) != 0.0)


@pytest.mark.parametrize("name", ["weno", "weno_deriv"])
@pytest.mark.parametrize("scale", [1e-308, 1e-200, 1e-77, 1e38, 1e76, 1e153])
def test_weno_of_any_size(oracle_lib, native_lib, name, scale):
    f, dq, _ = lines(4, 60, 4, 6)
    _check(oracle_lib, name, f * scale, dq * scale)


def test_weno_up_to_the_largest_smoothness_sum(oracle_lib, native_lib):
    """Evenly rising values: second differences vanish, first differences e up
    to 2.6e154, whose 0.25 e e is finite and e e not."""
    step = np.linspace(0.5e154, 1.3e154, 6)[:, None, None]
    f = np.arange(1.0, 21.0)[None, :, None] * step + np.zeros((1, 1, 4))
    assert np.all(np.isfinite(_check(oracle_lib, "weno", f, np.zeros_like(f))))
