"""The network's fused kernels at the edges of their tiles and variants.

A row's output does not depend on the other rows or on which variant of the
kernel carries its tile (one block to an SM up to one tile per SM, two
beyond), so outputs of different calls are equal bit for bit; gradients are
checked against the oracle as in test_gpu_mlp.py (2% in norm, BF16
activations)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _rows(n, seed):
    import torch
    rng = np.random.default_rng(seed)
    f = rng.uniform(-1.5, 1.5, (n, 5)).astype(np.float32)
    t = np.stack([np.sin(f[:, 0]), f[:, 1] * f[:, 3], np.cos(f[:, 4]), f[:, 2] ** 2], axis=1).astype(np.float32)
    return f, t, torch.from_numpy(f).cuda(), torch.from_numpy(t).cuda()


@pytest.mark.parametrize("n", [1, 127, 128, 129, 1000, 19456, 19457, 45000])
def test_forward_rows_do_not_depend_on_the_call(native_lib, n):
    import torch
    from hamstr_oop_gb300 import native
    net = native.Mlp(batch_capacity=256, seed=3)
    _, _, fd, _ = _rows(45000, 1)
    y = net.forward(fd[:n].contiguous())
    take = torch.unique(torch.cat([torch.arange(min(n, 200)), torch.arange(max(0, n - 200), n)]))
    z = net.forward(fd[take.cuda()].contiguous())
    assert torch.equal(y[take.cuda()], z)


@pytest.mark.parametrize("n", [1, 127, 129, 300])
def test_gradient_of_ragged_batches_matches_the_oracle(native_lib, oracle_lib, n):
    from hamstr_oop_gb300 import native
    net = native.Mlp(batch_capacity=384, seed=5)
    f, t, fd, td = _rows(n, 7)
    loss_o, g_o, _ = oracle_lib.mlp_loss_grad(net.get_params().astype(np.float64), f, t, bf16=True)
    assert abs(net.grad(fd, td) - loss_o) <= 2e-3 * loss_o
    g = net.get_grads().astype(np.float64)
    bounds = np.cumsum([0, 1280, 256, 65536, 256, 65536, 256, 1024, 4])
    for a, b in zip(bounds[:-1], bounds[1:]):
        assert np.linalg.norm(g[a:b] - g_o[a:b]) <= 2e-2 * np.linalg.norm(g_o[a:b]), (a, b)


def test_a_batch_below_capacity_trains_the_same(native_lib):
    """4,864 rows use more splits of the weight gradients than 16,384 do."""
    from hamstr_oop_gb300 import native
    _, _, fd, td = _rows(9000, 9)
    got = []
    for capacity in (4864, 16384):
        net = native.Mlp(batch_capacity=capacity, seed=2)
        loss = [net.train_step(fd, td, batch=4864, seed=11, step=k, lr=1e-3) for k in range(2)]
        got.append((loss, net.get_params()))
    assert got[0][0] == got[1][0] and np.array_equal(got[0][1], got[1][1])


def test_threads_read_parameters_and_gradients_at_once(native_lib):
    import threading
    from hamstr_oop_gb300 import native
    net = native.Mlp(batch_capacity=256, seed=4)
    _, _, fd, td = _rows(200, 3)
    net.grad(fd, td)
    want = net.get_params(), net.get_grads()
    bad = []

    def read(k):
        for _ in range(200):
            got = net.get_grads() if k % 2 else net.get_params()
            if not np.array_equal(got, want[k % 2]):
                bad.append(k)
    threads = [threading.Thread(target=read, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad


def test_forward_of_the_most_rows(native_lib):
    """2^31 - 1 rows, 77 GB of inputs and outputs."""
    import torch
    from hamstr_oop_gb300 import native
    n = 2 ** 31 - 1
    if torch.cuda.mem_get_info()[0] < 100e9:
        pytest.skip("needs 77 GB of device memory")
    net = native.Mlp(batch_capacity=256, seed=6)
    _, _, fd, _ = _rows(1 << 16, 4)
    feat = torch.empty((n, 5), device="cuda")
    whole = n // (1 << 16) << 16
    feat[:whole].view(-1, 1 << 16, 5).copy_(fd.expand(whole >> 16, 1 << 16, 5))
    feat[whole:].copy_(fd[:n - whole])
    y, z = net.forward(feat), net.forward(fd)
    del feat
    same = all(bool(torch.equal(y[k << 16:(k + 1) << 16], z)) for k in (0, 1, 1000, (whole >> 16) - 1))
    same = same and bool(torch.equal(y[whole:], z[:n - whole]))
    del y
    torch.cuda.empty_cache()
    assert same


@pytest.mark.parametrize("tile", [0, 5, 17, 18])
def test_forward_reports_a_loader_that_gave_up(native_lib, tile):
    """At the first, a middle and the last weight tile (after which no other
    role waits any more); the next pass is whole again."""
    from hamstr_oop_gb300 import native
    net = native.Mlp(batch_capacity=256, seed=8)
    _, _, fd, _ = _rows(128, 5)
    want = net.forward(fd).cpu().numpy()
    assert native_lib.hamstr_check_mlp_wait(net.h, tile) == 0
    with pytest.raises(native.HamstrError):
        net.forward(fd)
    assert np.array_equal(net.forward(fd).cpu().numpy(), want)


@pytest.mark.parametrize("tile", [0, 18, 30, 36])
def test_a_failed_step_changes_nothing(native_lib, tile):
    """Parameters, gradients and moments: two steps after it are the two steps
    of a network that never failed."""
    from hamstr_oop_gb300 import native
    _, _, fd, td = _rows(1000, 6)
    got = []
    for fail in (False, True):
        net = native.Mlp(batch_capacity=256, seed=9)
        loss = [net.train_step(fd, td, batch=256, seed=3, step=0, lr=1e-3)]
        if fail:
            before = net.get_params(), net.get_grads()
            for call in (lambda: net.train_step(fd, td, batch=256, seed=3, step=1, lr=1e-3),
                         lambda: net.grad(fd[:200].contiguous(), td[:200].contiguous())):
                assert native_lib.hamstr_check_mlp_wait(net.h, tile) == 0
                with pytest.raises(native.HamstrError):
                    call()
            assert np.array_equal(net.get_params(), before[0]) and np.array_equal(net.get_grads(), before[1])
        loss.append(net.train_step(fd, td, batch=256, seed=3, step=1, lr=1e-3))
        got.append((loss, net.get_params(), net.get_grads()))
    assert got[0][0] == got[1][0]
    assert np.array_equal(got[0][1], got[1][1]) and np.array_equal(got[0][2], got[1][2])
