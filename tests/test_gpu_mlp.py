"""The learned-MDF network on the tensor cores against the CPU oracle
(oracle/mlp.py): forward outputs, gradients (the oracle follows the GPU's
BF16 rounding points; the exact FP64 gradients bound the BF16 effect), Adam
updates and deterministic training."""
import numpy as np
import pytest

from oracle import mlp as Q

pytestmark = pytest.mark.gpu


def _net(seed=3):
    from softflow_b200.learned import MDFNetwork
    net = MDFNetwork(0, seed=seed)
    return net


def _data(n, seed=0):
    rng = np.random.default_rng(seed)
    X = rng.normal(0, 1, (n, 8)).astype(np.float32)
    T = np.stack([np.tanh(X[:, 0] - 0.5 * X[:, 1]) + 0.1 * X[:, 4],
                  X[:, 2] * X[:, 3] * 0.3 - X[:, 7]], 1).astype(np.float32)
    return X, T


def rel(a, b):
    return float(np.linalg.norm(np.asarray(a, np.float64) - b) / np.linalg.norm(b))


def test_forward_matches_oracle(sfg):
    net = _net()
    p = net.params()
    X, _ = _data(1000)      # not a multiple of 128: ragged last tile
    y = net.forward(X).cpu().numpy()
    yq, _ = Q.forward_q(p, X)
    ye, _ = Q.forward_exact(p, X)
    assert rel(y, yq) < 5e-3
    assert rel(y, ye) < 3e-2


def test_forward_normalisation(sfg):
    net = _net()
    rng = np.random.default_rng(1)
    im, isd = rng.normal(0, 1, 8), rng.uniform(0.5, 2.0, 8)
    om, osd = rng.normal(0, 1, 2), rng.uniform(0.5, 2.0, 2)
    net.set_normalization(im, isd, om, osd)
    X, _ = _data(300, 2)
    y = net.forward(X).cpu().numpy()
    Xn = ((X - im.astype(np.float32)) / isd.astype(np.float32)).astype(np.float32)
    yq, _ = Q.forward_q(net.params(), Xn)
    assert rel(y, yq * osd + om) < 5e-3


@pytest.mark.parametrize("n", [128, 1000, 8192])
def test_gradients_match_oracle(sfg, n):
    net = _net()
    p = net.params()
    X, T = _data(n, 4)
    g, loss = net.gradients(X, T)
    gq = Q.gradients_q(p, X, T)
    ge = Q.gradients_exact(p, X, T)
    assert rel(g, gq) < 2e-2, "vs BF16-rounding oracle"
    assert rel(g, ge) < 6e-2, "vs exact FP64"
    assert abs(loss - Q.loss_exact(p, X, T)) / Q.loss_exact(p, X, T) < 2e-2
    # every block of the parameter vector carries gradient
    W1, b1, W2, b2, W3, b3 = Q.unpack(g)
    for blk in (W1, b1, W2, b2, W3, b3):
        assert np.linalg.norm(blk) > 0


def test_adam_step_matches_oracle(sfg):
    net = _net()
    p0 = net.params()
    X, T = _data(8192, 5)
    g, _ = net.gradients(X, T)
    net.train(X, T, epochs=1, batch=8192, lr=1e-3, seed=0)   # one step, whole batch
    p1 = net.params()
    # the shuffled batch is the same set, so the gradient is the same sum
    pe, _, _ = Q.adam(p0, g, np.zeros_like(p0), np.zeros_like(p0), 1, lr=1e-3)
    assert np.max(np.abs(p1 - pe)) < 2e-5
    assert net.steps() == 1


def test_training_reduces_loss_and_is_deterministic(sfg):
    X, T = _data(65536, 6)
    a, b = _net(7), _net(7)
    la = a.train(X, T, epochs=3, batch=8192, lr=1e-3, seed=11)
    lb = b.train(X, T, epochs=3, batch=8192, lr=1e-3, seed=11)
    assert np.array_equal(la, lb)
    assert np.array_equal(a.params(), b.params())
    assert la[-1] < 0.5 * la[0]
    # the trained network generalises to fresh samples of the same law
    Xv, Tv = _data(4096, 8)
    yv = a.forward(Xv).cpu().numpy()
    assert np.mean((yv - Tv) ** 2) < 0.5 * np.mean((Q.forward_exact(Q.he_init(7), Xv)[0] - Tv) ** 2)


@pytest.mark.parametrize("n,batch", [(1, 1), (129, 129), (1000, 300), (8192, 4100)])
def test_training_by_row_list_equals_training_on_copies(sfg, n, batch):
    """A row list is the same as rows copied into its order, bit for bit; the
    sizes leave a last tile of 1, 1, 44 and 4 samples, and rows unused."""
    import ctypes as C
    import torch
    X, T = _data(n, 12)
    x, t = torch.tensor(X, device="cuda"), torch.tensor(T, device="cuda")
    rows = torch.randperm(n, device="cuda", generator=torch.Generator("cuda").manual_seed(3))
    ptr = lambda a: C.c_void_p(a.data_ptr())
    out = []
    for copied in (False, True):
        net = _net(9)
        loss = np.zeros(n // batch, np.float32)
        lp = loss.ctypes.data_as(C.POINTER(C.c_float))
        lib, st = net._lib, C.c_void_p(torch.cuda.current_stream().cuda_stream)
        for _ in range(2):
            if copied:
                xs, ts = x[rows].contiguous(), t[rows].contiguous()
                rc = lib.sfg_mlp_train(net.handle, ptr(xs), ptr(ts), n, batch, 1e-3, lp, st)
            else:
                rc = lib.sfg_mlp_train_rows(net.handle, ptr(x), ptr(t), ptr(rows), n, batch,
                                            1e-3, lp, st)
            assert rc == 0
        out.append((net.params(), loss, net.forward(X).cpu().numpy()))
    for a, b in zip(*out):
        assert np.isfinite(a).all() and np.array_equal(a, b)
    first = Q.loss_exact(Q.he_init(9), X, T) if n == batch else None
    if first is not None:
        net = _net(9)
        one = net.train(X, T, epochs=1, batch=batch, lr=1e-3, seed=0)
        assert abs(one[0] - first) / first < 2e-2


def test_row_list_out_of_range_is_an_error(sfg):
    import ctypes as C
    import torch
    X, T = _data(256, 13)
    x, t = torch.tensor(X, device="cuda"), torch.tensor(T, device="cuda")
    rows = torch.arange(256, device="cuda")
    ptr = lambda a: C.c_void_p(a.data_ptr())
    net = _net(9)
    st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    run = lambda: net._lib.sfg_mlp_train_rows(net.handle, ptr(x), ptr(t), ptr(rows), 256, 256,
                                              1e-3, None, st)
    rows[7] = 256
    assert run() == 1
    assert b"row index" in net._lib.sfg_last_error()
    rows[7] = -1
    assert run() == 1
    rows[7] = 7
    assert run() == 0


@pytest.mark.parametrize("n,batch,where", [(1024, 128, 1000), (1024, 128, 0), (1000, 300, 899)])
def test_row_list_out_of_range_leaves_the_network_alone(sfg, n, batch, where):
    """A bad row in the last batch (or the first) fails the call before any update:
    parameters, step count and moments, and so all later training and predictions,
    are those of a network that never saw the call.  A row that no whole batch uses
    is not looked at."""
    import ctypes as C
    import torch
    X, T = _data(n, 14)
    x, t = torch.tensor(X, device="cuda"), torch.tensor(T, device="cuda")
    ptr = lambda a: C.c_void_p(a.data_ptr())
    st = C.c_void_p(torch.cuda.current_stream().cuda_stream)

    def run(net, rows):
        return net._lib.sfg_mlp_train_rows(net.handle, ptr(x), ptr(t), ptr(rows), n, batch, 1e-3,
                                           None, st)

    a, b = _net(9), _net(9)
    good = torch.randperm(n, device="cuda", generator=torch.Generator("cuda").manual_seed(4))
    assert run(a, good) == 0 and run(b, good) == 0
    before = a.params()
    for value in (n, -1, 1 << 40):
        bad = good.clone()
        bad[where] = value
        assert run(a, bad) == 1
        assert b"row index" in a._lib.sfg_last_error()
        assert np.array_equal(a.params(), before) and a.steps() == b.steps()
        assert np.array_equal(a.forward(X).cpu().numpy(), b.forward(X).cpu().numpy())
    unused = good.clone()
    if n % batch:
        unused[n - 1] = n + 5
    assert run(a, unused) == 0 and run(b, good) == 0
    assert np.array_equal(a.params(), b.params()) and a.steps() == b.steps()
