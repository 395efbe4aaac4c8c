"""Surrogate MLP kernels: forward and gradients against the float64 CPU oracle,
and training that fits a smooth function."""
import ctypes

import numpy as np
import pytest
import torch

from oracle import mlp_oracle
from digital_twin_brain_b200 import _lib
from digital_twin_brain_b200._lib import DtbError
from digital_twin_brain_b200.surrogate import MLP, RateSurrogate

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B", [1, 37, 3000])
def test_forward_and_gradient_match_oracle(B):
    rng = np.random.default_rng(B)
    m = MLP(12, 256, seed=3, device=0)
    x = rng.normal(0, 1, (B, 12)).astype(np.float32)
    t = rng.normal(0, 1, B).astype(np.float32)
    w = m.params()
    y_ref, loss_ref, g_ref = mlp_oracle.forward_backward(w, x, t, 12, 256)
    y = m.forward(torch.from_numpy(x)).cpu().numpy()
    np.testing.assert_allclose(y, y_ref, rtol=1e-4, atol=1e-5)
    g, loss = m.gradient(torch.from_numpy(x), torch.from_numpy(t))
    g = g.cpu().numpy()
    assert abs(loss - loss_ref) <= 1e-4 * max(loss_ref, 1e-6)
    scale = np.abs(g_ref).max()
    assert np.abs(g - g_ref).max() <= 1e-4 * scale, np.abs(g - g_ref).max() / scale


def test_training_fits_a_function():
    rng = np.random.default_rng(0)
    x = rng.uniform(-2, 2, (20000, 12)).astype(np.float32)
    t = (np.sin(x[:, 0]) + 0.5 * x[:, 1] * x[:, 2] - 0.3 * x[:, 3]).astype(np.float32)
    m = MLP(12, 256, seed=1, device=0)
    hist = m.fit(torch.from_numpy(x), torch.from_numpy(t), epochs=40, batch=1024, lr=2e-3)
    assert hist[-1] < 0.05 * hist[0] and hist[-1] < 0.02


def test_rate_surrogate_learns_rate_map():
    """A synthetic rate law (rate depends on g factors and the last window) is learned
    well enough to beat the persistence forecast (the method without the network)."""
    rng = np.random.default_rng(1)
    n = 30000
    gui = rng.uniform(0.5, 1.5, (n, 4)).astype(np.float32)
    hist = rng.uniform(0.0005, 0.01, (n, 8)).astype(np.float32)
    target = (0.6 * hist[:, -1] * gui[:, 0] / gui[:, 2] + 0.002 * gui[:, 1]).astype(np.float32)
    s = RateSurrogate(seed=2, context=0)
    s.fit(torch.from_numpy(gui), torch.from_numpy(hist), torch.from_numpy(target), epochs=40, lr=2e-3)
    pred = s.predict(torch.from_numpy(gui), torch.from_numpy(hist)).cpu().numpy()
    err_net = np.sqrt(np.mean((pred - target) ** 2))
    err_persist = np.sqrt(np.mean((hist[:, -1] - target) ** 2))
    assert err_net < 0.25 * err_persist, (err_net, err_persist)


@pytest.mark.parametrize("inputs,hidden", [(1, 256), (16, 256), (17, 256), (32, 256), (33, 256), (14, 64)])
@pytest.mark.parametrize("B", [64, 128, 129, 4801])
def test_shapes_match_oracle(inputs, hidden, B):
    """Whole and partial row tiles, the input paddings, and sizes the fused kernels do not take."""
    rng = np.random.default_rng([B, inputs])
    m = MLP(inputs, hidden, seed=5, device=0)
    x = rng.normal(0, 1, (B, inputs)).astype(np.float32)
    t = rng.normal(0, 1, B).astype(np.float32)
    y_ref, loss_ref, g_ref = mlp_oracle.forward_backward(m.params(), x, t, inputs, hidden)
    np.testing.assert_allclose(m.forward(torch.from_numpy(x)).cpu().numpy(), y_ref, rtol=1e-4, atol=1e-5)
    g, loss = m.gradient(torch.from_numpy(x), torch.from_numpy(t))
    assert abs(loss - loss_ref) <= 1e-4 * loss_ref
    assert np.abs(g.cpu().numpy() - g_ref).max() <= 1e-4 * np.abs(g_ref).max()


@pytest.mark.parametrize("inputs", [14, 32])
@pytest.mark.parametrize("B", [4736, 4737, 9472, 9473, 11521, 37889])
def test_row_copies_match_oracle(inputs, B):
    """The fused kernels at the row counts where a tile holds four, two or one copy of each row, whole
    and partial last tiles, more tiles than SMs."""
    rng = np.random.default_rng([B, inputs])
    m = MLP(inputs, 256, seed=5, device=0)
    x = rng.normal(0, 1, (B, inputs)).astype(np.float32)
    t = rng.normal(0, 1, B).astype(np.float32)
    y_ref, loss_ref, g_ref = mlp_oracle.forward_backward(m.params(), x, t, inputs, 256)
    y = m.forward(torch.from_numpy(x)).cpu().numpy()
    g, loss = m.gradient(torch.from_numpy(x), torch.from_numpy(t))
    g = g.cpu().numpy()
    # float32 sums of 256 terms (16 roundings of 2^-24 as a random walk, 1e-6) through two layers and,
    # for the gradient, sums over the batch; a BF16 term lost from a split would be 2^-17 = 8e-6 or more
    for part, ref in ((y, y_ref), (g, g_ref)):
        assert np.linalg.norm(part - ref) <= 4e-6 * np.linalg.norm(ref)
    assert np.abs(y - y_ref).max() <= 1e-5 * np.abs(y_ref).max()
    assert abs(loss - loss_ref) <= 1e-5 * loss_ref


@pytest.mark.parametrize("hidden", [256, 64])
def test_failed_growth_leaves_other_owners_alone(hidden):
    """Activations that cannot grow: the call reports it, the network stays usable, and closing it
    frees nothing that another network has been given in the meantime."""
    rng = np.random.default_rng(7)
    x = torch.from_numpy(rng.normal(0, 1, (360, 14)).astype(np.float32)).cuda()
    t = torch.from_numpy(rng.normal(0, 1, 360).astype(np.float32)).cuda()
    a = MLP(14, hidden, seed=5, device=0)
    want, loss = a.gradient(x, t)
    with pytest.raises(DtbError):      # 2^40 rows: refused by the allocation, before anything is launched
        _lib.call("dtb_mlp_gradient", a._h, ctypes.c_void_p(x.data_ptr()), ctypes.c_void_p(t.data_ptr()), 1 << 40,
                  None, None)
    b = MLP(14, hidden, seed=5, device=0)
    b.gradient(x, t)                   # the same sizes: the memory a gave back
    a.close()
    g, again = b.gradient(x, t)
    # the gradient's partial sums meet in any order
    np.testing.assert_allclose(g.cpu().numpy(), want.cpu().numpy(), rtol=1e-4, atol=1e-5 * float(want.abs().max()))
    assert abs(again - loss) <= 1e-5 * loss
    c = MLP(14, hidden, seed=5, device=0)
    with pytest.raises(DtbError):
        _lib.call("dtb_mlp_gradient", c._h, ctypes.c_void_p(x.data_ptr()), ctypes.c_void_p(t.data_ptr()), 1 << 40,
                  None, None)
    assert abs(c.gradient(x, t)[1] - loss) <= 1e-5 * loss
    c.close()


@pytest.mark.parametrize("B", [1, 300, 5000, 9500])     # four, two and one copy of a row in the tile
@pytest.mark.parametrize("limit", [0, 1, 2])            # polls: none of the waits, or some, are given up
def test_given_up_waits_yield_no_results(B, limit):
    rng = np.random.default_rng(B)
    x = torch.from_numpy(rng.normal(0, 1, (B, 14)).astype(np.float32)).cuda()
    t = torch.from_numpy(rng.normal(0, 1, B).astype(np.float32)).cuda()
    m = MLP(14, 256, seed=5, device=0)
    w, y = m.params(), m.forward(x).cpu().numpy()
    _lib.call("dtb_mlp_set_wait_limit", m._h, limit)
    z = m.forward(x).cpu().numpy()
    lost = np.isnan(z)
    np.testing.assert_array_equal(z[~lost], y[~lost])
    g, loss = m.gradient(x, t)
    if limit == 0:
        assert lost.all() and np.isnan(loss) and float(g.abs().max()) == 0.0
    given_up = bool(lost.any()) or np.isnan(loss)
    if given_up:
        _lib.call("dtb_mlp_set_wait_limit", m._h, 1 << 22)
        m.train_step(x, t, 1e-2)                        # not reported yet
        with pytest.raises(DtbError):
            m.params()
        np.testing.assert_array_equal(m.params(), w)    # reported once; the step changed nothing
    _lib.call("dtb_mlp_set_wait_limit", m._h, 1 << 22)
    np.testing.assert_array_equal(m.forward(x).cpu().numpy(), y)
    assert np.isfinite(m.gradient(x, t)[1])
    m.train_step(x, t, 1e-2)
    assert (m.params() != w).any()
