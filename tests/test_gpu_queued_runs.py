"""Runs queued behind each other without a host synchronisation between their chunks: every chunk
works with its own call's noise rate and fills its own statistics rows, also while the host is
several chunks ahead of the device."""
import ctypes

import numpy as np
import pytest
import torch

from digital_twin_brain_b200 import Network, _lib, synthetic
from digital_twin_brain_b200._lib import DTB_DEVICE, FIELD_STEP, TUNE_PULL_METHOD
from digital_twin_brain_b200.network import MODES

pytestmark = pytest.mark.gpu

RATES = (0.01, 0.2, 0.05, 0.0, 0.1)


def _run(net, n, rate, out):
    p = [ctypes.c_void_p(t.data_ptr()) for t in out]
    _lib.call("dtb_block_run", net._h, n, rate, 1, MODES["push"], *p, DTB_DEVICE)


@pytest.mark.parametrize("steps", [32, 160, 37])     # one chunk a call, five, one and a rest
def test_queued_device_runs_equal_host_runs(steps):
    spec = synthetic.single_block(20000, 20, gen_seed=1)     # past the small-network loop: chunks of 32 steps
    a, b = (Network.from_spec(spec, device=0) for _ in range(2))
    side = torch.cuda.Stream()
    a.set_stream(side)
    a.run(1, noise_rate=0.01, isolated=True, mode="push")
    b.run(1, noise_rate=0.01, isolated=True, mode="push")
    outs = [(torch.empty((steps, a.n_sub), device="cuda"), torch.empty((steps, a.n_sub), device="cuda"),
             torch.empty((steps,), dtype=torch.int32, device="cuda")) for _ in RATES]
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        torch.cuda._sleep(20_000_000)                # about 10 ms: the calls below are all queued behind it
    for rate, out in zip(RATES, outs):
        _run(a, steps, rate, out)
    a.synchronize()
    for rate, (s, m, n) in zip(RATES, outs):
        hs, hm, hn = b.run(steps, noise_rate=rate, isolated=True, mode="push")
        np.testing.assert_array_equal(n.cpu().numpy().view(np.uint32), hn)   # isolated: the noise alone, exact
        # the additions into J come in another order: float32 rounding
        np.testing.assert_allclose(m.cpu().numpy(), hm, rtol=1e-4)
        assert np.abs(s.cpu().numpy() - hs).sum() <= 0.01 * hs.sum() + 5     # spikes a rounding moves by a step


def test_captured_run_replays_with_its_own_arguments():
    """A run inside the caller's CUDA graph: every replay takes the captured call's noise rate and
    writes its statistics rows, whatever runs came in between."""
    spec = synthetic.single_block(20000, 20, gen_seed=1)
    a, b = (Network.from_spec(spec, device=0) for _ in range(2))
    side = torch.cuda.Stream()
    a.set_stream(side)
    for net in (a, b):
        net.run(32, noise_rate=0.01, isolated=True, mode="push")     # buffers and the chunk graph exist
    out = (torch.empty((7, a.n_sub), device="cuda"), torch.empty((7, a.n_sub), device="cuda"),
           torch.empty((7,), dtype=torch.int32, device="cuda"))
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=side):
        _run(a, 7, 0.3, out)
    for _ in range(3):
        g.replay()
        torch.cuda.synchronize()
        np.testing.assert_array_equal(out[2].cpu().numpy().view(np.uint32),
                                      b.run(7, noise_rate=0.3, isolated=True, mode="push")[2])
        x, y = (net.run(5, noise_rate=0.02, isolated=True, mode="push")[2] for net in (a, b))
        np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize("N", [2000, 20000])     # one cluster launch; a chain of per-step kernels
def test_captured_run_outlives_new_statistics_tables(N):
    """The statistics tables that a captured run reads stay readable after BOLD is attached again."""
    spec = synthetic.single_block(N, 20, gen_seed=1)
    a, b = (Network.from_spec(spec, device=0) for _ in range(2))
    side = torch.cuda.Stream()
    a.set_stream(side)
    for net in (a, b):
        net.run(32, noise_rate=0.01, isolated=True, mode="push")
    out = (torch.empty((7, a.n_sub), device="cuda"), torch.empty((7, a.n_sub), device="cuda"),
           torch.empty((7,), dtype=torch.int32, device="cuda"))
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=side):
        _run(a, 7, 0.3, out)
    held = [a.info().device_bytes]
    for _ in range(3):
        a.attach_bold(spec.sub_to_region(), spec.R)
        held.append(a.info().device_bytes)
        filler = [torch.full((64,), -1, dtype=torch.int32, device="cuda") for _ in range(64)]   # what was given back is used
        g.replay()
        torch.cuda.synchronize()
        del filler
        np.testing.assert_array_equal(out[2].cpu().numpy().view(np.uint32),
                                      b.run(7, noise_rate=0.3, isolated=True, mode="push")[2])
    assert held[-1] - held[-2] <= 4096     # a few small tables a time


@pytest.mark.parametrize("mode,method", [("push", 0), ("pull", 0), ("pull", 1), ("pull", 4)])
def test_rows_start_with_their_run(mode, method, tmp_path):
    """Row 0 belongs to the run's first step after everything that moves the clock: single steps, forced
    steps, kernel timing, a step count set from outside, a checkpoint, a run of the small loop."""
    spec = synthetic.single_block(20000, 20, gen_seed=1)
    net = Network.from_spec(spec, device=0)
    net.set_tuning(TUNE_PULL_METHOD, method)

    def expected(step, n):      # the noise of each step, from a network that takes them one by one
        ref = Network.from_spec(spec, device=0)
        ref.set(FIELD_STEP, step)
        return np.concatenate([ref.run(1, noise_rate=0.05, isolated=True, mode="push")[2] for _ in range(n)])

    def check(n):
        step = int(net.get(FIELD_STEP))
        np.testing.assert_array_equal(net.run(n, noise_rate=0.05, isolated=True, mode=mode)[2], expected(step, n))
    check(3)
    net.run(1, noise_rate=0.2, mode=mode, out=None)
    check(2)
    net.step_forced(None, None, noise_rate=0.1, isolated=True, mode=mode)
    check(2)
    net.time_kernels(4, noise_rate=0.1, isolated=True, mode=mode)
    check(40)
    net.set(FIELD_STEP, 777)
    check(2)
    net.save(str(tmp_path / "ck.bin"))
    net.run(5, noise_rate=0.1, mode=mode)
    net.load(str(tmp_path / "ck.bin"))
    check(35)


def test_many_queued_runs_on_changing_streams():
    """More queued runs than parameter slots, on streams that take turns: each keeps its noise rate."""
    spec = synthetic.single_block(20000, 4, gen_seed=1)
    a, b = (Network.from_spec(spec, device=0) for _ in range(2))
    streams = [torch.cuda.Stream() for _ in range(2)]
    rates = np.random.default_rng(0).uniform(0.0, 0.3, 700)
    counts = torch.zeros((len(rates),), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    for k, rate in enumerate(rates):
        if k % 170 == 0:
            other, side = streams[k // 170 % 2], streams[(k // 170 + 1) % 2]
            side.wait_stream(other)                      # the runs follow each other
            a.set_stream(side)
            with torch.cuda.stream(side):
                torch.cuda._sleep(4_000_000)             # about 2 ms
        _lib.call("dtb_block_run", a._h, 1, float(rate), 1, MODES["push"], None, None,
                  ctypes.c_void_p(counts[k:].data_ptr()), DTB_DEVICE)
    torch.cuda.synchronize()
    want = np.concatenate([b.run(1, noise_rate=float(r), isolated=True, mode="push")[2] for r in rates])
    np.testing.assert_array_equal(counts.cpu().numpy().view(np.uint32), want)
