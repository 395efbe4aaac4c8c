"""The small-network step loop (one cluster, state in shared memory) against the per-step kernels with
the row gather: bit for bit at its edges (words, tiles, CTAs of the cluster, its largest size and one
past it), with slots that overflow, classes mixed inside a tile, members, BOLD and samples."""
import numpy as np
import pytest

from digital_twin_brain_b200 import Network, synthetic
from digital_twin_brain_b200._lib import (FIELD_ACTIVE, FIELD_EVENTS, FIELD_I_SYN, FIELD_J, FIELD_NEW_ACTIVE, FIELD_T,
                                          FIELD_T_LAST, FIELD_V, TUNE_BIN_WORDS, TUNE_J_CACHE, TUNE_PULL_METHOD,
                                          TUNE_PUSH_METHOD, TUNE_SCATTER_REVERSE, TUNE_SCATTER_VARIANT,
                                          TUNE_SCATTER_WORDS, TUNE_STAGE_WAIT_LIMIT, TUNE_STEP_VARIANT, TUNE_USE_GRAPHS)

pytestmark = pytest.mark.gpu
ROWS = 1


def _same(a, b):
    for f in (FIELD_V, FIELD_J, FIELD_T_LAST, FIELD_I_SYN, FIELD_ACTIVE, FIELD_NEW_ACTIVE):
        np.testing.assert_array_equal(a.get(f), b.get(f))
    assert a.get(FIELD_T) == b.get(FIELD_T) and a.get(FIELD_EVENTS) == b.get(FIELD_EVENTS)


@pytest.mark.parametrize("rate", [0.01, 0.09])
@pytest.mark.parametrize("N,K", [(2, 1), (31, 8), (33, 20), (384, 60), (385, 60), (1000, 130), (1900, 20), (2600, 20), (3072, 40), (3073, 40),
                                 (12288, 25), (12289, 25)])
def test_small_loop_equals_row_gather(N, K, rate):
    spec = synthetic.single_block(N, K, gen_seed=N, g_ui=(0.02, 0.001, 0.1, 0.005))
    a, b, c = (Network.from_spec(spec, device=0) for _ in range(3))
    b.set_tuning(TUNE_PULL_METHOD, ROWS)
    for n, iso in ((1, False), (70, False), (5, True), (40, False)):
        ra = a.run(n, noise_rate=rate, isolated=iso, mode="pull")
        rb = b.run(n, noise_rate=rate, isolated=iso, mode="pull")
        rc = c.run(n, noise_rate=rate, isolated=iso, mode="push", out="device")
        for x, y, z in zip(ra, rb, rc):
            np.testing.assert_array_equal(x, y)
            if N <= 12288:   # the small loop's push adds in pull order too
                np.testing.assert_array_equal(x, z.cpu().numpy().view(x.dtype))
    _same(a, b)


def test_small_loop_mixed_classes_members_bold_samples():
    rng = np.random.default_rng(0)
    members = [synthetic.whole_brain(R=5, mean_size=150, sigma=0.6, K=30, gen_seed=m) for m in range(4)]
    spec = synthetic.ensemble(members, g_scale=rng.uniform(0.5, 1.5, (4, 5, 4)))
    nets = [Network.from_spec(spec, device=0) for _ in range(2)]
    nets[1].set_tuning(TUNE_PULL_METHOD, ROWS)
    idx = np.array([0, 5, spec.N // 2, spec.N - 1])
    for net in nets:
        net.attach_bold(spec.sub_to_region(), spec.R)
        net.set_samples(idx, 64)
    for n in (3, 300, 17):
        ra, rb = (net.run(n, noise_rate=None, mode="pull") for net in nets)
        for x, y in zip(ra, rb):
            np.testing.assert_array_equal(x, y)
    _same(*nets)
    for f in ("s", "q", "v", "f_in", "bold", "act"):
        np.testing.assert_array_equal(nets[0].get_bold(f), nets[1].get_bold(f))
    for x, y in zip(nets[0].get_samples(), nets[1].get_samples()):
        np.testing.assert_array_equal(x, y)
    np.testing.assert_array_equal(nets[0].window_spikes(), nets[1].window_spikes())


@pytest.mark.parametrize("N,K,rate,mode,loop", [
    (2000, 100, 0.01, "push", True), (2200, 1000, 0.002, "push", True), (2200, 1000, 0.05, "push", False),
    (2200, 1000, 0.02, "pull", True), (9216, 300, 0.02, "push", False), (9216, 300, 0.05, "pull", True),
    (9217, 300, 0.05, "pull", False), (12288, 20, 0.05, "push", True), (12288, 20, 0.05, "pull", True),
    (12288, 100, 0.05, "push", False), (12288, 100, 0.05, "pull", False), (12288, 300, 0.02, "auto", False)])
def test_loop_serves_what_its_slots_hold(N, K, rate, mode, loop):
    """One launch for the steps, or two a step, by the contributions a neuron is expected to get; the
    results are the same either way (pull), or to rounding (push, whose reductions have no order)."""
    spec = synthetic.single_block(N, K, gen_seed=K, g_ui=tuple(g * 10.0 / K for g in synthetic.LIF["g_ui"]))
    a, b = (Network.from_spec(spec, device=0) for _ in range(2))
    b.set_tuning(TUNE_PULL_METHOD, ROWS)
    # refractory from the start: the noise alone propagates
    before = a.info().kernel_launches
    sa, ma, na = a.run(20, noise_rate=rate, mode=mode)
    launches = a.info().kernel_launches - before
    assert launches == 1 if loop else launches >= 40
    sb, mb, nb = b.run(20, noise_rate=rate, mode="pull")
    np.testing.assert_array_equal(na, nb)
    np.testing.assert_array_equal(sa, sb)
    if loop or mode == "pull":
        _same(a, b)
        np.testing.assert_array_equal(ma, mb)
    else:
        # 20 steps of up to ~30 additions in another order: 600 float32 roundings at most
        np.testing.assert_allclose(a.get(FIELD_J), b.get(FIELD_J), rtol=4e-5, atol=1e-5)
        np.testing.assert_allclose(ma, mb, rtol=1e-5)


def test_loop_follows_the_activity_seen():
    """A push run that shows more activity than its noise moves the next runs to the step kernels."""
    spec = synthetic.single_block(12288, 100, gen_seed=2, I_extern_Input=8.0, T_ref=0.5,
                                  g_ui=tuple(g * 0.01 for g in synthetic.LIF["g_ui"]))
    net = Network.from_spec(spec, device=0)

    def launches(n, isolated=False):
        before = net.info().kernel_launches
        _, _, na = net.run(n, noise_rate=0.0, isolated=isolated, mode="push")
        return net.info().kernel_launches - before, na.mean() / net.N
    first, _ = launches(300)                     # driven over threshold every dozen steps
    quiet, _ = launches(20, isolated=True)       # noise alone propagates: the loop again
    driven, f = launches(40)
    assert f > 0.04 and first < 2 * 300
    assert quiet == 1 and driven >= 80


def test_schedule_keys_choose_the_kernels():
    """A key of the per-step kernels set to its default, or back to it, keeps the loop; another value,
    or an explicit push method, selects these kernels."""
    net = Network.from_spec(synthetic.single_block(3000, 40, gen_seed=3), device=0)

    def loop(mode="push"):
        before = net.info().kernel_launches
        net.run(10, noise_rate=0.01, mode=mode)
        return net.info().kernel_launches - before == 1
    others = {TUNE_SCATTER_WORDS: 8, TUNE_STEP_VARIANT: 0, TUNE_J_CACHE: 1, TUNE_SCATTER_VARIANT: 1,
              TUNE_SCATTER_REVERSE: 1, TUNE_STAGE_WAIT_LIMIT: 5, TUNE_USE_GRAPHS: 0}
    for key, other in others.items():
        default = net.get_tuning(key)
        net.set_tuning(key, default)
        assert loop("push") and loop("pull"), key
        net.set_tuning(key, other)
        assert not loop("push") and not loop("pull"), key
        net.set_tuning(key, default)
        assert loop("push"), key
    assert net.get_tuning(TUNE_SCATTER_VARIANT) == 0
    net.set_tuning(TUNE_BIN_WORDS, 64)           # a key of the binned push alone
    assert loop("push")
    net.autotune(4, noise_rate=0.01)
    assert loop("push") and loop("pull")
    net.set_tuning(TUNE_PUSH_METHOD, 1)          # atomics into J, asked for
    assert not loop("push") and loop("pull")
