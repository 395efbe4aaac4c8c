"""The small-network step loop (one cluster, state in shared memory) against the per-step kernels with
the row gather: bit for bit at its edges (words, tiles, CTAs of the cluster, its largest size and one
past it), with slots that overflow, classes mixed inside a tile, members, BOLD and samples."""
import numpy as np
import pytest

from digital_twin_brain_b200 import Network, synthetic
from digital_twin_brain_b200._lib import (FIELD_ACTIVE, FIELD_EVENTS, FIELD_I_SYN, FIELD_J, FIELD_NEW_ACTIVE, FIELD_T,
                                          FIELD_T_LAST, FIELD_V, TUNE_PULL_METHOD)

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
