"""The per-step kernels of larger networks: runs of repeated lengths (replayed graphs), the push
scatter's words per warp and prefetch, statistics folded by the scatter, against the row gather."""
import numpy as np
import pytest

from digital_twin_brain_b200 import Network, synthetic
from digital_twin_brain_b200._lib import (FIELD_EVENTS, FIELD_J, FIELD_T_LAST, FIELD_V, TUNE_PULL_METHOD,
                                          TUNE_SCATTER_REVERSE, TUNE_SCATTER_VARIANT, TUNE_SCATTER_WORDS)

pytestmark = pytest.mark.gpu
ROWS = 1


def test_repeated_lengths_equal_row_gather():
    spec = synthetic.whole_brain(R=7, mean_size=3000, sigma=0.5, K=40, gen_seed=2)   # past the small-network loop
    a, b = (Network.from_spec(spec, device=0) for _ in range(2))
    assert a.N > 12288
    b.set_tuning(TUNE_PULL_METHOD, ROWS)
    for net in (a, b):
        net.attach_bold(spec.sub_to_region(), spec.R)
    for n in (7, 7, 7, 5, 5, 7, 9, 9, 9, 11, 11, 11, 13, 13, 7, 32, 32, 45, 45, 45):
        for x, y in zip(a.run(n, noise_rate=0.03, mode="pull"), b.run(n, noise_rate=0.03, mode="pull")):
            np.testing.assert_array_equal(x, y)
    for f in (FIELD_V, FIELD_J, FIELD_T_LAST):
        np.testing.assert_array_equal(a.get(f), b.get(f))
    assert a.get(FIELD_EVENTS) == b.get(FIELD_EVENTS)
    np.testing.assert_array_equal(a.get_bold("bold"), b.get_bold("bold"))


@pytest.mark.parametrize("words,variant,reverse", [(1, 0, 0), (3, 1, 0), (32, 0, 1), (4, 1, 1)])
def test_push_scatter_shapes(words, variant, reverse):
    spec = synthetic.whole_brain(R=7, mean_size=3000, sigma=0.5, K=150, gen_seed=3)
    a, b = (Network.from_spec(spec, device=0) for _ in range(2))
    b.set_tuning(TUNE_PULL_METHOD, ROWS)
    for key, value in ((TUNE_SCATTER_WORDS, words), (TUNE_SCATTER_VARIANT, variant), (TUNE_SCATTER_REVERSE, reverse)):
        a.set_tuning(key, value)
    sa, _, na = a.run(40, noise_rate=0.05, mode="push")
    sb, _, nb = b.run(40, noise_rate=0.05, mode="pull")
    np.testing.assert_array_equal(na, nb)          # refractory: noise alone propagates, the same on both sides
    np.testing.assert_array_equal(sa, sb)
    assert a.get(FIELD_EVENTS) == b.get(FIELD_EVENTS)
    # 40 steps of up to ~25 additions in another order: 1000 float32 roundings at most
    np.testing.assert_allclose(a.get(FIELD_J), b.get(FIELD_J), rtol=1e-5, atol=1e-5)


def test_scatter_variant_zero_is_the_default():
    """Also for a network whose J exceeds L2 (16 bytes a neuron): setting the default changes nothing."""
    net = Network.from_spec(synthetic.single_block(8_400_000, 2, gen_seed=4), device=0)
    assert net.get_tuning(TUNE_SCATTER_VARIANT) == 0
    took = []
    for _ in range(2):
        net.run(8, noise_rate=0.02, isolated=True, mode="push", out=None)
        took.append(net.info().kernel_launches)
        net.set_tuning(TUNE_SCATTER_VARIANT, 0)
        assert net.get_tuning(TUNE_SCATTER_VARIANT) == 0
    assert took[1] == 2 * took[0]
