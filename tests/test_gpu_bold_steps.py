"""Windows of BOLD steps (constant input) against the CPU oracle's step, in float64: steps around the
look-ahead of the kernel, the model's own exponents and others, inputs below the floor."""
import numpy as np
import pytest
import torch

from oracle import oracle as O
from digital_twin_brain_b200.network import BoldModel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("alpha,E_0", [(0.2, 0.8), (0.32, 0.34), (0.2, 0.34)])
@pytest.mark.parametrize("n_steps", [0, 1, 3, 4, 5, 1001])
def test_run_steps_matches_oracle(alpha, E_0, n_steps):
    rng = np.random.default_rng(n_steps)
    R, dt = 67, 1e-3
    u = np.maximum(rng.lognormal(-6, 2, R), 0.0)
    st = [rng.normal(0, 0.1, R), rng.uniform(0.5, 1.2, R), rng.uniform(0.9, 1.3, R), rng.uniform(0.0, 1.6, R)]
    st[3][:5] = 0.0                                            # no flow: the extraction's other branch
    m = BoldModel(R, dtype=torch.float64, delta_t=dt, alpha=alpha, E_0=E_0)
    for i, a in enumerate(st):
        m.set(i, torch.from_numpy(a))
    out = m.run_steps(torch.from_numpy(u), n_steps).cpu().numpy()
    params = dict(epsilon=200, tao_s=0.8, tao_f=0.4, tao_0=1, alpha=alpha, E_0=E_0, V_0=0.02)
    ref = [a.copy() for a in st]
    for _ in range(n_steps):
        sig = O.bold_step(np.maximum(u, 1e-5), *ref, params, dt)
        np.testing.assert_array_equal(np.isfinite(sig), True)
    # 1e-16 a step from the products and reciprocals against pow and division, over the steps
    for i in range(4):
        np.testing.assert_allclose(m.get(i).cpu().numpy(), ref[i], rtol=1e-12, atol=1e-13)
    if n_steps:
        np.testing.assert_allclose(out, sig, rtol=1e-11, atol=1e-13)
