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
    # 1e-16 a step from the powers' rounding, over the steps
    for i in range(4):
        np.testing.assert_allclose(m.get(i).cpu().numpy(), ref[i], rtol=1e-12, atol=1e-13)
    if n_steps:
        np.testing.assert_allclose(out, sig, rtol=1e-11, atol=1e-13)


@pytest.mark.parametrize("bad", [False, True], ids=["finite", "nonfinite"])
@pytest.mark.parametrize("alpha,E_0", [(0.2, 0.8), (0.2, 0.34), (0.32, 0.34)])
@pytest.mark.parametrize("n_steps", [1, 4, 7, 600])
def test_window_equals_single_steps(alpha, E_0, n_steps, bad):
    """f_in and s bit for bit, q and v to the rounding of their powers (bit for bit with exponents that
    take pow); infinities, NaN and values near the ends of the range as in single steps."""
    rng = np.random.default_rng(3)
    R = 200
    u = np.maximum(rng.lognormal(-6, 1, R), 1e-5)
    st = [rng.normal(0, 0.02, R), rng.uniform(0.7, 1.1, R), rng.uniform(0.95, 1.2, R), rng.uniform(0.8, 1.6, R)]
    if bad:
        for k, (field, x) in enumerate([(0, np.inf), (0, 1e308), (1, -np.inf), (1, 1e308), (2, np.nan), (2, np.inf),
                                        (2, 1e100), (2, 1e-90), (2, 0.0), (3, np.inf), (3, 1e-310), (3, np.nan)]):
            st[field][3 * k] = x
        u[100:102] = [np.inf, 1e308]
    a, b = (BoldModel(R, dtype=torch.float64, delta_t=1e-4, alpha=alpha, E_0=E_0) for _ in range(2))
    for m in (a, b):
        for i, x in enumerate(st):
            m.set(i, torch.from_numpy(x))
    out = a.run_steps(torch.from_numpy(u), n_steps).cpu().numpy()
    for _ in range(n_steps):
        ref = b.run(torch.from_numpy(u)).cpu().numpy()
    got, want = ([m.get(i).cpu().numpy() for i in range(4)] for m in (a, b))
    for i in (0, 3) if alpha == 0.2 else range(4):
        np.testing.assert_array_equal(got[i], want[i])
    for x, y in zip(got + [out], want + [ref]):
        np.testing.assert_array_equal(np.isnan(x), np.isnan(y))
        np.testing.assert_array_equal(np.isinf(x), np.isinf(y))
    for i in (1, 2):      # an ulp of q and v at most in a step's increment, which the model damps
        fin = np.isfinite(want[i])
        np.testing.assert_allclose(got[i][fin], want[i][fin], rtol=2e-16 * (4 + n_steps / 100), atol=0)
