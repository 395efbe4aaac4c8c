"""The work that users of this package have it do, as cases that can be timed and compared.

Every case is a plain dict.  ``prepare(case, seed)`` builds what a program holds before the call
(the network with its state, the surrogate with its weights, the inputs), ``run(state)`` is one
pass through the public entry points, ``exact(case, seed)`` the same result in 64 bits from plain
torch.  The kinds:

``block``     the drop-in ``models.block.block`` of a small network, one call per time step.
``network``   ``Network.run`` of a chunk of steps: host-array networks, generated regions, the
              whole brain, ensembles, with or without BOLD, bit-exact pull or push.
``da``        one forecast window of the ensemble data assimilation.
``forward``   the surrogate's forecast of a batch.
``gradient``  its loss gradient on a batch.
``adapt``     Adam steps on the judges' windows.
``bold``      the hemodynamics of a window with forecast rates.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from digital_twin_brain_b200 import Network, synthetic
from digital_twin_brain_b200._lib import FIELD_J, FIELD_STEP, FIELD_T, FIELD_T_LAST, FIELD_V
from digital_twin_brain_b200.assimilation import DAConfig, EnsembleDA
from digital_twin_brain_b200.models.block import block
from digital_twin_brain_b200.network import BoldModel
from digital_twin_brain_b200.surrogate import MLP

DEV = torch.device("cuda", 0)
DT = 0.1                 # ms, the step of every configuration of this repository
T0 = 500.0               # ms simulated before the pass
G_UI = synthetic.LIF["g_ui"]
BOLD_DT = DT / 1000.0    # s


def listed():
    return [
        # the single-block configuration through the drop-in class, stepped call by call as the
        # reference's own test loops do; bit-exact pull, the class's default
        dict(name="block_2k_by_step", kind="block", n=2000, k=100, p=0.01, steps=20),
        # the same network in a closed loop, statistics of every step on the host
        dict(name="closed_loop_2k", kind="network", source="region", n=2000, k=100, p=0.01, mode="pull", steps=1000,
             out="host", bold=False, tune=False),
        # a network handed over as host arrays (a loaded population), ragged size
        dict(name="population_31k_push", kind="network", source="arrays", n=31013, k=64, p=0.01, mode="push", steps=24,
             out="device", bold=False, tune=False),
        # one region of 1e6 neurons, 1e8 synapses: the bit-exact pull and the push
        dict(name="region_1m_pull", kind="network", source="region", n=1_000_000, k=100, p=0.01, mode="pull", steps=32,
             out="device", bold=False, tune=False),
        dict(name="region_1m_push", kind="network", source="region", n=1_000_000, k=100, p=0.01, mode="push", steps=32,
             out="device", bold=False, tune=False),
        # the whole-brain network at half its size (three states fit the device), tuned before the
        # run and with BOLD per region, as the benchmark runs it
        dict(name="whole_brain_half_push", kind="network", source="brain", n=11_700_000, k=100, p=0.01, mode="push",
             steps=32, out="none", bold=True, tune=True),
        # ensemble members side by side, one BOLD region per member
        dict(name="ensemble_64_push", kind="network", source="ensemble", n=1_460_000, members=64, k=100, p=0.01,
             mode="push", steps=64, out="device", bold=True, tune=False),
        # a forecast window of the assimilation, shortened from 8000 steps
        dict(name="da_window_8x90", kind="da", members=8, regions=90, n=2000, k=100, steps=400),
        # 128 members x 90 regions through the surrogate
        dict(name="surrogate_forward_11520", kind="forward", rows=11520, inputs=14, hidden=256),
        # a training minibatch
        dict(name="surrogate_gradient_4096", kind="gradient", rows=4096, inputs=14, hidden=256),
        # the per-window adaptation on half of the eight judges' regions
        dict(name="surrogate_adapt_360", kind="adapt", rows=360, inputs=14, hidden=256, steps=20),
        # the 120 surrogate-served members' hemodynamics over one 800 ms window
        dict(name="bold_window_10800", kind="bold", n=10800, steps=8000),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["block", "arrays", "region", "region", "region", "brain", "ensemble", "da", "forward",
                       "gradient", "adapt", "bold"])
    p = round(math.exp(rng.uniform(math.log(0.001), math.log(0.05))), 5)
    mode = rng.choice(["pull", "push"])
    if kind == "block":
        return dict(kind="block", n=_log_int(rng, 300, 4000), k=rng.randint(20, 100), p=p, steps=rng.randint(1, 30))
    if kind == "arrays":
        return dict(kind="network", source="arrays", n=_log_int(rng, 1000, 40000), k=rng.randint(8, 80), p=p, mode=mode,
                    steps=rng.randint(8, 32), out=rng.choice(["host", "device"]), bold=False, tune=False)
    if kind == "region":
        n = _log_int(rng, 500, 1_000_000)
        steps = rng.randint(200, 1000) if n < 20000 else rng.randint(8, 64)
        return dict(kind="network", source="region", n=n, k=rng.randint(20, 100), p=p, mode=mode, steps=steps,
                    out=rng.choice(["host", "device"]), bold=rng.choice([False, True]), tune=False)
    if kind == "brain":
        return dict(kind="network", source="brain", n=_log_int(rng, 100_000, 6_000_000), k=rng.randint(40, 100), p=p,
                    mode=mode, steps=rng.randint(8, 32), out="none", bold=True, tune=rng.choice([False, True]))
    if kind == "ensemble":
        return dict(kind="network", source="ensemble", n=_log_int(rng, 60_000, 1_460_000), members=rng.randint(2, 64),
                    k=rng.randint(40, 100), p=p, mode="push", steps=rng.randint(16, 64), out="device", bold=True,
                    tune=False)
    if kind == "da":
        return dict(kind="da", members=rng.randint(1, 8), regions=rng.randint(8, 90), n=rng.randint(300, 2000), k=100,
                    steps=rng.randint(50, 400))
    if kind == "forward":
        return dict(kind="forward", rows=_log_int(rng, 90, 46080), inputs=rng.choice([12, 14]), hidden=256)
    if kind == "gradient":
        return dict(kind="gradient", rows=_log_int(rng, 64, 8192), inputs=rng.choice([12, 14]), hidden=256)
    if kind == "adapt":
        return dict(kind="adapt", rows=_log_int(rng, 90, 4096), inputs=rng.choice([12, 14]), hidden=256,
                    steps=rng.randint(1, 60))
    return dict(kind="bold", n=_log_int(rng, 90, 10800), steps=rng.randint(1000, 8000))


# ------------------------------------------------------------ inputs
def _property(n, n_exc):
    rows = np.stack([synthetic.property_row(0), synthetic.property_row(1)])
    return np.repeat(rows, [n_exc, n - n_exc], axis=0).astype(np.float32)


def _synapses(case, seed):
    """(post, pre, kind, weight): K distinct sources per neuron, rows in ascending source order."""
    n, k = case["n"], case["k"]
    rng = np.random.default_rng([seed, 1])
    step = max(1, (n - 1) // k)                      # one source from each of k strata of the others
    off = np.arange(k) * step + 1 + rng.integers(0, step, (n, k))
    pre = np.sort((np.arange(n)[:, None] + off) % n, axis=1).astype(np.uint32).reshape(-1)
    post = np.repeat(np.arange(n, dtype=np.uint32), k)
    kind = np.where(pre < int(0.8 * n), 0, 2).astype(np.uint8)
    return post, pre, kind, rng.random((n * k, 2), np.float32)


def _dynamic_state(n, seed):
    """V, J [4, N], t_last of a network past its spin-up: the stationary mean and spread of the
    single-block configuration, some neurons about to fire, some refractory.  t_last lies half a
    step off the time grid, so no neuron leaves its refractory period on a rounding."""
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) * 2654435761 % (1 << 62) + 17)
    V = torch.randn(n, generator=g, device=DEV).mul_(4.0).sub_(63.0).clamp_(-75.0, -50.05)
    J = torch.randn((4, n), generator=g, device=DEV)
    J.mul_(torch.tensor([[1.8], [14.6], [3.0], [12.0]], device=DEV))
    J.add_(torch.tensor([[8.15], [156.0], [10.0], [47.0]], device=DEV)).clamp_(min=0.0)
    ago = torch.randint(0, 1000, (n,), generator=g, device=DEV).float()
    refractory = ago < 50
    V[refractory] = -55.0
    return V.cpu().numpy(), J.cpu().numpy(), (T0 - (ago + 0.5) * DT).cpu().numpy()


def _set_state(net, seed):
    V, J, t_last = _dynamic_state(net.N, seed)
    net.set(FIELD_V, V)
    net.set(FIELD_J, J)
    net.set(FIELD_T_LAST, t_last)
    net.set(FIELD_T, T0)
    net.set(FIELD_STEP, int(T0 / DT))


def _spec(case, seed):
    if case["source"] == "region":
        return synthetic.single_block(case["n"], case["k"], gen_seed=seed, seed=seed)
    # the sizes belong to the case, the synapses, the noise and the members' factors to the seed
    if case["source"] == "brain":
        spec = synthetic.whole_brain(90, case["n"] / 102.0, 0.5, case["k"], seed=seed)
        spec.gen_seed = seed
        return spec
    members, g = synthetic.ensemble_members(case["members"], case["n"] // (2 * case["members"]),
                                            3 * case["n"] // (2 * case["members"]), case["k"])
    for m, t in enumerate(members):
        t.gen_seed = seed * 1000 + m
    return synthetic.ensemble(members, g_scale=np.roll(g, seed, axis=0))


def _decay():
    return torch.exp(-DT / torch.tensor(synthetic.LIF["tao_ui"], dtype=torch.float32)).numpy()


def _mlp_inputs(case, seed):
    rng = np.random.default_rng([seed, 2])
    h, d = case["hidden"], case["inputs"]
    w = np.concatenate([rng.uniform(-1, 1, h * d) / math.sqrt(d), rng.normal(0, 0.05, h),
                        rng.uniform(-1, 1, h * h) / math.sqrt(h), rng.normal(0, 0.05, h),
                        rng.uniform(-1, 1, h) / math.sqrt(h), rng.normal(0, 0.05, 1)]).astype(np.float32)
    x = rng.normal(0, 1, (case["rows"], d)).astype(np.float32)        # standardised log features
    t = (0.5 * x[:, 0] - 0.3 * x[:, 1] * x[:, 2] + 0.1 * rng.normal(0, 1, len(x))).astype(np.float32)
    return w, x, t


def _bold_inputs(case, seed):
    rng = np.random.default_rng([seed, 3])
    n = case["n"]
    u = rng.lognormal(math.log(2e-3), 1.0, n)                          # spikes per neuron and step
    s, q, v, f = (rng.normal(0, 0.02, n), rng.uniform(0.7, 1.1, n), rng.uniform(0.95, 1.2, n), rng.uniform(0.8, 1.6, n))
    return u, s, q, v, f


def prepare(case, seed):
    kind = case["kind"]
    if kind == "block":
        post, pre, k, w = _synapses(case, seed)
        n = case["n"]
        ch = np.stack([k, k + 1], 1).astype(np.int64)
        idx = np.stack([ch.reshape(-1), np.repeat(post, 2).astype(np.int64), np.repeat(pre, 2).astype(np.int64)])
        w_uij = torch.sparse_coo_tensor(torch.from_numpy(idx), torch.from_numpy(w.reshape(-1)), (4, n, n),
                                        check_invariants=False)
        b = block(torch.from_numpy(_property(n, int(0.8 * n))), w_uij, delta_t=DT, seed=seed, device=0)
        _set_state(b.network, seed)
        return dict(case=case, block=b)
    if kind == "network":
        if case["source"] == "arrays":
            n = case["n"]
            prop = _property(n, int(0.8 * n))
            net = Network.from_arrays(prop, *_synapses(case, seed), dt=DT, seed=seed,
                                      decay=np.broadcast_to(_decay(), (n, 4)))
        else:
            spec = _spec(case, seed)
            net = Network.from_spec(spec, class_decay=np.broadcast_to(_decay(), (2 * spec.R, 4)))
            if case["bold"]:
                net.attach_bold(spec.sub_to_region(), spec.R)
        if case["tune"]:
            net.autotune(8, noise_rate=case["p"])
        _set_state(net, seed)
        return dict(case=case, net=net)
    if kind == "da":
        template = synthetic.whole_brain(R=case["regions"], mean_size=case["n"], sigma=0.5, K=case["k"],
                                         g_ui=(2 * G_UI[0], 2 * G_UI[1], G_UI[2], G_UI[3]))
        template.gen_seed = seed
        da = EnsembleDA(template, DAConfig(n_members=case["members"], steps_per_window=case["steps"], seed=seed))
        da.hp_random_initialize()
        _set_state(da.net, seed)
        return dict(case=case, da=da)
    if kind == "bold":
        u, s, q, v, f = _bold_inputs(case, seed)
        m = BoldModel(case["n"], dtype=torch.float64, delta_t=BOLD_DT)
        for i, a in enumerate((s, q, v, f)):
            m.set(i, torch.from_numpy(a))
        return dict(case=case, bold=m, u=torch.from_numpy(u).to(DEV))
    w, x, t = _mlp_inputs(case, seed)
    m = MLP(case["inputs"], case["hidden"], seed=0)
    m.set_params(w)
    return dict(case=case, mlp=m, x=torch.from_numpy(x).to(DEV), t=torch.from_numpy(t).to(DEV))


# ------------------------------------------------------------ one pass
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "block":
        b = state["block"]
        rows = [b.run(case["p"]) for _ in range(case["steps"])]
        return dict(sums=[r[0] for r in rows], means=[r[1] for r in rows][-1], V=b.V_i, J=b.J_ui)
    if kind == "network":
        net = state["net"]
        out = None if case["out"] == "none" else case["out"]
        stats = net.run(case["steps"], noise_rate=case["p"], mode=case["mode"], out=out)
        device = case["out"] != "host"
        got = dict(V=net.get(FIELD_V, device=device), J=net.get(FIELD_J, device=device))
        if stats is not None:
            got.update(sums=stats[0], means=stats[1], nact=stats[2])
        if case["bold"]:
            got["bold"] = net.get_bold("bold", device=device)
        return got
    if kind == "da":
        da = state["da"]
        return dict(hidden=da.evolve(), rates=da.window_rates())
    if kind == "forward":
        return dict(y=state["mlp"].forward(state["x"]))
    if kind == "gradient":
        g, loss = state["mlp"].gradient(state["x"], state["t"])
        return dict(grad=g, loss=loss)
    if kind == "adapt":
        m = state["mlp"]
        for _ in range(case["steps"]):
            loss = m.train_step(state["x"], state["t"], 5e-4)
        return dict(params=m.params(), loss=loss)
    m = state["bold"]
    out = m.run_steps(state["u"], case["steps"])
    return dict(bold=out, s=m.get(0), q=m.get(1), v=m.get(2), f=m.get(3))


# ------------------------------------------------------------ what a pass cannot do without
def work(case):
    kind = case["kind"]
    if kind in ("block", "network", "da"):
        n, steps, p = case["n"], case["steps"], case.get("p", 0.01)
        if kind == "da":
            n = int(case["members"] * case["regions"] * case["n"] * 1.13)    # mean of the region sizes
        events = n * case["k"] * p
        # V, J, t_last read, V and J written, one bit a neuron; a firing row's bounds, 12 bytes a synapse
        per_step = 44 * n + n / 8 + 16 * n * p + 12 * events
        return dict(bytes=steps * per_step + (0 if kind == "da" else 20 * n), flops=steps * (40 * n + 2 * events))
    if kind == "bold":
        return dict(bytes=8 * 10 * case["n"], flops=60.0 * case["n"] * case["steps"])
    b, d, h = case["rows"], case["inputs"], case["hidden"]
    params = h * d + h * h + 3 * h + 1
    macs = b * (d * h + h * h + h)
    if kind == "forward":
        return dict(bytes=4 * b * (d + 1) + 2 * params, flops=2 * macs)
    grad = 2 * macs + 2 * b * (d * h + 2 * h * h + 2 * h)
    if kind == "gradient":
        return dict(bytes=4 * b * (d + 2) + 6 * params, flops=grad)
    return dict(bytes=case["steps"] * (4 * b * (d + 1) + 24 * params), flops=case["steps"] * grad)


def tolerance(case):
    kind = case["kind"]
    if kind == "block" or (kind == "network" and case["mode"] == "pull"):
        return "exact"                       # sums in a fixed order: the same bits
    if kind == "network":
        # float32 additions in another order (about 1e-7), and a spike that a rounding moves to the next
        # step: its 100 targets' J differ by a weight
        return dict(rel=2e-5, max=0.9, differ=1e-2)
    if kind == "da":
        return dict(rel=5e-3, max=0.9)       # last-step activity of 2000-neuron regions, a few spikes apart
    if kind == "forward":
        return dict(rel=2e-6, max=2e-5)
    if kind == "gradient":
        return dict(rel=4e-6, max=4e-5)
    if kind == "adapt":
        return dict(rel=1e-3, max=0.1)       # Adam divides by a gradient's own size; weights pass through BF16
    return dict(rel=1e-12, max=1e-11)


# ------------------------------------------------------------ 64 bits
_M0, _M1, _MASK = 0xD2511F53, 0xCD9E8D57, 0xFFFFFFFF


def _philox(c, key):
    """Philox4x32-10 (Salmon et al., SC'11) on int64 tensors holding 32-bit words."""
    def mulhilo(a, x):
        lo, hi = a * (x & 0xFFFF), a * (x >> 16)
        low = (lo + ((hi & 0xFFFF) << 16)) & _MASK
        return ((hi + (lo >> 16)) >> 16) & _MASK, low

    x, y, z, w = c
    k0, k1 = key & _MASK, (key >> 32) & _MASK
    for r in range(10):
        if r:
            k0, k1 = (k0 + 0x9E3779B9) & _MASK, (k1 + 0xBB67AE85) & _MASK
        h0, l0 = mulhilo(_M0, x)
        h1, l1 = mulhilo(_M1, z)
        x, y, z, w = h1 ^ y ^ k0, l1, h0 ^ w ^ k1, l0
    return x, y, z, w


def _uniform(n, seed, step):
    """The noise uniforms of step `step`: a call serves four neurons 32 apart of a 128-neuron tile."""
    tiles = -(-n // 128)
    c = torch.arange(tiles * 32, dtype=torch.int64)
    o = _philox((c, torch.zeros_like(c), torch.full_like(c, step & _MASK), torch.zeros_like(c)), seed)
    u = torch.stack(o, 0).reshape(4, tiles, 32).permute(1, 0, 2).reshape(-1)[:n]
    return (u >> 8).double() / 16777216.0


def _exact_steps(case, seed):
    n, steps = case["n"], case["steps"]
    post, pre, kind, w = (torch.from_numpy(a) for a in _synapses(case, seed))
    post, pre, kind, w = post.long(), pre.long(), kind.long(), w.double()
    prop = torch.from_numpy(_property(n, int(0.8 * n))).double()
    decay = torch.from_numpy(_decay()).double()[:, None]
    V, J, t_last = (torch.from_numpy(a) for a in _dynamic_state(n, seed))
    V, J = V.double(), J.double()
    g, Vu = prop[:, 10:14].T, prop[:, 14:18].T
    sub = prop[:, 3].long()
    count = torch.bincount(sub).double()
    dt, t = np.float32(DT), np.float32(T0)
    sums, means, nact = [], [], []
    for i in range(steps):
        t = np.float32(t + dt)
        isyn = (g * (Vu - V) * J).sum(0)
        Vn = V + float(dt) / prop[:, 4] * (-prop[:, 6] * (V - prop[:, 7]) + isyn + prop[:, 2])
        free = torch.from_numpy(t >= t_last.numpy() + np.float32(5.0))
        Vn = torch.where(free, Vn, prop[:, 9])
        active = Vn >= prop[:, 8]
        V = torch.minimum(Vn, prop[:, 8])
        fires = active | (_uniform(n, seed, int(T0 / DT) + i) < float(np.float32(case["p"])))
        on = fires[pre]
        J = J * decay
        J.view(-1).index_add_(0, kind[on] * n + post[on], w[on, 0])
        J.view(-1).index_add_(0, (kind[on] + 1) * n + post[on], w[on, 1])
        t_last = torch.where(active, torch.tensor(float(t)), t_last)
        sums.append(torch.bincount(sub, active.double()))
        means.append(torch.bincount(sub, V) / count)
        nact.append(int(fires.sum()))
    if case["kind"] == "block":
        return dict(sums=sums, means=means[-1], V=V, J=J)
    return dict(V=V, J=J, sums=torch.stack(sums), means=torch.stack(means), nact=torch.tensor(nact))


def _exact_mlp(case, seed):
    w, x, t = (torch.from_numpy(a) for a in _mlp_inputs(case, seed))
    h, d = case["hidden"], case["inputs"]
    sizes = [h * d, h, h * h, h, h, 1]
    parts = [p.bfloat16().double() if i in (0, 2, 4) else p.double() for i, p in enumerate(w.split(sizes))]
    parts = [p.requires_grad_() for p in parts]
    gelu = torch.nn.functional.gelu
    z = gelu(x.double() @ parts[0].reshape(h, d).T + parts[1])
    z = gelu(z @ parts[2].reshape(h, h).T + parts[3])
    y = z @ parts[4] + parts[5]
    if case["kind"] == "forward":
        return dict(y=y.detach())
    loss = (y - t.double()).square().mean()
    loss.backward()
    return dict(grad=torch.cat([p.grad for p in parts]), loss=float(loss.detach()))


def _exact_bold(case, seed):
    u, s, q, v, f = (torch.from_numpy(a).to(DEV) for a in _bold_inputs(case, seed))
    u = u.clamp(min=1e-5)
    for _ in range(case["steps"]):
        ds = 200.0 * u - s / 0.8 - (f - 1.0) / 0.4
        dq = (f * torch.where(f > 0, 1.0 - 0.2 ** (1.0 / f), 1.0) / 0.8 - q * v ** 4) / 1.0
        dv = f - v ** 5
        q, v = q + dq * BOLD_DT, v + dv * BOLD_DT
        f, s = (f + s * BOLD_DT).clamp(min=0.0), s + ds * BOLD_DT
    out = 0.02 * (7.0 * 0.8 * (1.0 - q) + 2.0 * (1.0 - q / v) + (2.0 * 0.8 - 0.2) * (1.0 - v))
    return dict(bold=out, s=s, q=q, v=v, f=f)


def exact(case, seed):
    kind = case["kind"]
    if kind == "block" or (kind == "network" and case["source"] == "arrays"):
        return _exact_steps(case, seed)
    if kind in ("forward", "gradient"):
        return _exact_mlp(case, seed)
    if kind == "bold":
        return _exact_bold(case, seed)
    # networks generated on the device (their synapses come from this package), and Adam steps (a weight
    # that rounds to the other BF16 value grows into the next step): no 64-bit counterpart
    return None
