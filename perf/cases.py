"""The work that this framework is measured on, each case through its public entry points.

Kinds of case (``case["kind"]``):

* ``lif``, ``adex``, ``layer``, ``hh``: a network on the plain path
  (:class:`edlut_b200.simulation.Simulation`).  A pass is what a program that drives a
  running network does: hand it the input spikes of the next ``steps`` integration
  steps, advance it, read the spikes and the membrane potentials back, and the weights
  where they are plastic.  The network goes on from pass to pass; its inputs repeat
  every ``trial`` steps, as in repeated trials of one experiment.
* ``sweep``: many small LIF networks of uneven sizes in one launch
  (:class:`edlut_b200.sweep.Sweep`): reset, run, read the observed membrane traces and
  the spike counts (and every network's spikes where ``spikes`` is set).
* ``fit``: one step of fitting parameters and weights to membrane traces
  (:class:`edlut_b200.adjoint.TraceModel`): forward, mean squared error, backward.
* ``fold``: one call of the delivery op ``eb_fold_arrivals`` on device arrays, which an
  engine that delivers spikes itself makes once per integration step.

Networks, weights and input spikes are synthetic (:mod:`edlut_b200.configs`).
"""
import ctypes
import math

import numpy as np
import torch

from edlut_b200 import _lib, configs
from edlut_b200.adjoint import TraceModel
from edlut_b200.network import poisson_input_times
from edlut_b200.simulation import Simulation
from edlut_b200.sweep import Sweep

DEVICE = "cuda" if torch.cuda.is_available() else "cpu"


def listed():
    return [
        # A closed loop that exchanges spikes with a small running network every
        # millisecond: launches and host work count.
        dict(name="closed_loop", kind="lif", n=1000, inputs=100, integrator="Euler", steps=10, trial=1000, settle=300),
        # The 1,000-neuron recurrent LIF workload, a 0.3 s stretch of it.
        dict(name="lif_1k", kind="lif", n=1000, inputs=100, integrator="Euler", steps=3000, trial=3000, settle=0),
        # A recurrent AdEx network of odd size: excitation and inhibition, three delays, STDP.
        dict(name="adex_delays", kind="adex", n=2501, inputs=300, integrator="RK2", steps=500, trial=1000, settle=0),
        # A tenth-size cerebellar layer: granule cells on few inputs each, Purkinje cells on
        # thousands of plastic synapses.
        dict(name="layer_25k", kind="layer", granule=25_000, purkinje=20, fan_in=5_000, steps=1000, trial=1000, settle=0),
        # The cerebellar layer at its full granule count and Purkinje fan-in (fewer Purkinje
        # cells, so that the network is built in seconds).
        dict(name="layer_250k", kind="layer", granule=250_000, purkinje=40, fan_in=50_000, steps=2000, trial=2000, settle=0),
        # Stiff Hodgkin-Huxley neurons under BDF: a small ragged network, and the 100,000
        # neurons of the benchmark at a lower in-degree (built in seconds).
        dict(name="hh_3k", kind="hh", n=3001, indegree=100, steps=200, trial=400, settle=0),
        dict(name="hh_100k", kind="hh", n=100_000, indegree=20, steps=200, trial=400, settle=0),
        # A parameter scan of few networks whose spikes are all read, and one of many.
        dict(name="sweep_24", kind="sweep", networks=24, n_min=500, n_max=1500, integrator="RK4", steps=500, observed=16, spikes=True),
        dict(name="sweep_600", kind="sweep", networks=600, n_min=500, n_max=5000, integrator="RK2", steps=1000, observed=8, spikes=False),
        # Fitting a few small networks, and the shape of the fitting benchmark (10,000
        # neurons a network, fewer networks, so that they are built in seconds).
        dict(name="fit_small", kind="fit", networks=5, n_min=300, n_max=900, integrator="RK4", steps=100, observed=32),
        dict(name="fit_10k", kind="fit", networks=8, n_min=4000, n_max=10_000, integrator="RK2", steps=500, observed=256),
        # Arrivals of one step of an engine that delivers spikes itself.
        dict(name="fold_100k", kind="fold", arrivals=100_000, targets=30_000),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["lif", "adex", "layer", "hh", "sweep", "fit", "fold"])
    if kind == "lif":
        steps = _log_int(rng, 5, 2000)
        return dict(kind=kind, n=_log_int(rng, 200, 3000), inputs=_log_int(rng, 20, 300),
                    integrator=rng.choice(["Euler", "RK2", "RK4", "BDF"]), steps=steps, trial=steps * rng.randint(1, 3), settle=300)
    if kind == "adex":
        steps = _log_int(rng, 100, 500)
        return dict(kind=kind, n=_log_int(rng, 200, 3000), inputs=_log_int(rng, 40, 400),
                    integrator=rng.choice(["Euler", "RK2", "RK4", "BDF"]), steps=steps, trial=steps, settle=0)
    if kind == "layer":
        granule = _log_int(rng, 5_000, 250_000)
        steps = _log_int(rng, 300, 2000)
        return dict(kind=kind, granule=granule, purkinje=rng.randint(3, 30), fan_in=max(1200, granule // 5), steps=steps,
                    trial=steps, settle=0)
    if kind == "hh":
        n = _log_int(rng, 500, 100_000)
        steps = _log_int(rng, 50, 300)
        return dict(kind=kind, n=n, indegree=rng.randint(10, 20 if n > 15_000 else 100), steps=steps, trial=steps, settle=0)
    if kind == "sweep":
        n_min = _log_int(rng, 500, 1000)
        return dict(kind=kind, networks=_log_int(rng, 3, 400), n_min=n_min, n_max=n_min * rng.randint(2, 5),
                    integrator=rng.choice(["Euler", "RK2", "RK4"]), steps=_log_int(rng, 100, 1000), observed=rng.randint(1, 32),
                    spikes=rng.random() < 0.3)
    if kind == "fit":
        n_min = _log_int(rng, 200, 4000)
        return dict(kind=kind, networks=rng.randint(1, 8), n_min=n_min, n_max=2 * n_min,
                    integrator=rng.choice(["Euler", "RK2", "RK4"]), steps=_log_int(rng, 50, 500), observed=rng.randint(1, 128))
    return dict(kind=kind, arrivals=_log_int(rng, 100, 1_000_000), targets=_log_int(rng, 50, 300_000))


# ---------------------------------------------------------------- inputs --
def _network(case, seed):
    """A plain-path case's network description and the input spikes of its settling
    time and one trial: (net, times, cells)."""
    total = case["settle"] + case["trial"]
    if case["kind"] == "lif":
        return configs.lif_recurrent(seed=seed, n=case["n"], n_inputs=case["inputs"], rate_hz=20.0, p=min(0.1, 100.0 / case["n"]),
                                     t_end=total * 1e-4, integrator=case["integrator"])
    if case["kind"] == "adex":
        # (connectivity is the case's, weights and input spikes come from the seed)
        net, _, _ = configs.parity_network("AdExTimeDrivenModel", case["integrator"], n=case["n"], n_inputs=case["inputs"],
                                      p=min(0.1, 100.0 / case["n"]), t_end=1e-3, stdp=True, delays=(1e-3, 2e-3, 3.5e-3),
                                           weights=dict(w_in=240.0 / case["inputs"], w_exc=40.0 / min(0.1 * case["n"], 100.0),
                                                        w_inh=80.0 / min(0.1 * case["n"], 100.0)))
        rng = np.random.default_rng([seed, 3])
        net.weight = (rng.random(net.n_synapses) * net.max_weight).astype(np.float32)
        return net, *poisson_input_times(rng, case["inputs"], 20.0, total * 1e-4)
    if case["kind"] == "layer":
        g = case["granule"]
        return configs.cerebellar_layer(seed=seed, n_granule=g, n_mossy=max(40, g // 50), n_purkinje=case["purkinje"],
                                        pf_per_purkinje=case["fan_in"], t_end=total * 1e-4, w_pf=2500.0 / case["fan_in"],
                                        w_pf_max=5000.0 / case["fan_in"])
    scale = 100.0 / case["indegree"]  # the same mean recurrent drive at every in-degree
    return configs.hh_network(seed=seed, n=case["n"], indeg=case["indegree"], t_end=total * 5e-5, w_exc=3.0 * scale,
                              w_inh=12.0 * scale, unique_times=False)


def _prepare_network(case, seed):
    net, times, cells = _network(case, seed)
    sim = Simulation.from_description(net, record_capacity=4 << 20, bucket_limit=64 if case["kind"] == "hh" else 0)
    dt = net.layers[1].dt
    settled = case["settle"]
    if settled:
        now = times < settled * dt
        sim.inject_spikes(times[now], cells[now])
        sim.run(settled)
        sim.spikes()
    # the inputs of each pass, as times after the pass's first step
    passes = []
    for k in range(settled, settled + case["trial"] - case["steps"] + 1, case["steps"]):
        start = sim.step_time(k)
        m = (times >= start) & (times < sim.step_time(k + case["steps"]))
        passes.append((times[m].astype(np.float64) - start, cells[m]))
    first, count = net.layers[0].n, net.n_neurons - net.layers[0].n
    return dict(kind="network", sim=sim, steps=case["steps"], done=settled, at=0, passes=passes, first=first, count=count,
                plastic=bool(net.rules), spikes=_Padded(count, case["steps"], dt, {"layer": 20.0, "hh": 1000.0}.get(case["kind"], 400.0)))


class _Padded:
    """Buffers that a program keeps for a pass's spikes, -1 after the last one."""

    def __init__(self, neurons, steps, dt, mean_hz):
        room = int(min(neurons * steps, neurons * steps * dt * mean_hz + 1000))
        self.step, self.cell, self.used = np.full(room, -1, np.int64), np.full(room, -1, np.int64), 0

    def put(self, step, cell):
        n = len(step)
        for buffer, new in ((self.step, step), (self.cell, cell)):
            buffer[:n] = new
            buffer[n:self.used] = -1
        self.used = n
        return dict(step=self.step, cell=self.cell)


def _run_network(s):
    sim = s["sim"]
    times, cells = s["passes"][s["at"] % len(s["passes"])]
    sim.inject_spikes(times + sim.step_time(s["done"]), cells)
    sim.run(s["steps"])
    s["done"] += s["steps"]
    s["at"] += 1
    out = dict(s["spikes"].put(*sim.spikes()), v=sim.get_state(s["first"], s["count"], 0))
    if s["plastic"]:
        out["weights"] = sim.weights()
    return out


def _sweep_specs(case, seed):
    """Networks whose sizes and parameters are the case's; connectivity, weights and input
    spikes come from the seed."""
    specs = configs.sweep_networks(seed=1, n_networks=case["networks"], n_min=case["n_min"], n_max=case["n_max"],
                                   t_end=1e-3)
    for i, sp in enumerate(specs):
        times, cells = poisson_input_times(np.random.default_rng([seed, i]), sp["n_in"], 10.0, case["steps"] * 1e-4)
        sp.update(times=times, cells=cells.astype(np.int32))
    return specs


def _prepare_sweep(case, seed):
    specs = _sweep_specs(case, seed)
    sw = Sweep.from_specs(specs, n_steps_max=case["steps"], integrator=case["integrator"], seed=seed, max_rate_hz=500.0)
    sw.set_observed(np.stack([np.linspace(0, sp["n"] - 1, case["observed"]).astype(np.int32) for sp in specs]))
    trace = torch.empty(case["networks"], case["steps"], case["observed"], device=DEVICE)
    spikes = _Padded(int(sw.sizes.sum()), case["steps"], 1e-4, 400.0) if case["spikes"] else None
    return dict(kind="sweep", sweep=sw, steps=case["steps"], trace=trace, spikes=spikes)


def _run_sweep(s):
    sw = s["sweep"]
    sw.reset()
    sw.run(s["steps"])
    out = dict(trace=sw.trace(s["steps"], out=s["trace"]), counts=sw.spike_counts())
    if s["spikes"]:
        spikes = [sw.spikes(i) for i in range(sw.n_networks)]
        out.update(s["spikes"].put(np.concatenate([a for a, _ in spikes]), np.concatenate([b for _, b in spikes])))
    return out


def _fit_specs(case, seed):
    rng = np.random.default_rng([seed, 7])
    sizes = np.exp(np.linspace(np.log(case["n_min"]), np.log(case["n_max"]), case["networks"] + 1)[1:]).astype(int)
    specs, hidden, observed = [], [], []
    for i, n in enumerate(sizes):
        sp = configs.adjoint_networks(seed=seed + 1000 * i, n_networks=1, n=int(n), indeg=min(100, int(n) // 4), rate_hz=20.0,
                                      t_end=case["steps"] * 1e-4)[0]
        hidden.append([configs.perturbed_params(sp["params"], rng)[k] for k in configs.ADJOINT_PARAMS])
        specs.append(sp)
        observed.append(rng.choice(int(n), case["observed"], replace=False))
    return specs, np.array(hidden), np.stack(observed)


def _prepare_fit(case, seed):
    specs, hidden, observed = _fit_specs(case, seed)
    model = TraceModel(specs, case["steps"], observed, integrator=case["integrator"], checkpoint_every=100)
    params = model.initial_params()
    weights = model.initial_weights()
    with torch.no_grad():
        target = model(torch.from_numpy(hidden), weights)
    return dict(kind="fit", model=model, params=params.requires_grad_(), weights=weights.requires_grad_(), target=target)


def _run_fit(s):
    s["params"].grad = s["weights"].grad = None
    trace = s["model"](s["params"], s["weights"])
    loss = ((trace - s["target"]) ** 2).mean()
    loss.backward()
    return dict(trace=trace.detach(), loss=loss.detach(), params=s["params"].grad, weights=s["weights"].grad)


def _fold_inputs(case, seed):
    g = torch.Generator().manual_seed(seed)
    n, m = case["arrivals"], case["targets"]
    target = torch.randint(0, m, (n,), generator=g, dtype=torch.int32)
    # three of four synapses excitatory, a few NMDA; a step's arrivals share few distinct times
    kind = torch.tensor([0, 0, 0, 0, 0, 0, 1, 1, 2, 0, 0, 0], dtype=torch.int8)[torch.randint(0, 12, (n,), generator=g)]
    weight = torch.rand(n, generator=g)
    time = 0.1 + torch.randint(0, 50, (n,), generator=g).double() * 1e-6
    return target, kind, weight, time, [5.0 * torch.rand(m, generator=g) for _ in range(3)]


def _prepare_fold(case, seed):
    target, kind, weight, time, conductance = _fold_inputs(case, seed)
    return dict(kind="fold", lib=_lib.load(), batch=[x.to(DEVICE) for x in (target, kind, weight, time)], targets=case["targets"],
                conductance=[x.to(DEVICE) for x in conductance])


def _run_fold(s):
    out = [g.clone() for g in s["conductance"]]
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    _lib.check(s["lib"].eb_fold_arrivals(stream, s["batch"][0].numel(), *(x.data_ptr() for x in s["batch"]), s["targets"],
                                         *(x.data_ptr() for x in out)))
    return out


def prepare(case, seed):
    seed = int(seed)
    if case["kind"] == "sweep":
        return _prepare_sweep(case, seed)
    if case["kind"] == "fit":
        return _prepare_fit(case, seed)
    if case["kind"] == "fold":
        return _prepare_fold(case, seed)
    return _prepare_network(case, seed)


def run(state):
    return {"network": _run_network, "sweep": _run_sweep, "fit": _run_fit, "fold": _run_fold}[state["kind"]](state)


# ------------------------------------------------------------------ work --
def work(case):
    """Bytes: each neuron's state read and written once a step (32 B; 48 B for HH and 96 B
    of its BDF2 history), 8 B per synaptic event at the rates these networks settle to,
    and the outputs.  Flops: the integrator's derivative evaluations."""
    kind = case["kind"]
    if kind == "fold":
        return dict(bytes=17.0 * case["arrivals"] + 24.0 * case["targets"], flops=1.0 * case["arrivals"])
    steps = case["steps"]
    if kind in ("sweep", "fit"):
        mean = (case["n_max"] - case["n_min"]) / math.log(case["n_max"] / case["n_min"])
        n = case["networks"] * mean
        evals = {"Euler": 1, "RK2": 2, "RK4": 4}[case["integrator"]]
        if kind == "sweep":
            return dict(bytes=32.0 * n + 8.0 * steps * n * 0.002 * 0.1 * mean + 4.0 * case["networks"] * steps * case["observed"],
                        flops=12.0 * evals * n * steps)
        # forward, recomputation and adjoint; the weights and their gradients once
        synapses = n * (min(100, case["n_min"] // 4) + 10)
        return dict(bytes=8.0 * synapses + 8.0 * case["networks"] * steps * case["observed"], flops=12.0 * 4 * evals * n * steps)
    if kind == "layer":
        neurons, evals, ops = case["granule"] + case["purkinje"], 4, 20
        synapses, per_neuron = 4 * case["granule"] + case["purkinje"] * case["fan_in"], 32
        events = case["granule"] * 4 * 27e-4 + case["purkinje"] * case["fan_in"] * 0.7e-4
        plastic = True
    elif kind == "hh":
        neurons, evals, ops, per_neuron, plastic = case["n"], 5, 160, 144, False
        synapses = case["n"] * (case["indegree"] + 1)
        events = case["n"] * (case["indegree"] * 5e-3 + 1e-2)
    else:
        neurons, per_neuron, plastic = case["n"], 32, kind == "adex"
        evals, ops = {"Euler": 1, "RK2": 2, "RK4": 4, "BDF": 10}[case["integrator"]], 14
        synapses = case["n"] * min(0.1 * case["n"], 100)
        events = synapses * 2e-3
    return dict(bytes=float(steps) * (per_neuron * neurons + 8.0 * events) + (4.0 * synapses if plastic else 0.0) + 4.0 * neurons,
                flops=float(steps) * neurons * evals * ops)


# ----------------------------------------------------------------- exact --
# The same methods in 64 bits with plain torch: exponentials evaluated where the models
# tabulate them, sums in any order, implicit steps solved to convergence.
def _arrivals(grid, when):
    """First step whose update time is after each time of `when`."""
    return np.searchsorted(grid, when, side="right")


def _grid(dt, steps):
    return np.concatenate([[0.0], np.cumsum(np.full(steps, float(np.float32(dt))))])


def _factor(dt_ms, tau):
    return torch.exp(-dt_ms / tau) if isinstance(tau, torch.Tensor) else math.exp(-dt_ms / tau)


def _decay(g, factors):
    return [torch.where(x < 1e-9, torch.zeros_like(x), x * f) for x, f in zip(g, factors)]


def _refractory(updates, tau_ref, dt):
    """Fraction of the derivative that a LIF neuron integrates, from its updates since a spike."""
    since, dt_ms = updates.double() * dt * 1000.0, dt * 1000.0
    part = ((since + dt_ms - tau_ref) / dt_ms).clamp(0.0, 1.0)
    return torch.where((updates < 0) | (since > tau_ref), torch.ones_like(part), part)


def _explicit(f, x, g, dt_ms, factors, method):
    """One step of Euler, RK2 or RK4 on the state tuple x with decaying conductances g
    (RK4's factors are those of half a step)."""
    step = lambda a, k, h: [u + v * h for u, v in zip(a, k)]  # noqa: E731
    k1 = f(x, g)
    if method == "Euler":
        return step(x, k1, dt_ms), _decay(g, factors)
    if method == "RK2":
        after = _decay(g, factors)
        k2 = f(step(x, k1, dt_ms), after)
        return step(x, [(a + b) * 0.5 for a, b in zip(k1, k2)], dt_ms), after
    half = _decay(g, factors)
    k2 = f(step(x, k1, dt_ms / 2), half)
    k3 = f(step(x, k2, dt_ms / 2), half)
    after = _decay(half, factors)
    k4 = f(step(x, k3, dt_ms), after)
    return step(x, [(a + 2 * (b + c) + d) / 6 for a, b, c, d in zip(k1, k2, k3, k4)], dt_ms), after


def _derivative(model, p, state):
    if model == "LIFTimeDrivenModel":
        def f(x, g):
            v = x[0]
            return [state["fraction"] * (g[0] * (p["e_exc"] - v) + g[1] * (p["e_inh"] - v) + p["g_leak"] * (p["e_leak"] - v)) / p["c_m"]]
    elif model == "AdExTimeDrivenModel":
        def f(x, g):
            v = x[0].clamp(max=p["v_thr"] + 6 * p["thr_slo_fac"])
            dv = (p["g_leak"] * (p["e_leak"] - v) + p["g_leak"] * p["thr_slo_fac"] * torch.exp((v - p["v_thr"]) / p["thr_slo_fac"])
                  - x[1] + g[0] * (p["e_exc"] - v) + g[1] * (p["e_inh"] - v)) / p["c_m"]
            dw = (p["a"] * (x[0] - p["e_leak"]) - x[1]) / p["tau_w"]
            below = x[0] <= 0.0
            return [torch.where(below, d, torch.zeros_like(d)) for d in (dv, dw)]
    else:
        def f(x, g):
            v, m, h, n = x[0].clamp(p["e_k"], p["e_na"] - 1.0), x[1].clamp(0, 1), x[2].clamp(0, 1), x[3].clamp(0, 0.72)
            u = v - p["v_thr"]
            current = g[0] * (p["e_exc"] - v) + g[1] * (p["e_inh"] - v)
            dv = (current + p["g_leak"] * (p["e_leak"] - v) + p["g_na"] * m ** 3 * h * (p["e_na"] - v) + p["g_kd"] * n ** 4 * (p["e_k"] - v)) / p["c_m"]
            am, bm = 0.32 * (13.0 - u) / torch.expm1((13.0 - u) / 4.0), 0.28 * (u - 40.0) / torch.expm1((u - 40.0) / 5.0)
            ah, bh = 0.128 * torch.exp((17.0 - u) / 18.0), 4.0 / (1.0 + torch.exp((40.0 - u) / 5.0))
            an, bn = 0.032 * (15.0 - u) / torch.expm1((15.0 - u) / 5.0), 0.5 * torch.exp((10.0 - u) / 40.0)
            return [dv, am * (1 - m) - bm * m, ah * (1 - h) - bh * h, an * (1 - n) - bn * n]
    return f


def _bdf2(f, x, g, dt_ms, factors, state):
    """One step of the second-order backward differentiation formula (the first step of a
    neuron's history is backward Euler), solved by Newton's method."""
    after = _decay(g, factors)
    deep = (state["history"] >= 2)[:, None]
    now = torch.stack(x, 1)
    c0 = torch.where(deep, 2.0 / 3.0, 1.0)
    known = torch.where(deep, (4.0 * now - state["last"]) / 3.0, now)
    y = now + torch.where(state["history"][:, None] > 0, now - state["last"], torch.zeros_like(now))
    rate = lambda z: torch.stack(f(list(z.unbind(1)), after), 1)  # noqa: E731
    eye = torch.eye(len(x), dtype=y.dtype, device=y.device)
    for _ in range(12):
        fy = rate(y)
        jac = torch.stack([(rate(y + 1e-7 * eye[j]) - fy) / 1e-7 for j in range(len(x))], 2)
        move = torch.linalg.solve(c0[..., None] * dt_ms * jac - eye, y - c0 * dt_ms * fy - known)
        y = y + move
        if float(move.abs().max()) < 1e-9:
            break
    state["last"] = now
    state["history"] = (state["history"] + 1).clamp(max=2)
    return list(y.unbind(1)), after, state


def _exact_network(case, seed):
    net, times, cells = _network(case, seed)
    steps = case["settle"] + case["steps"]
    cost = steps * (net.n_synapses * 2e-10 + 1.5e-3 * (12 if any(l.integrator == "BDF" for l in net.layers) else 1))
    if cost > 15.0:
        return None
    dt = float(np.float32(net.layers[1].dt))
    dt_ms = dt * 1000.0
    grid = _grid(dt, steps + 200)
    dev = lambda a, t=torch.float64: torch.as_tensor(np.ascontiguousarray(a), dtype=t, device=DEVICE)  # noqa: E731
    size = net.n_neurons
    units = np.floor(net.delay.astype(np.float64) * 1e4 + 5e-5).astype(np.int64)
    weight, cap = dev(net.weight), dev(net.max_weight)
    source, slot = dev(net.src, torch.int64), dev(net.tgt + size * net.stype, torch.int64)
    target, plastic = dev(net.tgt, torch.int64), dev(net.wchange >= 0, torch.bool)
    groups = {int(u): dev(np.nonzero(units == u)[0], torch.int64) for u in np.unique(units)}
    pre, post, last = (torch.zeros_like(weight) for _ in range(3))
    rule = net.rules[0][1] if net.rules else None
    into = dev(np.nonzero(net.wchange >= 0)[0], torch.int64)
    g_all = torch.zeros(2 * size, dtype=torch.float64, device=DEVICE)
    learns = np.zeros(size, bool)
    learns[net.src[net.wchange >= 0]] = True
    # what arrives at each step: (time, delay group, sources); the time within the step
    # matters to plastic synapses alone
    due = [[] for _ in range(steps + 1)]
    for u in groups:
        ka = _arrivals(grid, times.astype(np.float64) + u * 1e-4)
        for t, c, k in zip(times.astype(np.float64), cells, ka):
            if k <= steps:
                due[k].append((t + u * 1e-4, u, np.array([c])))
    pops, first = [], 0
    for layer in net.layers:
        if layer.model != "InputSpikeNeuronModel":
            p = layer.full_params()
            half = dt_ms / 2 if layer.integrator == "RK4" else dt_ms
            z = lambda v: torch.full((layer.n,), float(v), dtype=torch.float64, device=DEVICE)  # noqa: E731
            x = [z(p["e_leak"])]
            if layer.model == "AdExTimeDrivenModel":
                x.append(z(0.0))
            state = dict(history=torch.zeros(layer.n, dtype=torch.int64, device=DEVICE), updates=torch.full((layer.n,), -1, device=DEVICE))
            if layer.model == "HHTimeDrivenModel":
                u = p["e_leak"] - p["v_thr"]
                rates = [(0.32 * (13 - u) / math.expm1((13 - u) / 4), 0.28 * (u - 40) / math.expm1((u - 40) / 5)),
                         (0.128 * math.exp((17 - u) / 18), 4 / (1 + math.exp((40 - u) / 5))),
                         (0.032 * (15 - u) / math.expm1((15 - u) / 5), 0.5 * math.exp((10 - u) / 40))]
                x += [z(a / (a + b)) for a, b in rates]
            state["last"] = torch.stack(x, 1)
            pops.append(dict(layer=layer, p=p, x=x, state=state, f=_derivative(layer.model, p, state), at=slice(first, first + layer.n),
                             factors=[_factor(half, p["tau_exc"]), _factor(half, p["tau_inh"])]))
        first += layer.n
    fired = torch.zeros(size, dtype=torch.bool, device=DEVICE)
    for k in range(1, steps + 1):
        events = {}
        for t, u, who in due[k]:
            events.setdefault((t if learns[who].any() else 0.0, u), []).append(who)
        for t, u in sorted(events):
            fired.zero_()
            fired[dev(np.concatenate(events[t, u]), torch.int64)] = True
            at = groups[u][fired[source[groups[u]]]]
            g_all.index_add_(0, slot[at], weight[at])
            at = at[plastic[at]]
            if rule and len(at):  # pre-synaptic update, at the arrival
                pre[at] = pre[at] * torch.exp(-(t - last[at]) / rule[1]) + 1.0
                post[at] = post[at] * torch.exp(-(t - last[at]) / rule[3])
                weight[at] = torch.minimum((weight[at] - rule[2] * post[at]).clamp(min=0.0), cap[at])
                last[at] = t
        for q in pops:
            s, p, layer = q["state"], q["p"], q["layer"]
            g = [g_all[:size][q["at"]], g_all[size:][q["at"]]]
            before = q["x"][0]
            if layer.model == "LIFTimeDrivenModel":
                s["fraction"] = _refractory(s["updates"], p["tau_ref"], dt)
            if layer.integrator == "BDF":
                x, g, _ = _bdf2(q["f"], q["x"], g, dt_ms, q["factors"], s)
            else:
                x, g = _explicit(q["f"], q["x"], g, dt_ms, q["factors"], layer.integrator)
            if layer.model == "HHTimeDrivenModel":
                spike = (x[0] > -30.0) & (before < -30.0)
            else:
                limit, reset = (p["v_thr"], p["e_leak"]) if layer.model == "LIFTimeDrivenModel" else (0.0, p["e_reset"])
                spike = x[0] > limit
                x[0] = torch.where(spike, reset, x[0])
                if layer.model == "AdExTimeDrivenModel":
                    x[1] = torch.where(spike, x[1] + p["b"], x[1])
                s["history"] = torch.where(spike, 0, s["history"])
                s["updates"] = torch.where(spike, 0, torch.where(s["updates"] >= 0, s["updates"] + 1, s["updates"]))
            q["x"] = x
            g_all[:size][q["at"]], g_all[size:][q["at"]] = g
            who = (torch.nonzero(spike)[:, 0] + q["at"].start).cpu().numpy()
            if not len(who):
                continue
            for u in groups:
                ka = int(_arrivals(grid, grid[k] + u * 1e-4))
                if ka <= steps:
                    due[ka].append((grid[k] + u * 1e-4, u, who))
            if rule:  # post-synaptic update, at the spike
                fired.zero_()
                fired[dev(who, torch.int64)] = True
                at = into[fired[target[into]]]
                pre[at] = pre[at] * torch.exp(-(grid[k] - last[at]) / rule[1])
                post[at] = post[at] * torch.exp(-(grid[k] - last[at]) / rule[3]) + 1.0
                weight[at] = torch.minimum((weight[at] + rule[0] * pre[at]).clamp(min=0.0), cap[at])
                last[at] = grid[k]
    out = dict(step=None, cell=None, v=torch.cat([q["x"][0] for q in pops]))
    if net.rules:
        out["weights"] = weight
    return out


def _mix(z):
    """splitmix64 on 64-bit words held in signed integers."""
    shift = lambda v, s: (v >> s) & ((1 << (64 - s)) - 1)  # noqa: E731
    z = z + (0x9E3779B97F4A7C15 - (1 << 64))
    z = (z ^ shift(z, 30)) * (0xBF58476D1CE4E5B9 - (1 << 64))
    z = (z ^ shift(z, 27)) * (0x94D049BB133111EB - (1 << 64))
    return z ^ shift(z, 31)


def _hash_synapses(spec, net, seed):
    """The connectivity that a sweep draws for network `net`: (source, target, weight)."""
    word = (net + 1) * 0xD1B54A32D192ED03 & ((1 << 64) - 1)
    key = _mix(torch.tensor([(seed ^ word) - (1 << 64 if (seed ^ word) >> 63 else 0)], dtype=torch.int64, device=DEVICE))
    s = torch.arange(spec["n"] + spec["n_in"], device=DEVICE)[:, None]
    t = torch.arange(spec["n"], device=DEVICE)[None, :]
    h = _mix(key ^ ((s << 32) | t))
    hit = ((h >> 11) & ((1 << 53) - 1)).double() * 2.0 ** -53 < float(np.float32(spec["p"]))
    src, tgt = torch.nonzero(hit, as_tuple=True)
    u = ((_mix(h[hit]) >> 40) & ((1 << 24) - 1)).float() * 2.0 ** -24
    top = torch.full((spec["n"] + spec["n_in"],), spec["w_in_max"], device=DEVICE)
    top[:spec["n_exc"]], top[spec["n_exc"]:spec["n"]] = spec["w_exc_max"], spec["w_inh_max"]
    return src, tgt, (u * top[src]).double()


def _lif_batch(specs, synapses, params, weight, steps, method, observed, dt=1e-4, delay=1e-3):
    """Membrane traces [network, step, observed] and spike counts of independent LIF
    networks in 64 bits; differentiable in `params` [network, 4] and `weight`."""
    dt = float(np.float32(dt))
    dt_ms = dt * 1000.0
    grid = _grid(dt, steps + 50)
    sizes = torch.tensor([s["n"] for s in specs], device=DEVICE)
    total, owner = int(sizes.sum()), torch.repeat_interleave(torch.arange(len(specs), device=DEVICE), sizes)
    start = np.concatenate([[0], np.cumsum([s["n"] for s in specs])])
    start_in = total + np.concatenate([[0], np.cumsum([s["n_in"] for s in specs])])
    src = torch.cat([torch.where(a < s["n"], a + int(start[i]), a - s["n"] + int(start_in[i])) for i, (s, (a, _, _)) in enumerate(zip(specs, synapses))])
    inhibitory = torch.cat([(a >= s["n_exc"]) & (a < s["n"]) for s, (a, _, _) in zip(specs, synapses)])
    slot = torch.cat([b + int(start[i]) for i, (_, b, _) in enumerate(synapses)]) + total * inhibitory
    each = {k: torch.tensor([s["params"][k] for s in specs], dtype=torch.float64, device=DEVICE)[owner] for k in ("e_exc", "e_inh", "v_thr", "c_m", "tau_ref")}
    each |= {k: params[:, j][owner] for j, k in enumerate(configs.ADJOINT_PARAMS)}
    half = dt_ms / 2 if method == "RK4" else dt_ms
    factors = [_factor(half, each["tau_exc"]), _factor(half, each["tau_inh"])]
    inputs = [[] for _ in range(steps + 1)]
    for i, s in enumerate(specs):
        for k, c in zip(_arrivals(grid, s["times"].astype(np.float64) + delay), s["cells"]):
            if k <= steps:
                inputs[k].append(int(start_in[i]) + int(c))
    state = dict(updates=torch.full((total,), -1, device=DEVICE))
    f = _derivative("LIFTimeDrivenModel", each, state)
    x, g = [each["e_leak"]], [torch.zeros(total, dtype=torch.float64, device=DEVICE) for _ in range(2)]
    due, counts, rows = {}, torch.zeros(len(specs), dtype=torch.int64, device=DEVICE), []
    watch = torch.cat([torch.as_tensor(o, device=DEVICE) + int(start[i]) for i, o in enumerate(observed)])
    for k in range(1, steps + 1):
        fired = torch.zeros(int(start_in[-1]), dtype=weight.dtype, device=DEVICE)
        if inputs[k]:
            fired.index_add_(0, torch.tensor(inputs[k], device=DEVICE), torch.ones(len(inputs[k]), dtype=weight.dtype, device=DEVICE))
        for spike in due.pop(k, []):
            fired[:total] += spike
        at = torch.nonzero(fired[src])[:, 0]
        if len(at):
            both = torch.cat(g).index_add(0, slot[at], weight[at] * fired[src[at]])
            g = [both[:total], both[total:]]
        state["fraction"] = _refractory(state["updates"], each["tau_ref"], dt)
        x, g = _explicit(f, x, g, dt_ms, factors, method)
        spike = x[0] > each["v_thr"]
        x = [torch.where(spike, each["e_leak"], x[0])]
        state["updates"] = torch.where(spike, 0, torch.where(state["updates"] >= 0, state["updates"] + 1, state["updates"]))
        counts += torch.bincount(owner[spike], minlength=len(specs))
        due.setdefault(int(_arrivals(grid, grid[k] + delay)), []).append(spike.to(weight.dtype))
        rows.append(x[0][watch])
    return torch.stack(rows, 1).reshape(len(specs), -1, steps).transpose(1, 2), counts


def _exact_sweep(case, seed):
    specs = _sweep_specs(case, seed)
    if sum(s["n"] ** 2 for s in specs) > 3e8:
        return None
    synapses = [_hash_synapses(s, i, seed) for i, s in enumerate(specs)]
    params = torch.tensor([[s["params"][k] for k in configs.ADJOINT_PARAMS] for s in specs], dtype=torch.float64, device=DEVICE)
    observed = [np.linspace(0, s["n"] - 1, case["observed"]).astype(np.int64) for s in specs]
    trace, _ = _lif_batch(specs, synapses, params, torch.cat([w for _, _, w in synapses]), case["steps"], case["integrator"], observed)
    return dict(trace=trace, counts=None, **(dict(step=None, cell=None) if case["spikes"] else {}))


def _exact_fit(case, seed):
    specs, hidden, observed = _fit_specs(case, seed)
    if sum(len(s["w"]) for s in specs) * case["steps"] > 5e8:
        return None
    synapses = [tuple(torch.from_numpy(s[k].astype(t)).to(DEVICE) for k, t in (("src", np.int64), ("tgt", np.int64), ("w", np.float64))) for s in specs]
    weight = torch.cat([w for _, _, w in synapses])
    args = (case["steps"], case["integrator"], list(observed))
    with torch.no_grad():
        target, _ = _lif_batch(specs, synapses, torch.from_numpy(hidden).to(DEVICE), weight, *args)
    params = torch.tensor([[s["params"][k] for k in configs.ADJOINT_PARAMS] for s in specs], dtype=torch.float64, device=DEVICE).requires_grad_()
    weight.requires_grad_()
    trace, _ = _lif_batch(specs, synapses, params, weight, *args)
    loss = ((trace - target) ** 2).mean()
    loss.backward()
    return dict(trace=trace.detach(), loss=loss.detach(), params=params.grad, weights=weight.grad)


def _exact_fold(case, seed):
    target, kind, weight, _, conductance = _fold_inputs(case, seed)
    return [g.double().index_add_(0, target[kind == j].long(), weight[kind == j].double()) for j, g in enumerate(conductance)]


def exact(case, seed):
    seed = int(seed)
    return {"sweep": _exact_sweep, "fit": _exact_fit, "fold": _exact_fold}.get(case["kind"], _exact_network)(case, seed)
