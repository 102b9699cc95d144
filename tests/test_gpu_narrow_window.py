"""GPU test of the staged window of the thread-per-neuron update: every step's
arrivals folded in delivery order whatever their number.  A population is driven by
bursts of inputs through plastic or fixed synapses, so that a window's arrivals
end just below, at and beyond the stage of a warp, one step's alone beyond it, and
a neuron's beyond 255 in one step, with inputs that deliver twice in a step; spikes,
traces and weights equal the CPU oracle's bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def burst_network(model, integrator, n, burst, plastic, dt=1e-4):
    from edlut_b200.network import Layer, NetworkDescription
    rng = np.random.default_rng([n, burst])
    net = NetworkDescription()
    inp = net.add_layer(Layer(burst, "InputSpikeNeuronModel", output=0))
    pop = net.add_layer(Layer(n, model, {}, integrator=integrator, dt=dt, name="pop"))
    net.rules.append(("STDP", [0.004, 0.02, 0.0042, 0.02]))
    w = 40.0 / burst
    # every input reaches every neuron; a third of them inhibitory; delays of 1 and 1.4 ms
    src, tgt = np.repeat(inp, n), np.tile(pop, burst)
    delay = np.where(rng.random(len(src)) < 0.5, 1e-3, 1.4e-3)
    net.add_synapses(src, tgt, delay, (src % 3 == 2).astype(np.int32), (rng.random(len(src)) * w).astype(np.float32), 2 * w,
                     np.where(rng.random(len(src)) < 0.7, 0, -1) if plastic else -1)
    # recurrent plastic synapses, so that a target's own spikes fall between arrivals
    rs, rt = rng.integers(0, n, 4 * n) + pop.start, rng.integers(0, n, 4 * n) + pop.start
    net.add_synapses(rs, rt, 1e-3, 0, np.float32(0.5), np.float32(1.0), 0 if plastic else -1)
    times, cells = [], []
    for step, size in ((5, 1), (20, burst), (21, burst // 2), (23, 2), (40, burst // 3), (41, burst // 3), (60, burst)):
        who = rng.choice(burst, max(1, size), replace=False)
        times.append((step + 0.1 + 0.5 * rng.random(len(who))) * dt)
        cells.append(who)
    for step in (50, 61):  # an input firing twice inside one step
        times.append((step + np.array([0.2, 0.75])) * dt)
        cells.append(np.array([0, 0]))
    t, c = np.concatenate(times).astype(np.float32), np.concatenate(cells)
    o = np.argsort(t, kind="stable")
    return net, t[o], c[o] + inp.start


@pytest.mark.parametrize("plastic", [True, False])
@pytest.mark.parametrize("model,integrator,n,burst", [
    ("LIFTimeDrivenModel", "Euler", 3, 15), ("LIFTimeDrivenModel", "RK4", 33, 16), ("AdExTimeDrivenModel", "RK2", 5, 17),
    ("LIFTimeDrivenModel", "BDF", 4, 64), ("AdExTimeDrivenModel", "Euler", 6, 300), ("HHTimeDrivenModel", "BDF", 9, 32),
    ("HHTimeDrivenModel", "RK4", 4, 130)])
def test_burst_sizes_match_oracle(model, integrator, n, burst, plastic):
    from edlut_b200.simulation import Simulation
    from oracle import oracle as O
    net, t, c = burst_network(model, integrator, n, burst, plastic)
    first, steps = net.layers[0].n, 96
    o = O.run(net, t, c, steps, trace=(steps, first, n))
    sim = Simulation.from_description(net)
    sim.inject_spikes(t, c)
    sim.set_trace(first, n, steps)
    sim.run(steps)
    st, ce = sim.spikes()
    trace, w = sim.get_trace(), sim.weights()
    sim.close()
    assert sorted(zip(st.tolist(), ce.tolist())) == sorted(zip(o["spike_step"].tolist(), o["spike_cell"].tolist()))
    np.testing.assert_array_equal(trace, o["trace"].astype(np.float32))
    np.testing.assert_array_equal(w, o["w_final"].astype(np.float32))


# Arrivals of one step at each neuron, around the 255 from which a lane's packed count is
# read again; all at one delay, so that they come in the same step.
SATURATED = (254, 255, 256, 300, 17, 1, 0, 511)


def saturated_network(model, integrator, plastic, dt=1e-4):
    from edlut_b200.network import Layer, NetworkDescription
    rng = np.random.default_rng(len(model))
    net = NetworkDescription()
    inp = net.add_layer(Layer(max(SATURATED), "InputSpikeNeuronModel", output=0))
    pop = net.add_layer(Layer(len(SATURATED), model, {}, integrator=integrator, dt=dt, name="pop"))
    net.rules.append(("STDP", [0.004, 0.02, 0.0042, 0.02]))
    src = np.concatenate([rng.choice(max(SATURATED), k, replace=False) for k in SATURATED])
    tgt = np.repeat(np.asarray(pop), SATURATED)
    net.add_synapses(src + inp.start, tgt, 1e-3, (src % 3 == 2).astype(np.int32), (rng.random(len(src)) * 0.15).astype(np.float32),
                     0.3, 0 if plastic else -1)
    net.add_synapses(np.asarray(pop), np.roll(pop, 1), 1e-3, 0, np.float32(0.5), np.float32(1.0), 0 if plastic else -1)
    steps = (5, 21, 22, 47)  # a burst alone, two in consecutive steps, one late in a window
    t = np.concatenate([(s + 0.1 + 0.5 * np.sort(rng.random(max(SATURATED)))) * dt for s in steps]).astype(np.float32)
    c = np.concatenate([rng.permutation(max(SATURATED)) for _ in steps]) + inp.start
    # the counts meant: every input fires once a burst, one delay, all inside one step
    grid = np.concatenate([[0.0], np.cumsum(np.full(100, float(np.float32(dt))))])
    arrival = np.searchsorted(grid, t.astype(np.float64) + 10 * 0.0001, side="right")
    for j, k in enumerate(SATURATED):
        own = np.bincount(arrival[np.isin(c - inp.start, src[tgt == pop.start + j])], minlength=100) if k else np.zeros(100, int)
        assert own.max() == k and (own == k).sum() == (len(steps) if k else 100)
    return net, t, c


@pytest.mark.parametrize("plastic", [True, False])
@pytest.mark.parametrize("model,integrator", [("LIFTimeDrivenModel", "Euler"), ("AdExTimeDrivenModel", "RK2"), ("HHTimeDrivenModel", "BDF")])
def test_counts_beyond_the_packed_byte_match_oracle(model, integrator, plastic):
    from edlut_b200.simulation import Simulation
    from oracle import oracle as O
    net, t, c = saturated_network(model, integrator, plastic)
    first, n, steps = net.layers[0].n, len(SATURATED), 80
    o = O.run(net, t, c, steps, trace=(steps, first, n))
    sim = Simulation.from_description(net)
    sim.inject_spikes(t, c)
    sim.set_trace(first, n, steps)
    sim.run(steps)
    st, ce = sim.spikes()
    trace, w, events = sim.get_trace(), sim.weights(), sim.counters()["events"]
    sim.close()
    assert sorted(zip(st.tolist(), ce.tolist())) == sorted(zip(o["spike_step"].tolist(), o["spike_cell"].tolist()))
    np.testing.assert_array_equal(trace, o["trace"].astype(np.float32))
    np.testing.assert_array_equal(w, o["w_final"].astype(np.float32))
    assert events == o["n_events"]
