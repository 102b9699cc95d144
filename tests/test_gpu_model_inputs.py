"""GPU test of input spikes injected into model neurons: they enter through the input
fan-out whether or not the network has an input layer, their targets' updates wait for
them, and one synapse may deliver twice in a step.  Injected before or after the network
is finalized, or between two runs; spikes, traces and weights equal the CPU oracle's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def model_input_network(inputs, dt=1e-4):
    from edlut_b200.network import Layer, NetworkDescription
    rng = np.random.default_rng(inputs + 1)
    net = NetworkDescription()
    inp = net.add_layer(Layer(inputs, "InputSpikeNeuronModel", output=0)) if inputs else None
    a = net.add_layer(Layer(20, "LIFTimeDrivenModel", {}, integrator="Euler", dt=dt, name="a"))
    b = net.add_layer(Layer(6, "LIFTimeDrivenModel", {}, integrator="RK2", dt=dt, name="b"))
    net.rules.append(("STDP", [0.004, 0.02, 0.0042, 0.02]))
    src, tgt = np.repeat(a, 6), np.tile(b, 20)
    delay = np.where(rng.random(len(src)) < 0.5, 1e-3, 1.4e-3)
    net.add_synapses(src, tgt, delay, 0, (1.0 + rng.random(len(src))).astype(np.float32), 4.0, 0)
    net.add_synapses(np.asarray(b), np.roll(b, 1), 1e-3, 0, np.float32(0.5), np.float32(1.0), 0)
    if inputs:
        net.add_synapses(np.repeat(inp, 20), np.tile(a, inputs), 1e-3, 0, np.float32(1.0), np.float32(2.0), -1)
    times, cells = [], []
    for step in (3, 4, 17, 18, 25, 40, 41, 42, 60, 77):
        who = rng.choice(20, 8, replace=False) + a.start
        times.append((step + 0.05 + 0.9 * rng.random(8)) * dt)
        cells.append(who)
        times.append((step + np.array([0.2, 0.75])) * dt)  # twice in a step
        cells.append(np.array([who[0], who[0]]))
        if inputs:
            times.append((step + 0.5) * dt * np.ones(inputs))
            cells.append(np.asarray(inp))
    t, c = np.concatenate(times).astype(np.float32), np.concatenate(cells)
    o = np.argsort(t, kind="stable")
    return net, t[o], c[o], a.start, 26


def build(net, before, **kw):
    from edlut_b200.network import MODEL_PARAM_ORDER
    from edlut_b200.simulation import Simulation
    sim = Simulation(**kw)
    for layer in net.layers:
        sim.add_population(layer.model, layer.n, layer.integrator, layer.bdf_order, layer.dt,
                           layer.full_params() if layer.model in MODEL_PARAM_ORDER else None)
    sim.add_stdp_rule(*net.rules[0][1])
    if before is not None:
        sim.inject_spikes(*before)
    sim.set_connectivity(net.src, net.tgt, net.delay, net.stype, net.weight, net.max_weight, net.wchange)
    sim.finalize()
    return sim


@pytest.mark.parametrize("when", ["before", "after", "between"])
@pytest.mark.parametrize("kernel", ["thread_per_neuron", "block_per_neuron", "persistent"])
@pytest.mark.parametrize("inputs", [0, 4])
def test_injected_model_neurons_match_oracle(inputs, kernel, when):
    from oracle import oracle as O
    net, t, c, first, n = model_input_network(inputs)
    steps = 96
    o = O.run(net, t, c, steps, trace=(steps, first, n))
    kw = dict(persistent=kernel == "persistent", wide_indegree=0 if kernel == "block_per_neuron" else None)
    sim = build(net, (t, c) if when == "before" else None, **kw)
    sim.set_trace(first, n, steps)
    if when == "between":  # the first model neuron's spikes come after a run
        early = (c < first) & (t < 2e-3)
        sim.inject_spikes(t[early], c[early])
        sim.run(2)
        sim.inject_spikes(t[~early], c[~early])
        sim.run(18)
        sim.run(steps - 20)
    else:
        if when == "after":
            sim.inject_spikes(t, c)
        sim.run(steps)
    st, ce = sim.spikes()
    trace, w = sim.get_trace(), sim.weights()
    sim.close()
    assert sorted(zip(st.tolist(), ce.tolist())) == sorted(zip(o["spike_step"].tolist(), o["spike_cell"].tolist()))
    np.testing.assert_array_equal(trace, o["trace"].astype(np.float32))
    np.testing.assert_array_equal(w, o["w_final"].astype(np.float32))
