"""GPU test of the update kernels of populations too large for the register counts of the
small ones (eb_update.cu): every conductance set that has a kernel of its own, with and
without plastic inputs, at sizes just above the line, in a short run.  Spikes, membrane
potentials and weights equal the CPU oracle's bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LIF, ADEX, HH = "LIFTimeDrivenModel", "AdExTimeDrivenModel", "HHTimeDrivenModel"


def large_network(model, integrator, n, types, plastic, steps, dt=1e-4):
    from edlut_b200.network import Layer, NetworkDescription
    rng = np.random.default_rng([n, len(types)])
    net = NetworkDescription()
    inp = net.add_layer(Layer(200, "InputSpikeNeuronModel", output=0))
    pop = net.add_layer(Layer(n, model, {}, integrator=integrator, dt=dt, name="pop"))
    net.rules.append(("STDP", [0.004, 0.02, 0.0042, 0.02]))
    rule = 0 if plastic else -1
    scale = 60.0 if model == HH else 12.0
    tgt = np.repeat(np.asarray(pop), 3)
    net.add_synapses(rng.integers(0, 200, len(tgt)) + inp.start, tgt, 1e-3, types[0],
                     (scale * rng.random(len(tgt))).astype(np.float32), 2 * scale, rule)
    tgt = np.repeat(np.asarray(pop), 2)
    net.add_synapses(rng.integers(0, n, len(tgt)) + pop.start, tgt, 1e-3, rng.choice(types, len(tgt)).astype(np.int32),
                     (0.1 * scale * rng.random(len(tgt))).astype(np.float32), scale, rule)
    t = np.sort(rng.random(200 * 6) * steps * dt).astype(np.float32)
    return net, t, rng.integers(0, 200, len(t)) + inp.start


@pytest.mark.parametrize("plastic", [True, False])
@pytest.mark.parametrize("model,integrator,types", [
    (HH, "BDF", (0,)), (HH, "BDF", (0, 1)), (HH, "BDF", (0, 1, 2)), (HH, "RK4", (0, 1)),
    (LIF, "RK2", (0, 1)), (LIF, "BDF", (0,)), (LIF, "Euler", (0, 1, 2)), (ADEX, "Euler", (0,)), (ADEX, "RK4", (0, 1, 2))])
def test_large_populations_match_oracle(model, integrator, types, plastic):
    from edlut_b200.simulation import Simulation
    from oracle import oracle as O
    n, steps = 148 * 32 * (12 if model == HH else 16) + 33, 60
    net, t, c = large_network(model, integrator, n, types, plastic, steps)
    o = O.run(net, t, c, steps, trace=(steps, 200, 64))
    sim = Simulation.from_description(net, record_capacity=1 << 22)
    sim.inject_spikes(t, c)
    sim.set_trace(200, 64, steps)
    sim.run(steps)
    st, ce = sim.spikes()
    trace, w = sim.get_trace(), sim.weights()
    sim.close()
    assert len(o["spike_step"]) > 100
    np.testing.assert_array_equal(np.lexsort((ce, st)), np.arange(len(st)))
    order = np.lexsort((o["spike_cell"], o["spike_step"]))
    np.testing.assert_array_equal(st, o["spike_step"][order])
    np.testing.assert_array_equal(ce, o["spike_cell"][order])
    np.testing.assert_array_equal(trace, o["trace"].astype(np.float32))
    np.testing.assert_array_equal(w, o["w_final"].astype(np.float32))
