"""GPU test of the weight transfer (eb_set_weights / eb_get_weights): every weight
comes back at its place in the network file's order, for synapse counts at the
edges of a block and of the empty network."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [0, 1, 255, 256, 257, 5000])
def test_weights_keep_file_order(m):
    from edlut_b200.network import Layer, NetworkDescription
    from edlut_b200.simulation import Simulation
    rng = np.random.default_rng(m)
    net = NetworkDescription()
    net.add_layer(Layer(7, "InputSpikeNeuronModel", output=0))
    net.add_layer(Layer(90, "LIFTimeDrivenModel", {}, integrator="RK2"))
    net.rules.append(("STDP", [0.01, 0.02, 0.0105, 0.02]))
    w = rng.random(m).astype(np.float32)
    # random sources, targets, delays and a mix of fixed and plastic synapses, in random order
    net.add_synapses(rng.integers(0, 97, m), 7 + rng.integers(0, 90, m), rng.choice([1e-3, 2e-3], m), rng.integers(0, 3, m), w,
                     np.float32(2.0), rng.integers(-1, 1, m))
    sim = Simulation.from_description(net)
    np.testing.assert_array_equal(sim.weights(), w)
    new = rng.random(m).astype(np.float32)
    sim.set_weights(new if m else np.zeros(1, np.float32))
    np.testing.assert_array_equal(sim.weights(), new)
    sim.close()


def test_weights_of_more_than_one_staging_pass():
    """More synapses than the staging buffer holds (8 << 20): the second pass takes the rest."""
    from edlut_b200.network import Layer, NetworkDescription
    from edlut_b200.simulation import Simulation
    m = (8 << 20) + 257
    rng = np.random.default_rng(1)
    net = NetworkDescription()
    net.add_layer(Layer(2000, "InputSpikeNeuronModel", output=0))
    net.add_layer(Layer(9000, "LIFTimeDrivenModel", {}, integrator="Euler"))
    w = rng.random(m, dtype=np.float32)
    net.add_synapses(rng.integers(0, 2000, m), 2000 + rng.integers(0, 9000, m), 1e-3, 0, w, np.float32(2.0), -1)
    sim = Simulation.from_description(net)
    np.testing.assert_array_equal(sim.weights(), w)
    new = rng.random(m, dtype=np.float32)
    sim.set_weights(new)
    np.testing.assert_array_equal(sim.weights(), new)
    sim.close()
