"""GPU parity through the C ABI: the sm_100a kernels against the reference's own
outputs (golden fixtures) and against the CPU oracle, on the same seeded inputs.

Criterion (bit-exact where the arithmetic is the reference's): spike (step, cell)
lists identical, state traces identical, final STDP weights identical, reference
synapse order identical.  The looser bound that the benchmark description allows
(>= 99.9% identical spike steps, the rest within one step; V RMS < 1e-3 mV over
the first 100 ms) is asserted as well, so a regression that breaks exactness but
not the bound is reported separately."""
import numpy as np
import pytest

from tests._cases import CASES, build_case, load_golden, perm_digest, spike_match_fraction, spike_pairs

pytestmark = pytest.mark.gpu


def run_gpu(net, t, c, nsteps, trace, **kw):
    from edlut_b200.simulation import Simulation
    sim = Simulation.from_description(net, **kw)
    sim.inject_spikes(t, c)
    ts, tf, tn = trace
    if tn:
        sim.set_trace(tf, tn, ts)
    sim.run(nsteps)
    st, ce = sim.spikes()
    out = dict(spikes=spike_pairs(st, ce), trace=sim.get_trace() if tn else None, w=sim.weights(),
               perm=sim.sorted_perm, counters=sim.counters())
    sim.close()
    return out


@pytest.mark.parametrize("kernel", ["default", "block_per_neuron"])
@pytest.mark.parametrize("persistent", [True, False], ids=["persistent", "graphs"])
@pytest.mark.parametrize("name", sorted(CASES))
def test_gpu_matches_reference_fixture(name, persistent, kernel):
    """kernel "default": a block per neuron only above 1,024 inputs (the Purkinje-
    type cells); "block_per_neuron": for every population that one step can give
    more than 16 arrivals, so both update kernels meet every fixture."""
    net, t, c, nsteps, trace = build_case(name)
    g = load_golden(name)
    r = run_gpu(net, t, c, nsteps, trace, persistent=persistent,
                wide_indegree=0 if kernel == "block_per_neuron" else None)
    ref = spike_pairs(g["spike_step"], g["spike_cell"])
    same, near = spike_match_fraction(ref, r["spikes"])
    assert same >= 0.999 and near == 1.0, (same, near)
    np.testing.assert_array_equal(r["spikes"], ref)
    nd = g["trace"].shape[2]
    a, b = r["trace"][:, :, 0], g["trace"][:, :, 0]
    d = np.where(a == b, 0.0, a.astype(np.float64) - b)  # equal infinities count as equal
    v_rms = float(np.sqrt(np.mean(d ** 2)))
    assert v_rms < 1e-3
    np.testing.assert_array_equal(r["trace"][:, :, :nd], g["trace"])
    if "w_final" in g:
        np.testing.assert_array_equal(r["w"], g["w_final"])
    assert r["counters"]["events"] == int(g["counts"][1])
    assert perm_digest(r["perm"]) == str(g["perm_sha256"])


@pytest.mark.parametrize("name", sorted(CASES))
def test_gpu_matches_oracle(oracle, name):
    net, t, c, nsteps, trace = build_case(name)
    o = oracle.run(net, t, c, nsteps, trace=trace)
    r = run_gpu(net, t, c, nsteps, trace)
    np.testing.assert_array_equal(r["spikes"], spike_pairs(o["spike_step"], o["spike_cell"]))
    np.testing.assert_array_equal(r["trace"][:, :, :], o["trace"].astype(np.float32)[:, :, :])
    np.testing.assert_array_equal(r["w"], o["w_final"].astype(np.float32))
    np.testing.assert_array_equal(r["perm"], o["sorted_perm"])
    assert r["counters"]["events"] == o["n_events"]
    assert r["counters"]["spikes"] == len(o["spike_step"])


def test_fp64_error_is_reported(oracle):
    """Error of the GPU V trace against the FP64 oracle over the first 100 ms of the
    recurrent LIF workload (stated, not a parity criterion; bounded loosely)."""
    net, t, c, nsteps, trace = build_case("c1_lif_euler")
    r = run_gpu(net, t, c, 1000, (1000, 100, 16))
    o64 = oracle.run(net, t, c, 1000, fp64=True, trace=(1000, 100, 16))
    rms = float(np.sqrt(np.mean((r["trace"][:, :, 0] - o64["trace"][:, :, 0]) ** 2)))
    print("V RMS vs FP64 oracle over 100 ms: %.3g mV" % rms)
    assert rms < 1e-2


@pytest.mark.parametrize("persistent", [True, False], ids=["persistent", "graphs"])
def test_gpu_wide_fanin_matches_oracle(oracle, persistent):
    """Block-per-neuron update at every arrival-count regime (tens of arrivals, up
    to 256, up to 1024 and beyond in one step), with STDP on every delivered
    synapse, deferred post-synaptic spikes, and a population whose input synapses
    can deliver twice in one step: bit-exact against the oracle."""
    from edlut_b200.configs import wide_fanin_network
    net, t, c = wide_fanin_network()
    first = sum(l.n for l in net.layers[:2])
    trace = (400, first, 6)
    o = oracle.run(net, t, c, 400, trace=trace)
    r = run_gpu(net, t, c, 400, trace, persistent=persistent)
    np.testing.assert_array_equal(r["spikes"], spike_pairs(o["spike_step"], o["spike_cell"]))
    np.testing.assert_array_equal(r["trace"], o["trace"].astype(np.float32))
    np.testing.assert_array_equal(r["w"], o["w_final"].astype(np.float32))
    assert r["counters"]["events"] == o["n_events"]


def test_gpu_fused_windows_equal_single_steps():
    """With 1 ms delays at 0.1 ms steps a launch of the captured graph runs 8 steps
    of a population: 128 steps of the small cerebellar case (one graph) take 3
    chains x 16 windows + two deferred-STDP flushes of the Purkinje chain (3
    launches each) + the step counter (1) launches; spikes, traces and weights
    equal those of one launch per step."""
    from edlut_b200.simulation import Simulation
    net, t, c, _, trace = build_case("cereb_small_rk4")
    out = []
    for graph_steps in (0, 1):
        sim = Simulation.from_description(net, graph_steps=graph_steps)
        sim.inject_spikes(t, c)
        sim.set_trace(trace[1], trace[2], 128)
        l0 = sim.launch_count()
        sim.run(128)
        n_launch = sim.launch_count() - l0  # before the drain, whose sort launches kernels of its own
        st, ce = sim.spikes()
        out.append((spike_pairs(st, ce), sim.get_trace(), sim.weights(), n_launch))
        sim.close()
    (s0, tr0, w0, n0), (s1, tr1, w1, _) = out
    assert n0 == 3 * 16 + 2 * 3 + 1, n0
    np.testing.assert_array_equal(s0, s1)
    np.testing.assert_array_equal(tr0, tr1)
    np.testing.assert_array_equal(w0, w1)


@pytest.mark.parametrize("name", ["cereb_small_rk4", "adex_rk4_stdp"])
def test_gpu_uneven_runs_match_fixture(name):
    """Runs of uneven lengths mix whole graphs, remainder graphs and single-step
    launches, with deferred post-synaptic STDP carried across them (partial flushes
    between runs, a full one before the weights are read): the result is the
    reference's."""
    from edlut_b200.simulation import Simulation
    net, t, c, nsteps, trace = build_case(name)
    g = load_golden(name)
    sim = Simulation.from_description(net)
    sim.inject_spikes(t, c)
    done = 0
    for n in [100, 37, 5, 64, 200, 3, 129, 1, 70]:
        sim.run(n)
        done += n
    sim.run(nsteps - done)
    st, ce = sim.spikes()
    np.testing.assert_array_equal(spike_pairs(st, ce), spike_pairs(g["spike_step"], g["spike_cell"]))
    if "w_final" in g:
        np.testing.assert_array_equal(sim.weights(), g["w_final"])
    sim.close()


@pytest.mark.parametrize("n", [9, 17, 63, 65])
def test_gpu_short_last_window_matches_fixture(n):
    """Runs whose length is no multiple of the 8-step window end in a shorter one
    (one step at 9, 17 and 65), and their flushes of deferred post-synaptic STDP fall
    between windows: repeated, the result is the reference's."""
    from edlut_b200.simulation import Simulation
    net, t, c, nsteps, trace = build_case("cereb_small_rk4")
    g = load_golden("cereb_small_rk4")
    sim = Simulation.from_description(net)
    sim.inject_spikes(t, c)
    for done in range(0, nsteps, n):
        sim.run(min(n, nsteps - done))
    st, ce = sim.spikes()
    np.testing.assert_array_equal(spike_pairs(st, ce), spike_pairs(g["spike_step"], g["spike_cell"]))
    if "w_final" in g:
        np.testing.assert_array_equal(sim.weights(), g["w_final"])
    sim.close()
