"""CPU tests of the sweep workload generator and of the delay ring's size (no GPU)."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from edlut_b200.configs import LIF_C1, sweep_networks


def test_sweep_specs_are_seeded_and_in_range():
    a = sweep_networks(seed=3, n_networks=64, t_end=0.1)
    b = sweep_networks(seed=3, n_networks=64, t_end=0.1)
    sizes = np.array([s["n"] for s in a])
    assert sizes.min() >= 500 and sizes.max() <= 5000
    for x, y in zip(a, b):
        assert x["n"] == y["n"] and x["params"] == y["params"]
        np.testing.assert_array_equal(x["times"], y["times"])
        np.testing.assert_array_equal(x["cells"], y["cells"])
    gl = np.array([s["params"]["g_leak"] for s in a]) / LIF_C1["g_leak"]
    assert gl.min() >= 0.7 - 1e-6 and gl.max() <= 1.3 + 1e-6
    el = np.array([s["params"]["e_leak"] for s in a])
    assert (el < LIF_C1["v_thr"]).all()  # every network stays below threshold at rest
    # per-network Poisson seeds: input trains differ between networks
    assert not np.array_equal(a[0]["times"], a[1]["times"])
    for s in a:
        assert (np.diff(s["times"]) >= 0).all()
        assert s["cells"].min() >= 0 and s["cells"].max() < s["n_in"]


def test_sweep_weight_scaling_keeps_mean_drive():
    a = sweep_networks(seed=4, n_networks=32, t_end=0.05)
    for s in a:
        # recurrent range x size / 1000 is the weight-scale factor, the same as the input range's
        k = s["w_exc_max"] * s["n"] / 1000.0 / 0.5
        assert abs(k - s["w_in_max"] / 0.5) < 1e-4 * max(1.0, k)


# The rows of a network's ring that are in use at once must have slots of their own: while
# one CTA still drains window w (or lists the sources of window w + 1), the others already
# write window w + 1.
RING_PROGRAM = r"""
#include <cstdio>
#include <set>
#include "eb_sweep.h"
int main() {
    long bad = 0;
    auto check = [&](int64_t most, int64_t fewest, bool arrives) {
        const ebsw::SweepRing r = ebsw::sweep_ring(most, fewest);
        bad += r.window < 1 || r.window > ebsw::kSweepWindow || r.window > fewest;
        const int64_t kw = 1000;  // first step of window w
        std::set<int64_t> rows;
        for (int64_t k = kw; k < kw + 2 * r.window; ++k) rows.insert(k);  // drained, written
        if (arrives)  // sources of window w + 1's lists
            for (int64_t k = kw + r.window; k < kw + 2 * r.window; ++k)
                for (int64_t j = k - most; j <= k - fewest; ++j) rows.insert(j);
        std::set<int64_t> slots;
        for (int64_t k : rows) slots.insert(k % r.slots);
        bad += slots.size() != rows.size();
    };
    for (int64_t fewest = 1; fewest <= 40; ++fewest)
        for (int64_t most = fewest; most <= fewest + 3; ++most) check(most, fewest, true);
    check(1, INT32_MAX, false);  // no spike arrives within the run
    printf("%ld\n", bad);
}
"""


@pytest.mark.skipif(not shutil.which("g++"), reason="needs g++")
def test_ring_keeps_a_window_apart_from_the_one_being_drained(tmp_path):
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    src = tmp_path / "ring.cpp"
    src.write_text(RING_PROGRAM)
    exe = str(tmp_path / "ring")
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    if not os.path.exists(os.path.join(cuda, "include", "cuda_runtime.h")):
        pytest.skip("needs the CUDA headers")
    subprocess.run(["g++", "-std=c++17", "-O1", "-w", "-I" + os.path.join(root, "edlut_b200", "csrc"),
                    "-I" + os.path.join(root, "include"), "-I" + os.path.join(cuda, "include"), str(src), "-o", exe,
                    "-L" + os.path.join(cuda, "lib64"), "-lcudart"], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, check=True).stdout
    assert int(out) == 0
