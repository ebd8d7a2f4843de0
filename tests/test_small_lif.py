"""The one-CTA form of small LIF networks without delays (state in registers, one launch for many
chunks) against the same network with every launch site a kernel of its own: the same spikes and
state, bit for bit."""
import numpy as np
import pytest

from brian2cuda_b200 import models
from brian2cuda_b200.network import LIF

pytestmark = pytest.mark.gpu
DT = 1e-4
VARS = ("v", "ge", "gi", "lastspike", "not_refractory")


def _run(make, n, dtype, indegree, small, inputs=False, groups=1):
    net = make(DT, small=small, checked=not small)
    rng = np.random.default_rng(n + indegree)
    gs = []
    for k in range(groups):
        p = LIF(El=-49e-3 - 1e-3 * k, taum=20e-3, taue=5e-3, taui=10e-3, ke=1.0, ki=1.0, Vt=-50e-3,
                Vr=-60e-3, refractory=0.0 if k == 1 else 5e-3, unless_refractory=k != 1)
        g = net.lif_group(n, p, dtype)
        net.set_state(g, "v", rng.uniform(-60e-3, -50e-3, n))
        gs.append(g)
    if inputs:
        net.timed_array(gs[0], rng.uniform(0, 4e-3, 40), 2e-3)
    for a in gs:
        for b in gs:
            i, j = models.bernoulli_pairs(rng, n, n, min(1.0, indegree / n))
            exc = i < int(0.8 * n)
            net.synapses(a, b, "ge", i[exc], j[exc], w_scalar=1.62e-3)
            net.synapses(a, b, "gi", i[~exc], j[~exc], w_scalar=-9e-3)
    for g in gs:
        net.spike_monitor(g, 10**6)
    net.finalize()
    for steps in (1, 2, 50, 247, 1100):
        net.run(steps)
    assert net.run_mode == ("small" if small else "per-step")
    assert net.sync() == 0
    return [net.spikes(g) + tuple(net.get_state(g, v) for v in VARS) for g in gs], net.timestep


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("n,indegree", [(1, 1), (127, 40), (128, 128), (700, 80), (1024, 80),
                                        (1025, 80), (1000, 400), (2048, 30), (2049, 60),
                                        (4096, 20)])
def test_equals_separate_launches(gpu_factory, n, indegree, dtype):
    """One, two and four neurons per thread; connectivity in shared memory and (1000 x 400, 2049 x
    60 and above) in L2; no spike, and spikes in nearly every step."""
    a, ta = _run(gpu_factory, n, dtype, indegree, True)
    b, tb = _run(gpu_factory, n, dtype, indegree, False)
    assert ta == tb == 1400
    for x, y in zip(a[0], b[0]):
        np.testing.assert_array_equal(x, y)


@pytest.mark.parametrize("groups,inputs", [(1, True), (3, False)])
def test_groups_and_inputs(gpu_factory, groups, inputs):
    a, _ = _run(gpu_factory, 300, "float64", 60, True, inputs, groups)
    b, _ = _run(gpu_factory, 300, "float64", 60, False, inputs, groups)
    assert sum(len(x[0]) for x in b) > 0
    for x, y in zip(a, b):
        for p, q in zip(x, y):
            np.testing.assert_array_equal(p, q)
