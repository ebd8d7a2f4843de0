"""Event-driven STDP with its traces kept per bundle (pre, delay) and per target neuron: every
synapse's w, Apre, Apost and lastupdate against the oracle, which keeps them per synapse."""
import numpy as np
import pytest

from brian2cuda_b200 import models
from brian2cuda_b200.network import LIF

pytestmark = pytest.mark.gpu
DT = 1e-4

# (inputs, targets, delays): work items are 128 synapses, warps 32 lanes
SHAPES = [(1, 1, "none"), (33, 127, "none"), (40, 128, "scalar"), (40, 129, "per synapse"),
          (300, 5, "per synapse"), (129, 260, "more than 64")]


def _build(net, n_in, n_out, delays):
    rng = np.random.default_rng(n_in + 7 * n_out)
    steps = 160
    when, who = np.nonzero(rng.random((steps, n_in)) < 0.03)
    inp = net.spikegen_group(n_in, who, when)
    out = net.lif_group(n_out, LIF(El=-74e-3, taum=10e-3, taue=5e-3, ke=60e-3, Vt=-54e-3,
                                   Vr=-60e-3), "float64")
    net.set_state(out, "v", rng.uniform(-60e-3, -54e-3, n_out))
    rule = models.stdp_rule(0.01)
    sids = []
    # two Synapses objects of one rule from two ranges of the inputs (one projection), dense
    # and sparse
    for lo, hi, p in ((0, n_in // 2, 1.0), (n_in // 2, n_in, 0.6)):
        i, j = np.nonzero(rng.random((hi - lo, n_out)) < p)
        if len(i) == 0:
            continue
        d = {"none": 0, "scalar": 7}.get(delays)
        if d is None:
            d = rng.integers(0, 9 if delays == "per synapse" else 90, len(i)).astype(np.int32)
        sids.append(net.synapses(inp, out, "ge", i + lo, j, w=rng.random(len(i)) * 0.2 / n_in
                                 + 0.004, delay=d, stdp=rule))
    net.spike_monitor(out, 10**6)
    net.finalize()
    return out, sids, steps


@pytest.mark.parametrize("order", [None, 0, 1])
@pytest.mark.parametrize("n_in,n_out,delays", SHAPES)
def test_traces_match_oracle(gpu_factory, oracle_factory, n_in, n_out, delays, order):
    """Float64: at most a few hundred roundings per value, 1e-10 relative leaves three digits."""
    got = {}
    for name, make in (("gpu", gpu_factory), ("orc", oracle_factory)):
        net = make(DT)
        out, sids, steps = _build(net, n_in, n_out, delays)
        if name == "gpu" and order is not None:
            net.tune_apply([{"site_kind": 8, "site_index": 0, "choice_a": order, "choice_b": 0}])
        net.run(steps)
        got[name] = (net.spikes(out), net.get_state(out, "ge"),
                     [{v: net.syn_get(s, v) for v in ("w", "Apre", "Apost", "lastupdate")}
                      for s in sids])
    np.testing.assert_array_equal(got["gpu"][0][0], got["orc"][0][0])
    np.testing.assert_array_equal(got["gpu"][0][1], got["orc"][0][1])
    np.testing.assert_allclose(got["gpu"][1], got["orc"][1], rtol=1e-10, atol=1e-18)
    for g, o in zip(got["gpu"][2], got["orc"][2]):
        for v in g:
            np.testing.assert_allclose(g[v], o[v], rtol=1e-10, atol=1e-18, err_msg=v)
    assert any(np.any(o["w"] != 0) for o in got["orc"][2])
