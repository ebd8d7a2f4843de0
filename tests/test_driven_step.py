"""Two populations of a step updated in one launch and a step's kernels launched chained, against
the same network with every launch on its own (checked=True)."""
import numpy as np
import pytest

from brian2cuda_b200 import models

pytestmark = pytest.mark.gpu
DT = 1e-4


def _net(make, source, kind, n_in, n_out, dtype, checked, swapped, stdp):
    net = make(DT, checked=checked, seed=5)
    rng = np.random.default_rng(n_in + n_out)

    def add_source():
        if source == "poisson":
            return net.poisson_group(n_in, 300.0, dtype if n_in % 2 else "float32")
        when, who = np.nonzero(rng.random((200, n_in)) < 0.03)
        return net.spikegen_group(n_in, who, when)

    def add_target():
        if kind == "lif":
            g = net.lif_group(n_out, models.cuba_lif(), dtype)
            net.set_state(g, "v", rng.uniform(-60e-3, -50e-3, n_out))
            return g
        g = net.hh_group(n_out, models.cobahh_hh(), dtype)
        models.cobahh_init(net, g, n_out, rng)
        return g

    if swapped:
        T, S = add_target(), add_source()
    else:
        S, T = add_source(), add_target()
    k = 8 * n_out
    weight = {"lif": {"ge": 1.62e-3, "gi": -9e-3, "v": 2e-4}, "hh": {"ge": 6e-9, "gi": 67e-9}}
    # one weight per variable: the order of the additions does not matter; the membrane as a
    # target defers the reset to after the deliveries
    for pre, n_pre, var, delay in ((S, n_in, "ge", 0), (T, n_out, "gi", 3), (S, n_in, "v", 2)):
        if var in weight[kind]:
            net.synapses(pre, T, var, rng.integers(0, n_pre, k).astype(np.int32),
                         rng.integers(0, n_out, k).astype(np.int32),
                         w_scalar=weight[kind][var], delay=delay)
    sid = None
    if stdp:
        i, j = np.nonzero(rng.random((n_in, n_out)) < 0.3)
        sid = net.synapses(S, T, "ge", i, j, w=rng.random(len(i)) * 1e-4,
                           stdp=models.stdp_rule(1e-4))
    net.spike_monitor(S, 10**6)
    net.spike_monitor(T, 10**6)
    rate = net.rate_monitor(T, 1000)
    # (a state monitor's launch stands between two steps)
    trace = (net.state_monitor(T, "v", indices=[0, n_out - 1], every=3, capacity=1000)
             if n_in % 2 else None)
    net.finalize()
    return net, S, T, sid, rate, trace


@pytest.mark.parametrize("source", ["poisson", "spikegen"])
@pytest.mark.parametrize("kind,dtype,n_in,n_out,stdp", [
    ("lif", "float32", 1, 5, False), ("lif", "float64", 255, 257, False),
    ("lif", "float32", 300, 60_001, False), ("lif", "float64", 512, 128, False),
    ("hh", "float32", 256, 131, False), ("hh", "float64", 129, 260, False),
    ("hh", "float64", 64, 40_003, False), ("hh", "float32", 257, 70_002, False),
    ("lif", "float64", 255, 257, True), ("lif", "float64", 512, 128, True)])
def test_driven_step_equals_separate_launches(gpu_factory, source, kind, dtype, n_in, n_out, stdp):
    """Bit for bit without STDP.  With it, weights differ per synapse and are added in any order:
    200 steps of sums of at most a few hundred terms, 1e-10 relative in float64."""
    out = {}
    for checked in (False, True):
        net, S, T, sid, rate, trace = _net(gpu_factory, source, kind, n_in, n_out, dtype, checked,
                                           swapped=n_in % 2 == 0, stdp=stdp)
        launches = net.kernel_launches
        for steps in (1, 50, 57, 92):         # whole chunks and odd ones
            net.run(steps)
        out[checked] = dict(
            launches=net.kernel_launches - launches, src=net.spikes(S), spk=net.spikes(T),
            state={v: net.get_state(T, v) for v in ("v", "ge", "gi")}, rate=net.rate_counts(rate),
            trace=() if trace is None else net.state_values(trace),
            syn={} if sid is None else {v: net.syn_get(sid, v) for v in ("w", "Apre", "Apost")})
        assert net.run_mode == "per-step"
    a, b = out[False], out[True]
    assert a["launches"] < b["launches"]      # one launch for the two updates
    assert len(a["src"][0]) > 0 or source == "spikegen"
    for x, y in zip(a["src"], b["src"]):
        np.testing.assert_array_equal(x, y)
    if not stdp:
        pairs = [*zip(a["spk"], b["spk"]), *zip(a["rate"], b["rate"]),
                 *zip(a["trace"], b["trace"]), *((a["state"][v], b["state"][v]) for v in b["state"])]
        for x, y in pairs:
            np.testing.assert_array_equal(x, y)
        return
    for x, y in zip(a["spk"], b["spk"]):
        np.testing.assert_array_equal(x, y)
    for v in b["syn"]:
        np.testing.assert_allclose(a["syn"][v], b["syn"][v], rtol=1e-10, atol=1e-18)
