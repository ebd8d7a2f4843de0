"""Additive delivery of a heavily driven projection by counting events per target, against one
atomic per event (the same network with a tuned delivery shape): the same state and spikes, bit for
bit."""
import numpy as np
import pytest

from brian2cuda_b200 import models

pytestmark = pytest.mark.gpu
DT = 1e-4
W = {"lif": {"ge": 1.62e-6, "gi": -9e-6, "v": 2e-7}, "hh": {"ge": 6e-12, "gi": 67e-12}}


def _net(make, kind, dtype, n_in, n_out, p, delays, targets, rate=5000.0, shared=False):
    """A part of the sources per target (groups of one population: one projection), or all of
    them for each (one projection per target)."""
    net = make(DT, seed=11)
    bounds = np.linspace(0, n_in, len(targets) + 1).astype(int)
    parts = [n_in] * len(targets) if shared else np.diff(bounds)
    S = [net.poisson_group(int(n), rate, "float32") for n in (parts[:1] if shared else parts)]
    if kind == "lif":
        P = net.lif_group(n_out, models.cuba_lif(), dtype)
        net.set_state(P, "v", np.linspace(-60e-3, -49.9e-3, n_out))
    else:
        P = net.hh_group(n_out, models.cobahh_hh(), dtype)
        models.cobahh_init(net, P, n_out, np.random.default_rng(n_out))
    rng = np.random.default_rng(n_in)
    for k, (t, n) in enumerate(zip(targets, parts)):
        if p == 1:
            i, j = np.divmod(np.arange(n * n_out), n_out)
        else:
            m = int(p * n * n_out)
            i, j = rng.integers(0, n, m), rng.integers(0, n_out, m)
        d = rng.integers(delays[0], delays[1] + 1, len(i)) if delays[1] > delays[0] else delays[0]
        net.synapses(S[0 if shared else k], P, t, i.astype(np.int32), j.astype(np.int32),
                     w_scalar=W[kind][t], delay=d)
    net.spike_monitor(P, 10**6)
    net.finalize()
    return net, P


# (bundles of about 200 in two items, 25, 7, 80, 7 with multiple synapses, 2, 10,600 in 83 items),
# tails of four targets, nearly the most targets that fit, and more than fit
SHAPES = [("lif", "float32", 9000, 2001, 0.1, (0, 0), ("ge",)),
          ("lif", "float64", 9000, 1002, 0.1, (1, 4), ("gi", "ge")),
          ("lif", "float64", 9000, 1003, 0.12, (0, 16), ("ge", "v", "gi")),
          ("hh", "float32", 1300, 100_003, 0.05, (2, 63), ("ge", "gi")),
          ("hh", "float64", 3300, 65, 3.5, (0, 31), ("ge", "gi", "ge")),
          ("lif", "float32", 30_000, 70, 1, (0, 40), ("gi", "ge", "ge", "v")),
          ("hh", "float32", 600, 105_800, 0.1, (0, 0), ("gi", "ge")),
          ("hh", "float32", 600, 107_001, 0.1, (0, 0), ("gi", "ge"))]


@pytest.mark.parametrize("shared", [False, True])
@pytest.mark.parametrize("kind,dtype,n_in,n_out,p,delays,targets", SHAPES)
def test_counted_delivery_equals_atomics(gpu_factory, kind, dtype, n_in, n_out, p, delays, targets,
                                         shared):
    if shared and len(set(targets)) < len(targets):
        targets = targets[:2]                 # one weight per variable and projection
    out = {}
    for counted in (True, False):
        net, P = _net(gpu_factory, kind, dtype, n_in, n_out, p, delays, targets, shared=shared)
        if not counted:
            net.tune_apply([{"site_kind": 6, "site_index": 0, "choice_a": 16, "choice_b": 592}])
        before = net.kernel_launches
        for steps in (1, 50, 67, 2):
            net.run(steps)
        out[counted] = (net.kernel_launches - before, net.spikes(P),
                        {v: net.get_state(P, v) for v in ("v", "ge", "gi")})
    fits = n_out < 106_000
    more = 2 * len(targets) - 1 if shared else 1      # two launches per projection and step
    assert out[True][0] - out[False][0] == (120 * more if fits else 0)
    for a, b in zip(out[True][1], out[False][1]):
        np.testing.assert_array_equal(a, b)
    for v in ("v", "ge", "gi"):
        assert np.any(out[True][2][v] != 0) or v not in targets
        np.testing.assert_array_equal(out[True][2][v], out[False][2][v], err_msg=v)


def test_in_degrees_beyond_16_bits_and_few_events_are_not_counted(gpu_factory):
    """70,000 synapses onto each of 70 targets would overflow a count, 1e5 events are too few, and
    bundles onto all targets make atomics on neighbouring addresses."""
    for n_in, rate, delays in ((70_000, 5000.0, (0, 40)), (30_000, 500.0, (0, 40)),
                               (30_000, 5000.0, (0, 0))):
        launches = []
        for tuned in (False, True):
            net, P = _net(gpu_factory, "lif", "float32", n_in, 70, 1, delays, ("ge",), rate)
            if tuned:
                net.tune_apply([{"site_kind": 6, "site_index": 0, "choice_a": 16,
                                 "choice_b": 592}])
            before = net.kernel_launches
            net.run(10)
            launches.append(net.kernel_launches - before)
        assert launches[0] == launches[1]


def test_delays_changed_under_counted_delivery(gpu_factory):
    """Bundles sent before a change arrive at their old delays (two projections, atomics), then
    counting goes on with the new ones."""
    out = {}
    for counted in (True, False):
        net, P = _net(gpu_factory, "lif", "float64", 9000, 2001, 0.1, (5, 5), ("ge",))
        shape = [{"site_kind": 6, "site_index": 0, "choice_a": 16, "choice_b": 592}]
        if not counted:
            net.tune_apply(shape)
        net.run(20)
        net.syn_set_delays(0, np.full(net.syn_count(0), 3))
        net.run(4)
        net.run(40)
        out[counted] = net.get_state(P, "ge")
    np.testing.assert_array_equal(out[True], out[False])
