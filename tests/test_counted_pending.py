"""Two concurrent launches per step with event counts as the pending input (large populations of
one weight per variable) against the per-step form: the same spikes and state, bit for bit."""
import numpy as np
import pytest

from brian2cuda_b200 import models

pytestmark = pytest.mark.gpu
DT = 1e-4
LIMIT = 1 << 18      # up to here the pending input is a sum of weights


def _net(make, kind, dtype, n, delays, weights, **kw):
    net = make(DT, seed=4, **kw)
    rng = np.random.default_rng(n)
    if kind == "lif":
        P = net.lif_group(n, models.cuba_lif(), dtype)
        net.set_state(P, "v", rng.uniform(-60e-3, -49.9e-3, n))
        scale = 1e-3
    else:
        P = net.hh_group(n, models.cobahh_hh(), dtype)
        models.cobahh_init(net, P, n, rng)
        scale = 4e-9
    # (target, weight); duplicates of a pair, and one target of every fourth synapse
    sids = []
    for var, w in weights:
        k = 4 * n
        i, j = rng.integers(0, n, k), rng.integers(0, n, k)
        j[::4] = 7
        sids.append(net.synapses(P, P, var, i.astype(np.int32), j.astype(np.int32),
                                 w_scalar=w * scale, delay=rng.integers(*delays, k)))
    net.spike_monitor(P, 10**7)
    net.finalize()
    return net, P, sids


def _result(net, P, kind):
    names = ("v", "ge", "gi") + (("m", "h", "n") if kind == "hh" else ())
    return (*net.spikes(P), *(net.get_state(P, v) for v in names))


@pytest.mark.parametrize("kind,dtype,n,delays,weights", [
    ("lif", "float32", LIMIT + 1, (1, 2), (("ge", 1.62), ("gi", -9.0))),
    ("lif", "float64", LIMIT + 130, (1, 30), (("ge", 1.62), ("ge", 1.62), ("gi", -9.0))),
    ("hh", "float32", LIMIT + 3, (1, 70), (("gi", 67 / 4), ("ge", 6 / 4))),
    ("hh", "float32", 290_001, (2, 9), (("ge", 6 / 4),)),
    ("hh", "float64", LIMIT + 2, (1, 9), (("ge", 6 / 4), ("gi", 67 / 4)))])
def test_counted_pending_equals_per_step(gpu_factory, kind, dtype, n, delays, weights):
    out = []
    for kw in ({}, {"two_launch": False}):
        net, P, sids = _net(gpu_factory, kind, dtype, n, delays, weights, **kw)
        assert net.run_mode == ("per-step" if kw else "two-launch")
        for steps in (1, 50, 57, 2):
            net.run(steps)
        d = np.full(net.syn_count(sids[0]), 3)
        net.syn_set_delays(sids[0], d)            # both bundles due for a while
        net.run(1)
        net.run(40)
        out.append(_result(net, P, kind))
    assert len(out[0][0]) > 1000
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)


def test_forms_of_large_populations(gpu_factory):
    """Several weights per variable cannot be counted; explicit forms stay."""
    for weights, kw, mode in (((("ge", 1.62), ("ge", 1.0)), {}, "per-step"),
                              ((("ge", 0.0),), {}, "two-launch"),
                              ((("ge", 1.62),), {"two_launch": True}, "two-launch"),
                              ((("ge", 1.62),), {}, "two-launch")):
        net, _, _ = _net(gpu_factory, "lif", "float32", LIMIT + 1, (1, 2), weights, **kw)
        assert net.run_mode == mode


@pytest.mark.parametrize("kind,dtype", [("hh", "float32"), ("lif", "float64")])
def test_counted_pending_of_several_groups(gpu_factory, kind, dtype):
    """Groups of one population (a parameter sweep), each with weights of its own."""
    out = []
    for kw in ({}, {"two_launch": False}):
        net = gpu_factory(DT, seed=4, **kw)
        rng = np.random.default_rng(3)
        groups = []
        for g, n in enumerate((1001, 150_000, 90_003, 64, 30_000)):
            if kind == "lif":
                P = net.lif_group(n, models.cuba_lif(), dtype)
                net.set_state(P, "v", rng.uniform(-60e-3, -49.9e-3, n))
                we, wi = 1e-3 * (1 + 0.3 * g), -7e-3 * (1 + 0.1 * g)
            else:
                P = net.hh_group(n, models.cobahh_hh(), dtype)
                models.cobahh_init(net, P, n, rng)
                we, wi = 4e-9 * (1 + 0.3 * g), 67e-9
            for var, w in (("ge", we), ("gi", wi)):
                net.synapses(P, P, var, rng.integers(0, n, 5 * n).astype(np.int32),
                             rng.integers(0, n, 5 * n).astype(np.int32), w_scalar=w,
                             delay=rng.integers(1, 20, 5 * n))
            net.spike_monitor(P, 10**6)
            groups.append(P)
        net.finalize()
        assert net.run_mode == ("per-step" if kw else "two-launch")
        for steps in (1, 50, 60):
            net.run(steps)
        out.append([x for P in groups for x in _result(net, P, kind)])
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)
