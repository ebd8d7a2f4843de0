"""The per-step form of a network without delays as one launch per step (event counts instead of
additions) against the same network with every launch site a kernel of its own (checked=True): the
same spikes and state, bit for bit."""
import numpy as np
import pytest

from brian2cuda_b200 import models

pytestmark = pytest.mark.gpu
DT = 1e-4


def _net(make, kind, n, dtype, checked, rate=False):
    net = make(DT, checked=checked, seed=3)
    rng = np.random.default_rng(n)
    if kind == "lif":
        P = net.lif_group(n, models.cuba_lif(), dtype)
        net.set_state(P, "v", rng.uniform(-60e-3, -50e-3, n))
        we, wi = 1.62e-3, -9e-3
    else:
        P = net.hh_group(n, models.cobahh_hh(), dtype)
        models.cobahh_init(net, P, n, rng)
        we, wi = 6e-9, 67e-9
    ne = int(0.8 * n)
    # several objects of one weight onto ge, one onto gi; random pairs hold duplicates
    k = 20 * n
    parts = ((0, ne // 2), (ne // 2, ne), (ne, n))
    sids = []
    for lo, hi in parts:
        i = rng.integers(lo, hi, k).astype(np.int32)
        j = rng.integers(0, n, k).astype(np.int32)
        i[: k // 8] = lo                      # one neuron with a bundle of thousands
        exc = hi <= ne
        sids.append(net.synapses(P, P, "ge" if exc else "gi", i, j, w_scalar=we if exc else wi))
    net.spike_monitor(P, 10**6)
    mon = net.rate_monitor(P, 1000) if rate else None
    net.finalize()
    return net, P, sids, mon


def _state(net, P, kind):
    return {v: net.get_state(P, v) for v in ("v", "ge", "gi", "lastspike", "not_refractory") +
            (("m", "h", "n") if kind == "hh" else ())}


@pytest.mark.parametrize("kind", ["lif", "hh"])
@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("n", [64, 129, 1000, 4097, 100_003])
def test_fused_step_equals_separate_launches(gpu_factory, kind, dtype, n):
    out = {}
    for checked in (False, True):
        net, P, _, mon = _net(gpu_factory, kind, n, dtype, checked, rate=n == 1000)
        launches = net.kernel_launches
        for steps in (1, 50, 57, 2):          # whole chunks and odd ones
            net.run(steps)
        out[checked] = (net.spikes(P), _state(net, P, kind), net.kernel_launches - launches,
                        net.rate_counts(mon) if mon is not None else ())
        assert net.run_mode == "per-step"
    assert len(out[True][0][0]) > 0
    assert out[False][2] < out[True][2]       # the fused form is the one that ran
    for a, b in zip(out[False][0], out[True][0]):
        np.testing.assert_array_equal(a, b)
    for v in out[True][1]:
        np.testing.assert_array_equal(out[False][1][v], out[True][1][v], err_msg=v)
    for a, b in zip(out[False][3], out[True][3]):
        np.testing.assert_array_equal(a, b)


def test_fused_step_around_profiles_snapshots_and_delays(gpu_factory):
    """Profiling (separate launches), a snapshot, a tuned delivery shape (separate launches) and a
    change of delays between runs leave the same network."""
    out = {}
    for checked in (False, True):
        net, P, sids, _ = _net(gpu_factory, "lif", 1000, "float64", checked)
        net.run(30)
        net.store(0)
        net.profile(11)
        net.run(53)
        a = _state(net, P, "lif")
        net.restore(0)
        net.run(64)
        b = _state(net, P, "lif")
        net.tune_apply([{"site_kind": 6, "site_index": 0, "choice_a": 8, "choice_b": 0}])
        net.run(20)
        net.tune_apply([{"site_kind": 6, "site_index": 0, "choice_a": 0, "choice_b": 0}])
        net.run(20)
        net.syn_set_delays(sids[0], np.arange(net.syn_count(sids[0]), dtype=np.int32) % 4)
        net.run(40)
        net.syn_set_delays(sids[0], np.zeros(net.syn_count(sids[0]), np.int32))
        net.run(60)
        out[checked] = (a, b, _state(net, P, "lif"), net.spikes(P))
    for k in range(3):
        for v in out[True][k]:
            np.testing.assert_array_equal(out[False][k][v], out[True][k][v], err_msg=v)
    for v in out[True][0]:
        np.testing.assert_array_equal(out[True][0][v], out[True][1][v], err_msg=v)
    np.testing.assert_array_equal(out[False][3][0], out[True][3][0])


def test_fused_step_with_many_synapses_objects(gpu_factory):
    """More members than the launch's parameters hold, and two projections (overlapping source
    ranges do not merge)."""
    out = {}
    for checked in (False, True):
        net = gpu_factory(DT, checked=checked)
        rng = np.random.default_rng(8)
        n = 900
        P = net.lif_group(n, models.cuba_lif(), "float64")
        net.set_state(P, "v", rng.uniform(-60e-3, -50e-3, n))
        for lo in range(0, n, 150):            # six objects of one projection
            i, j = rng.integers(lo, lo + 150, 4000), rng.integers(0, n, 4000)
            exc = lo < 600
            net.synapses(P, P, "ge" if exc else "gi", i, j, w_scalar=1.62e-3 if exc else -9e-3)
        net.synapses(P, P, "ge", rng.integers(0, n, 9000), rng.integers(0, n, 9000),
                     w_scalar=1.62e-3)         # from every neuron: a projection of its own
        net.spike_monitor(P, 10**5)
        net.finalize()
        net.run(120)
        out[checked] = (net.spikes(P), _state(net, P, "lif"))
    assert len(out[True][0][0]) > 0
    np.testing.assert_array_equal(out[False][0][0], out[True][0][0])
    for v in out[True][1]:
        np.testing.assert_array_equal(out[False][1][v], out[True][1][v], err_msg=v)
