"""The two launches that a net takes by its size, run as one chained grid: the same spikes and state
as two launches asked for, bit for bit (one weight per variable), in one launch per step."""
import numpy as np
import pytest

from brian2cuda_b200 import models

pytestmark = pytest.mark.gpu
DT = 1e-4


def _net(make, kind, dtype, n, groups, **kw):
    net = make(DT, seed=6, **kw)
    rng = np.random.default_rng(n)
    ids = []
    for _ in range(groups):
        if kind == "lif":
            P = net.lif_group(n, models.cuba_lif(), dtype)
            net.set_state(P, "v", rng.uniform(-60e-3, -49.9e-3, n))
            we, wi = 1e-3, -7e-3
        else:
            P = net.hh_group(n, models.cobahh_hh(), dtype)
            models.cobahh_init(net, P, n, rng)
            we, wi = 6e-9, 67e-9
        for var, w in (("ge", we), ("gi", wi)):
            net.synapses(P, P, var, rng.integers(0, n, 6 * n).astype(np.int32),
                         rng.integers(0, n, 6 * n).astype(np.int32), w_scalar=w,
                         delay=rng.integers(1, 20, 6 * n))
        net.spike_monitor(P, 10**6)
        ids.append(P)
    net.finalize()
    return net, ids


@pytest.mark.parametrize("kind,dtype,n,groups,merged", [
    ("lif", "float32", 5, 1, True), ("lif", "float64", 1001, 1, True),
    ("lif", "float32", 150_000, 1, True), ("lif", "float32", 151_001, 1, False),
    ("hh", "float32", 4099, 1, True), ("hh", "float64", 8001, 1, True),
    ("hh", "float64", 33_000, 1, False), ("hh", "float32", 3000, 2, False)])
def test_merged_equals_two_launches(gpu_factory, kind, dtype, n, groups, merged):
    out = []
    for kw in ({}, {"two_launch": True}):
        net, ids = _net(gpu_factory, kind, dtype, n, groups, **kw)
        assert net.run_mode == "two-launch"
        before = net.kernel_launches
        for steps in (1, 50, 57):
            net.run(steps)
        launches = net.kernel_launches - before
        net.profile(3)                             # two launches, timed one by one
        net.store(0)
        net.run(60)
        names = ("v", "ge", "gi") + (("m", "h", "n") if kind == "hh" else ())
        out.append((launches, [x for P in ids for x in
                               (*net.spikes(P), *(net.get_state(P, v) for v in names))]))
    assert out[0][0] - out[1][0] == (-108 if merged else 0)
    for a, b in zip(out[0][1], out[1][1]):
        np.testing.assert_array_equal(a, b)


def test_a_tuned_net_runs_the_form_it_names(gpu_factory):
    net, _ = _net(gpu_factory, "lif", "float32", 1001, 1)
    counts = []
    for tune in (None, {"site_kind": 1, "choice_a": 1, "choice_b": 128},
                 {"site_kind": 1, "choice_a": 0, "choice_b": 0},
                 {"site_kind": 11, "choice_a": 1, "choice_b": 0},
                 {"site_kind": 11, "choice_a": 3, "choice_b": 0}):
        if tune:
            net.tune_apply([{"site_index": 0, **tune}])
        before = net.kernel_launches
        net.run(7)
        counts.append(net.kernel_launches - before)
    one, two = 7 + 2, 14 + 2                       # and the fold and the clock
    assert counts == [one, two, one, two, one]
