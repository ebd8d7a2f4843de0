"""Building blocks every step of a network goes through: the spike generator's search for its
step's entries, and the pending input's rows across chunks of any length."""
import numpy as np
import pytest

from brian2cuda_b200 import models

pytestmark = pytest.mark.gpu
DT = 1e-4


@pytest.mark.parametrize("period", [0, 40])
@pytest.mark.parametrize("entries", [0, 1, 31, 32, 33, 1023, 1025, 40_000])
def test_spike_generator_emits_its_entries(gpu_factory, entries, period):
    """The warp search probes 32 places per round: sizes around one and two rounds, steps with
    no entry and steps with many."""
    rng = np.random.default_rng(entries + period)
    # unique (neuron, step) pairs, crowded into some steps
    pairs = rng.choice(5000 * 40, size=entries, replace=False)
    who, when = pairs % 5000, (pairs // 5000) ** 2 % 40
    keep = np.unique(when * 5000 + who)
    who, when = keep % 5000, keep // 5000
    order = rng.permutation(len(who))
    net = gpu_factory(DT, steps_per_graph=7)
    G = net.spikegen_group(5000, who[order], when[order], period=period)
    net.spike_monitor(G, 10**6)
    net.finalize()
    net.run(100)
    want = [(s + p, i) for p in ((0, 40, 80) if period else (0,))
            for i, s in zip(who.tolist(), when.tolist()) if s + p < 100]
    idx, st = net.spikes(G)
    assert sorted(zip(st.tolist(), idx.tolist())) == sorted(want)


@pytest.mark.parametrize("form", [{"two_launch": True}, {"one_launch": True}])
@pytest.mark.parametrize("n", [300, 1000])
def test_pending_input_across_odd_chunks(gpu_factory, form, n):
    """Runs of odd lengths (chunks that end on either row of the pending input) give the state
    of one run, bit for bit."""
    out = []
    for runs in ((97,), (1, 7, 50, 2, 37)):
        net = gpu_factory(DT, **form)
        ids = models.build_cobahh(net, n=n, p=0.1, generated=False, monitor_capacity=10**6)
        net.finalize()
        for k in runs:
            net.run(k)
        out.append([net.get_state(ids["P"], v) for v in ("v", "m", "ge", "gi", "lastspike")])
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("form", [{"two_launch": False}, {"two_launch": True},
                                  {"one_launch": True}])
@pytest.mark.parametrize("n,dmin", [(5, 1), (33, 1), (127, 1), (1000, 1), (31_900, 1), (2000, 0)])
def test_split_hh_update_equals_one_thread_per_neuron(gpu_factory, form, n, dmin):
    """Float64 COBAHH networks below 32,000 neurons update a neuron's variables in four warps;
    the tuned shape of one thread per neuron gives the same state, bit for bit.  dmin = 0: the
    per-step form's single launch without delays."""
    if dmin == 0 and form != {"two_launch": False}:
        pytest.skip("the other forms need delays of at least one step")
    out = []
    for e in (0, 1):
        net = gpu_factory(DT, **form)
        ids = models.build_cobahh(net, n=n, p=min(1.0, 30 / n), dmin=dmin,
                                  dmax=9 if dmin else 0, dtype="float64", monitor_capacity=10**6)
        net.finalize()
        if e:
            net.tune_apply([{"site_kind": 1, "site_index": 0, "choice_a": e, "choice_b": 128}])
        net.run(120)
        out.append([net.get_state(ids["P"], v) for v in
                    ("v", "m", "h", "n", "ge", "gi", "lastspike", "not_refractory")] +
                   list(net.spikes(ids["P"])))
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)
