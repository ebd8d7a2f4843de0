"""Bundles of the single-launch step without delays: those longer than a warp's round are shared by the
CTA, through a list that may be full, and networks of too many synapses per neuron run the update and
the delivery as two launches."""
import numpy as np
import pytest

from brian2cuda_b200 import models

pytestmark = pytest.mark.gpu
DT = 1e-4


@pytest.mark.parametrize("kind,dtype,n", [("lif", "float32", 1000), ("lif", "float64", 1000),
                                          ("lif", "float32", 151_000), ("hh", "float32", 3000),
                                          ("hh", "float64", 1000)])
def test_every_neuron_spikes_into_long_bundles(gpu_factory, kind, dtype, n):
    """All neurons reach the threshold in one step: two bundles per neuron, of up to 300 and 130
    synapses, more than a CTA's list holds.  Against every launch of its own (checked=True), bit
    for bit."""
    big = n > 100_000                      # fewer synapses per neuron: still fused
    out = []
    for checked in (False, True):
        net = gpu_factory(DT, checked=checked)
        rng = np.random.default_rng(n)
        if kind == "lif":
            P = net.lif_group(n, models.cuba_lif(), dtype)
            net.set_state(P, "v", np.full(n, -49e-3))
            we, wi = 1e-4, -2e-4
        else:
            P = net.hh_group(n, models.cobahh_hh(), dtype)
            models.cobahh_init(net, P, n, rng)
            net.set_state(P, "v", np.full(n, 25e-3))
            we, wi = 6e-10, 67e-10
        for var, w, most in (("ge", we, 300), ("gi", wi, 130)):
            some = np.arange(n) if not big else np.arange(0, n, 7)
            i = np.repeat(some, 1 + rng.integers(most // 2, most, len(some)))
            net.synapses(P, P, var, i, rng.integers(0, n, len(i)), w_scalar=w)
        net.spike_monitor(P, 10**6)
        net.finalize()
        before = net.kernel_launches
        for steps in (1, 3, 60):
            net.run(steps)
        out.append((net.kernel_launches - before, *net.spikes(P),
                    *(net.get_state(P, v) for v in ("v", "ge", "gi"))))
    assert out[0][0] < out[1][0] and len(out[1][1]) >= n
    for a, b in zip(out[0][1:], out[1][1:]):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("n,degree,fused", [(500, 495, True), (500, 505, False),
                                            (20_500, 295, True), (20_500, 305, False),
                                            (150_500, 98, True), (150_500, 102, False)])
def test_networks_of_many_synapses_per_neuron_deliver_by_a_launch(gpu_factory, n, degree, fused):
    net = gpu_factory(DT)
    rng = np.random.default_rng(1)
    P = net.lif_group(n, models.cuba_lif(), "float32")
    padded = -(-n // 128) * 128
    k = padded * degree
    net.synapses(P, P, "ge", rng.integers(0, n, k, dtype=np.int32),
                 rng.integers(0, n, k, dtype=np.int32), w_scalar=1e-5)
    net.finalize()
    before = net.kernel_launches
    net.run(5)
    assert net.kernel_launches - before == (5 + 2 if fused else 10 + 1)
