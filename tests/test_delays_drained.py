"""After a change of delays the bundles sent before it arrive through a projection of their own; once
the last has arrived the net runs the form that its delays allow again."""
import numpy as np
import pytest

from brian2cuda_b200 import models

pytestmark = pytest.mark.gpu
DT = 1e-4


def _launches(net, steps):
    before = net.kernel_launches
    net.run(steps)
    return net.kernel_launches - before


def _net(make, delay):
    n = 600
    net = make(DT, seed=6)
    rng = np.random.default_rng(n)
    P = net.lif_group(n, models.cuba_lif(), "float32")
    net.set_state(P, "v", rng.uniform(-60e-3, -49.9e-3, n))
    k = 10 * n
    sid = net.synapses(P, P, "ge", rng.integers(0, n, k), rng.integers(0, n, k), w_scalar=1e-3,
                       delay=np.full(k, delay))
    net.finalize()
    return net, P, sid, k


def test_one_launch_per_step_again_without_delays(gpu_factory):
    net, _, sid, k = _net(gpu_factory, 0)
    fused = _launches(net, 5)                  # and the last counts and the clock
    assert fused == 5 + 2
    net.syn_set_delays(sid, np.full(k, 3))
    net.run(20)
    net.syn_set_delays(sid, np.zeros(k, np.int32))
    assert _launches(net, 5) > fused           # the delayed spikes are under way
    assert _launches(net, 5) == fused


def test_one_chained_grid_again_after_long_delays(gpu_factory):
    """More than 64 delays of one projection are not for the chained grid."""
    net, _, sid, k = _net(gpu_factory, 2)
    one, two = 5 + 2, 10 + 2
    assert _launches(net, 5) == one
    net.syn_set_delays(sid, 1 + np.arange(k) % 80)
    net.run(20)
    assert _launches(net, 5) == two
    net.syn_set_delays(sid, np.full(k, 2))
    assert _launches(net, 5) == two            # the old delays are under way
    net.run(80)
    assert _launches(net, 5) == one
