"""A snapshot slot used again after the state it holds has grown (longer delays lengthen the spike
history): the second snapshot is complete, and a run from it repeats the run that followed it."""
import numpy as np
import pytest

from brian2cuda_b200 import models

pytestmark = pytest.mark.gpu
DT = 1e-4


def _state(net, P):
    return [net.get_state(P, v) for v in ("v", "ge", "gi", "lastspike", "not_refractory")]


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("n,longest", [(130, 7), (2001, 60), (2001, 300)])
def test_slot_used_again_after_the_history_has_grown(gpu_factory, dtype, n, longest):
    net = gpu_factory(DT, seed=4)
    rng = np.random.default_rng(n)
    P = net.lif_group(n, models.cuba_lif(), dtype)
    net.set_state(P, "v", rng.uniform(-60e-3, -49.9e-3, n))
    k = 20 * n
    sid = net.synapses(P, P, "ge", rng.integers(0, n, k).astype(np.int32),
                       rng.integers(0, n, k).astype(np.int32), w_scalar=1e-3,
                       delay=rng.integers(1, 4, k))
    net.finalize()
    net.run(30)
    net.store(0)
    net.syn_set_delays(sid, rng.integers(1, longest + 1, k).astype(np.int32))
    net.run(7)
    net.store(0)
    at = _state(net, P)
    net.run(50 + longest)
    after = _state(net, P)
    assert np.any(after[1] != at[1])
    net.restore(0)
    for a, b in zip(_state(net, P), at):
        np.testing.assert_array_equal(a, b)
    net.run(50 + longest)
    for a, b in zip(_state(net, P), after):
        np.testing.assert_array_equal(a, b)
