"""The form of the step that a net runs untuned (one chained grid per step) survives a tuner that
fails and tunings that name the built-in rule; a tuner's choice is the same form when it is applied
to another net."""
import numpy as np
import pytest

from brian2cuda_b200 import models
from brian2cuda_b200.network import B2BError

pytestmark = pytest.mark.gpu
DT = 1e-4
STEPS = 7
ONE, TWO = STEPS + 2, 2 * STEPS + 2        # launches: the fold and the clock besides the steps'


def _net(make, n=1001, dtype="float32", delays=(1, 20)):
    net = make(DT, seed=6)
    rng = np.random.default_rng(n)
    P = net.lif_group(n, models.cuba_lif(), dtype)
    net.set_state(P, "v", rng.uniform(-60e-3, -49.9e-3, n))
    net.synapses(P, P, "ge", rng.integers(0, n, 6 * n).astype(np.int32),
                 rng.integers(0, n, 6 * n).astype(np.int32), w_scalar=1e-3,
                 delay=rng.integers(delays[0], delays[1] + 1, 6 * n))
    net.finalize()
    return net, P


def _launches(net):
    before = net.kernel_launches
    net.run(STEPS)
    return net.kernel_launches - before


def test_a_failing_tuner_leaves_the_form(gpu_factory):
    net, _ = _net(gpu_factory)
    assert _launches(net) == ONE
    net.store(1023)                        # the last slot: none is left for the tuner's own
    with pytest.raises(B2BError):
        net.autotune(trial_steps=5)
    assert _launches(net) == ONE


@pytest.mark.parametrize("dtype", ["float32", "float64"])
def test_the_built_in_pending_shape_is_the_built_in_form(gpu_factory, dtype):
    net, _ = _net(gpu_factory, dtype=dtype)
    counts = []
    for a, b in ((0, 0), (4, 296), (0, 0)):
        net.tune_apply([{"site_kind": 5, "site_index": 0, "choice_a": a, "choice_b": b}])
        counts.append(_launches(net))
    assert counts == [ONE, TWO, ONE]


def test_a_tuners_choice_is_the_form_it_names(gpu_factory):
    """4097 neurons: beyond the small-network path."""
    net, P = _net(gpu_factory, n=4097)
    chosen = net.autotune(trial_steps=30)
    form = [r for r in chosen if r["site_kind"] == 11][-1]
    other, Q = _net(gpu_factory, n=4097)
    other.tune_apply(chosen)
    assert net.run_mode == other.run_mode
    assert _launches(net) == _launches(other)
    assert form["best_ms"] <= form["default_ms"]
    net.run(60)
    other.run(60)
    for v in ("v", "ge"):
        np.testing.assert_array_equal(net.get_state(P, v), other.get_state(Q, v))
