"""Large reads of state and synapse variables: whole chunks, a ragged last one, one value over."""
import numpy as np
import pytest

from brian2cuda_b200 import models
from brian2cuda_b200.network import LIF, STDP

pytestmark = pytest.mark.gpu
DT = 1e-4


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("n", [262_143, 262_144, 524_288, 524_289, 3_000_001])
def test_state_reads_back_as_set(gpu_factory, n, dtype):
    net = gpu_factory(DT)
    G = net.lif_group(1000, LIF(), dtype)       # the read one starts at an offset
    H = net.lif_group(n, LIF(), dtype)
    x = np.random.default_rng(n).standard_normal(n).astype(dtype)
    net.set_state(H, "v", x)
    net.finalize()
    np.testing.assert_array_equal(net.get_state(H, "v"), x)
    assert np.all(net.get_state(G, "v") == 0)
    assert len(net.get_state(H, "not_refractory")) == n


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("n_syn", [1000, 524_288, 1_000_003])
def test_synapse_variables_in_input_order(gpu_factory, n_syn, dtype):
    rng = np.random.default_rng(n_syn)
    i, j = rng.integers(0, 900, n_syn).astype(np.int32), rng.integers(0, 500, n_syn).astype(np.int32)
    d = rng.integers(0, 5, n_syn).astype(np.int32)
    w = rng.random(n_syn).astype(dtype)
    for stdp in (None, STDP(20e-3, 20e-3, 1e-4, -1e-4, 0.0, 1.0)):
        net = gpu_factory(DT)
        A = net.poisson_group(900, 10.0, "float32")
        B = net.lif_group(500, models.stdp_lif(), dtype)
        S = net.synapses(A, B, "ge", i, j, w=w, delay=d, stdp=stdp)
        net.finalize()
        for var, x in (("i", i), ("j", j), ("delay", d), ("w", w)):
            np.testing.assert_array_equal(net.syn_get(S, var), x, err_msg=var)
        if stdp is not None:
            assert not net.syn_get(S, "Apre").any() and not net.syn_get(S, "lastupdate").any()


def test_reads_of_several_threads(gpu_factory):
    """Nets of several threads read at the same time, each its own values."""
    import threading
    n, nets = 700_001, []
    for k in range(4):
        net = gpu_factory(DT)
        G = net.lif_group(n, LIF(), "float64")
        net.set_state(G, "v", np.arange(n) + 1e7 * k)
        net.finalize()
        nets.append((net, G))
    got = [None] * 4

    def read(k):
        got[k] = [nets[k][0].get_state(nets[k][1], "v") for _ in range(6)]

    threads = [threading.Thread(target=read, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for k in range(4):
        for x in got[k]:
            np.testing.assert_array_equal(x, np.arange(n) + 1e7 * k)
