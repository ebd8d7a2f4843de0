"""A projection of more than 2^31 bundles (presynaptic neurons x delays) against the same synapses
from a source population of only the neurons that have any."""
import numpy as np
import pytest

from brian2cuda_b200.network import LIF, STDP

pytestmark = pytest.mark.gpu
DT = 1e-4
N_IN, DELAYS, USED, N_OUT = 240_000, 9000, 300, 64      # 2.16e9 bundles
RULE = STDP(taupre=20e-3, taupost=20e-3, dApre=0.01, dApost=-0.0105, wmin=0.0, wmax=1.0,
            pre_adds_weight=False)


def _run(make, kind, n_in, who):
    """Sources who[0..USED) of n_in; every array of the synapses is the same."""
    rng = np.random.default_rng(5)
    net = make(DT)
    src, when = np.divmod(np.arange(3 * USED), 3)
    S = net.spikegen_group(n_in, who[src], 40 * when + src % 40)
    P = net.lif_group(N_OUT, LIF(El=-49e-3, taum=20e-3, taue=5e-3, ke=0.0, Vt=-50e-3, Vr=-60e-3),
                      "float32")
    net.set_state(P, "v", np.linspace(-60e-3, -50.1e-3, N_OUT))
    k = 4000
    i, j = rng.integers(0, USED, k), rng.integers(0, N_OUT, k)
    d = rng.integers(0, DELAYS, k)
    d[:2] = 0, DELAYS - 1
    if kind == "stdp":
        sid = net.synapses(S, P, "ge", who[i], j, w=rng.random(k), delay=d, stdp=RULE)
    else:
        sid = net.synapses(S, P, "ge", who[i], j, w_scalar=0.25, delay=d)
    net.finalize()
    out = []
    for steps in (150, 4000, DELAYS):
        net.run(steps)
        names = ("w", "Apre", "Apost", "lastupdate") if kind == "stdp" else ()
        out += [net.get_state(P, v) for v in ("v", "ge")]
        out += [net.syn_get(sid, v) for v in names]
    net.close()
    return out


@pytest.mark.parametrize("kind", ["add", "stdp"])
def test_more_than_2_to_31_bundles(gpu_factory, kind):
    torch = pytest.importorskip("torch")
    if torch.cuda.mem_get_info()[0] < 60 << 30:
        pytest.skip("the bundle table alone is 17 GB")
    rng = np.random.default_rng(2)
    who = np.sort(rng.choice(N_IN, USED, replace=False))
    who[0], who[-1] = 0, N_IN - 1
    wide = _run(gpu_factory, kind, N_IN, who)
    narrow = _run(gpu_factory, kind, USED, np.arange(USED))
    assert np.ptp(wide[-1]) > 0
    for a, b in zip(wide, narrow):
        np.testing.assert_array_equal(a, b)
