"""The multicompartment solver's variants against the oracle: neurons at the edges of the
compartments-per-thread variants and beyond them (the general variant), trees with more than two
children at a node, with more than 32 nodes of one depth, with a single section or compartment,
batches of fewer and of more neurons than the GPU has SMs, and batches side by side."""
import numpy as np
import pytest

from brian2cuda_b200 import models
from brian2cuda_b200.network import HinesParams

pytestmark = pytest.mark.gpu
DT = 25e-6


def _tree(rng, n_comp, kids, sec_len):
    """Sections of sec_len compartments attached breadth-first or at random to sections with
    fewer than `kids` children."""
    starts, ends, parents, free, nc = [], [], [], [], 0
    while nc < n_comp:
        k = int(min(rng.integers(sec_len[0], sec_len[1] + 1), n_comp - nc))
        if not parents:
            parents.append(-1)
        else:
            open_secs = [s for s, f in enumerate(free) if f > 0]
            par = open_secs[0] if kids > 8 else int(rng.choice(open_secs))
            parents.append(par)
            free[par] -= 1
        free.append(kids)
        starts.append(nc)
        ends.append(nc + k)
        nc += k
    return starts, ends, parents


def _batch(neurons, seed):
    rng = np.random.default_rng(seed)
    m = {"comp_off": [0], "sec_off": [0], "sec_start": [], "sec_end": [], "sec_parent": []}
    for n_comp, kids, sec_len in neurons:
        s, e, p = _tree(rng, n_comp, kids, sec_len)
        m["comp_off"].append(m["comp_off"][-1] + n_comp)
        m["sec_off"].append(m["sec_off"][-1] + len(s))
        m["sec_start"] += s
        m["sec_end"] += e
        m["sec_parent"] += p
    m["diameter"] = rng.uniform(0.5e-6, 2e-6, m["comp_off"][-1])
    m["length"] = rng.uniform(5e-6, 50e-6, m["comp_off"][-1])
    return m, rng.uniform(0.2e-9, 1e-9, len(neurons))


def _make(kind, owner, m, current, params, f32):
    from oracle.oracle import OracleHines
    args = [m[k] for k in ("comp_off", "sec_off", "sec_start", "sec_end", "sec_parent",
                           "diameter", "length")]
    args = [np.asarray(a, np.int64 if i == 0 else (np.int32 if i < 5 else np.float64))
            for i, a in enumerate(args)]
    h = OracleHines(DT, *args, params, f32=f32) if kind == "orc" else \
        owner.hines_batch(*args, params)
    for k, v in models.hines_rest_state().items():
        h.set_state(k, v)
    h.set_current(current)
    return h


BATCHES = {
    "one compartment, one section": [(1, 2, (1, 1)), (7, 2, (7, 7)), (2, 2, (1, 1))],
    "edges of the wide variants": [(n, 2, (2, 10)) for n in (511, 512, 300)],
    "edges of the wide variants, 2": [(n, 2, (2, 10)) for n in (513, 1024, 40)],
    "general variant": [(n, 2, (2, 10)) for n in (1025, 1400, 30)],
    "many children": [(200, 5, (1, 3)), (300, 3, (2, 6)), (64, 60, (1, 1))],
    "wide levels": [(240, 80, (1, 3)), (500, 40, (1, 4)), (90, 2, (1, 1))],
    "long sections": [(700, 2, (200, 300)), (400, 2, (1, 130))],
    "more neurons than SMs": [(20 + 37 * (k % 23), 2, (2, 10)) for k in range(180)],
    "more neurons than SMs, small": [(200 + k % 57, 2 + k % 3, (1, 9)) for k in range(180)],
    "more neurons than SMs, large": [(1100 if k == 5 else 60, 2, (2, 10)) for k in range(160)],
}


@pytest.mark.parametrize("channels", ["float64", "float32"])
@pytest.mark.parametrize("name", list(BATCHES))
def test_shapes_match_oracle(gpu_factory, name, channels):
    """Float64 channels: 1e-10 relative after 120 steps, as for the configured batch; float32
    channels: the oracle's exponentials round differently, 1e-4."""
    m, current = _batch(BATCHES[name], 3)
    params = HinesParams(channel_dtype=channels)
    net = gpu_factory(DT)
    f32 = channels == "float32"
    gpu = _make("gpu", net, m, current, params, f32)
    orc = _make("orc", None, m, current, params, f32)
    for steps in (1, 119):
        gpu.run(steps)
        orc.run(steps)
    tol, floor = (1e-4, 1e-6) if f32 else (1e-10, 1e-15)
    for v in ("v", "m", "h", "n"):
        np.testing.assert_allclose(gpu.get_state(v), orc.get_state(v), rtol=tol, atol=floor,
                                   err_msg=v)
    if not f32:
        np.testing.assert_array_equal(gpu.spike_counts(), orc.spike_counts())


def test_batches_side_by_side(gpu_factory):
    """A second, smaller batch leaves the first one's launch as it was."""
    net = gpu_factory(DT)
    params = HinesParams(channel_dtype="float64")
    out = []
    for alone in (True, False):
        hs = [_make("gpu", net, *_batch([(n, 2, (2, 10))], 4), params, False)
              for n in ((1000,) if alone else (1000, 300))]
        for h in hs:
            h.run(50)
        out.append(hs[0].get_state("v"))
    np.testing.assert_array_equal(out[0], out[1])
