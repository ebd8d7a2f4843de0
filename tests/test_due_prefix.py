"""Several projections with more than 64 delays in one launch: the prefix over the delays of one was
read while the next one's was written, and events went missing."""
import numpy as np
import pytest

from brian2cuda_b200 import models

pytestmark = pytest.mark.gpu
DT = 1e-4


@pytest.mark.parametrize("n,form", [(600, {"small": True}), (150_000, {"two_launch": True})])
def test_two_projections_beyond_64_delays(gpu_factory, n, form):
    """Every form against the per-step kernels (a CTA row per projection).  Sums of at most a few
    hundred roundings in float64, 1e-10 relative."""
    out = []
    for kw in (form, {"two_launch": False}):
        net = gpu_factory(DT, seed=4, **kw)
        rng = np.random.default_rng(n)
        P = net.lif_group(n, models.cuba_lif(), "float64")
        net.set_state(P, "v", rng.uniform(-60e-3, -49.9e-3, n))
        for var, w in (("gi", -0.9e-3), ("ge", 0.162e-3)):
            i, j = rng.integers(0, n, 4 * n), rng.integers(0, n, 4 * n)
            j[::4] = 7
            net.synapses(P, P, var, i.astype(np.int32), j.astype(np.int32), w_scalar=w,
                         delay=rng.integers(1, 90, 4 * n))
        net.finalize()
        g = []
        for _ in range(60):
            net.run(2)
            g.append(np.stack([net.get_state(P, v) for v in ("ge", "gi")]))
        out.append(np.stack(g))
    assert np.any(out[0] != 0)
    np.testing.assert_allclose(out[0], out[1], rtol=1e-10, atol=1e-16)
