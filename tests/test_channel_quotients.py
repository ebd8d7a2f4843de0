"""The channel rates' quotients by their constants: the IEEE quotient bit for bit over the range in
which the correction is exact, and within its exponentials' reach outside."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
CONSTANTS = (10e-3, 18e-3, 20e-3, 80e-3)


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("which", range(4))
def test_quotient_by_a_constant_is_the_rounded_one(dtype, which):
    from brian2cuda_b200 import _native
    lib = _native.lib()
    t = np.dtype(dtype).type
    rng = np.random.default_rng(which)
    # the residual, 2^-24 (2^-53) of x in the same number of places, is exact from 2^-101 (2^-968) on
    lo, hi = (-30, 36) if dtype == "float32" else (-289, 36)
    x = np.concatenate([rng.uniform(-0.2, 0.2, 2_000_000), rng.uniform(-0.03, 0.03, 2_000_000),
                        10.0 ** rng.uniform(lo, hi, 1_000_000),
                        -10.0 ** rng.uniform(lo, hi, 1_000_000),
                        [0.0, -0.0, np.inf, -np.inf, np.nan]]).astype(t)
    y = np.empty_like(x)

    def run(a, b):
        return lib.b2b_div_selftest(0, _native.F32 if dtype == "float32" else _native.F64, which,
                                    a.ctypes.data_as(C.c_void_p), b.ctypes.data_as(C.c_void_p),
                                    len(a))
    assert run(x, y) == 0
    with np.errstate(over="ignore"):
        np.testing.assert_array_equal(y, x / t(CONSTANTS[which]))
    # outside: the same to two places, where an exponential of it is 1, 0 or infinite
    tiny, huge = np.finfo(t).tiny, np.finfo(t).max
    x = np.array([tiny / 8, tiny, 3 * tiny, -tiny, 7e-37, huge / 3, huge / 200, -huge], t)
    y = np.empty_like(x)
    assert run(x, y) == 0
    with np.errstate(over="ignore"):
        want = x / t(CONSTANTS[which])
    small = np.abs(want) < 1
    np.testing.assert_array_equal(np.exp(y[small]), np.exp(want[small]))
    assert np.all((np.abs(y) > 1e4) | small)
    assert run(x, y) == 0 and lib.b2b_div_selftest(0, 7, 0, None, None, 1) != 0
