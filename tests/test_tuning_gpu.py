"""A tuned or applied pass count does not replace the three short passes that a
lone product of 2^17 or 2^18 points takes: two is the only count these lengths
accept, so it carries no choice."""
import ctypes

import numpy as np
import pytest

import oracle as O
import pi_gb300 as pm
from conftest import rand_limbs

pytestmark = pytest.mark.gpu


def _launches(a, b):
    """Kernel launches by class of one product a * b, and the product."""
    lib = pm.lib()
    lib.pimul_stats_get.argtypes = [ctypes.c_int, ctypes.POINTER(ctypes.c_char_p), ctypes.POINTER(ctypes.c_uint64),
                                    ctypes.POINTER(ctypes.c_uint64), ctypes.POINTER(ctypes.c_double)]
    lib.pimul_stats_reset()
    got = pm.mul_mag_ntt(a, b)
    out = {}
    for k in range(6):
        name, n, t, ms = ctypes.c_char_p(), ctypes.c_uint64(), ctypes.c_uint64(), ctypes.c_double()
        assert lib.pimul_stats_get(k, ctypes.byref(name), ctypes.byref(n), ctypes.byref(t), ctypes.byref(ms)) == 0
        out[name.value.decode()] = n.value
    return out, got


@pytest.mark.parametrize("L", [17, 18])
def test_lone_products_keep_their_split(L):
    n = 1 << (L - 3)
    a, b = rand_limbs(n, L), rand_limbs(n, L + 1)
    want = O.mul_mag(a, b)
    before, got = _launches(a, b)
    assert np.array_equal(got, want)
    try:
        pm.tuning_apply({f"np_{L}": 2})
        applied, got = _launches(a, b)
        assert applied == before and np.array_equal(got, want)
        pm.autotune(L, L, 2)
        tuned, got = _launches(a, b)
        assert tuned == before and np.array_equal(got, want)
    finally:
        pm.tuning_apply({f"np_{L}": 0})
