"""The two-round passes of the multiply at the edges of their shapes: every
transform length from the shortest pass pipeline (2^13) to three passes, with
operands that fill their transform exactly, that leave the upper half of an
operand's rows zero or one limb short of it, a one-limb operand, and a square.
Bit-exact against the CPU oracle."""
import numpy as np
import pytest

import oracle as O
import pi_gb300 as pm
from conftest import rand_limbs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L", range(13, 23))
def test_every_length_at_its_edges(L):
    q = 1 << (L - 2)  # limbs of a full transform
    for la, lb in ((q // 2, q // 2), (q // 2 + 1, q // 2 - 1), (q - 1, 1), (q // 4 + 1, q // 4)):
        a, b = rand_limbs(la, 3 * L + la), rand_limbs(lb, 5 * L + lb)
        assert np.array_equal(pm.mul_mag_ntt(a, b), O.mul_mag_ntt(a, b)), (L, la, lb)
    a = rand_limbs(q // 2, 7 * L)
    assert np.array_equal(pm.mul_mag_ntt(a, a), O.mul_mag_ntt(a, a)), L


@pytest.mark.parametrize("L,passes", [(19, 3), (22, 3), (25, 4), (31 - 5, 4)])
def test_all_ones_through_middle_passes(L, passes):
    """(2^(64 n) - 1)^2 = 2^(128 n) - 2^(64 n + 1) + 1: the largest coefficients."""
    n = 1 << (L - 3)
    assert pm.plan(n, n)[0] == 1 << L
    if pm.plan(n, n)[1] != passes:
        pm.tuning_apply({f"np_{L}": passes})
    try:
        got = pm.mul_mag_ntt(np.full(n, (1 << 64) - 1, np.uint64), np.full(n, (1 << 64) - 1, np.uint64))
    finally:
        pm.tuning_apply({f"np_{L}": 0})
    want = np.full(2 * n, (1 << 64) - 1, np.uint64)
    want[:n] = 0
    want[0] = 1
    want[n] = (1 << 64) - 2
    assert np.array_equal(got, want)
