"""Transforms of 2^L points where no shorter form takes the product over: more
than three quarters full, and short operands whose spectrum two products share
(which are not cut into segments).  Bit-exact against the CPU oracle."""
import numpy as np
import pytest

import oracle as O
import pi_gb300 as pm
from conftest import rand_limbs

pytestmark = pytest.mark.gpu


def _dev(x):
    import torch
    return torch.from_numpy(x.view(np.int64)).cuda()


@pytest.mark.parametrize("L", range(15, 23))
def test_more_than_three_quarters_full(L):
    """One limb past three quarters, with one operand's upper half of rows zero (q/2 limbs and fewer), one limb
    short of it, and a square."""
    q = 1 << (L - 2)  # limbs of a full transform
    for la, lb in ((q // 2, q // 4 + 1), (q // 2 + 1, q // 4 + 1), (q * 5 // 8, q * 3 // 8), (q * 3 // 5, q // 3)):
        assert 4 * (la + lb) - 1 > 3 << (L - 2) and max(la, lb) < 2 * min(la, lb)
        a, b = rand_limbs(la, 3 * L + la), rand_limbs(lb, 5 * L + lb)
        assert np.array_equal(pm.mul_mag_ntt(a, b), O.mul_mag_ntt(a, b)), (L, la, lb)
    a = rand_limbs(3 * q // 8 + 1, 7 * L)
    assert np.array_equal(pm.mul_mag_ntt(a, a), O.mul_mag_ntt(a, a)), L


@pytest.mark.parametrize("L", range(14, 21))
def test_one_limb_operand_at_full_length(L):
    import torch
    q = 1 << (L - 2)
    b = rand_limbs(1, 3 * L)
    host = [rand_limbs(q - 1, L), rand_limbs(q - 2, 2 * L)]
    db = _dev(b)
    jobs = [(_dev(a), db, torch.full((a.size + 1,), -1, dtype=torch.int64, device="cuda")) for a in host]
    torch.cuda.synchronize()
    pm.mul_batch(jobs)
    torch.cuda.synchronize()
    for a, (_, _, o) in zip(host, jobs):
        want = O.mul_mag(a, b)
        got = o.cpu().numpy().view(np.uint64)
        assert np.array_equal(got[: want.size], want) and not got[want.size :].any(), (L, a.size)


@pytest.mark.parametrize("passes", [3, 4])
def test_random_product_through_two_middle_passes(passes):
    # 2^25 points, 2^7 x 2^6 x 2^6 x 2^6 with four passes; all but 32 coefficients used
    n = (1 << 22) - 4
    a, b = rand_limbs(n, 25), rand_limbs(n, 26)
    pm.tuning_apply({"np_25": passes})
    try:
        got = pm.mul_mag_ntt(a, b)
    finally:
        pm.tuning_apply({"np_25": 0})
    assert np.array_equal(got, O.mul_mag(a, b))
