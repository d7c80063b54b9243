"""Transforms of 2^L points where no shorter form takes the product over: more
than three quarters full, and short operands whose spectrum two products share
(which are not cut into segments); and the longest transforms of 3 2^k points
against the same product in a power of two.  Bit-exact against the CPU oracle
where the case says nothing else."""
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


@pytest.mark.parametrize("k", [20, 21, 22, 23, 24])
def test_three_times_a_power_of_two_against_a_power_of_two(k):
    """Alone a product of at most 3 2^k coefficients runs at 3 2^k points; beside one that shares its b and needs
    2^(k+2), at 2^(k+2)."""
    import torch
    q = 3 << (k - 2)  # limbs of 3 2^k coefficients
    g = torch.Generator(device="cuda")
    g.manual_seed(k)

    def limbs(n):
        return torch.randint(-(1 << 63), (1 << 63) - 1, (n,), generator=g, device="cuda", dtype=torch.int64)

    a, long, b = limbs(q // 2 - 1), limbs(q // 2 + 3), limbs(q // 2 - 1)
    alone = torch.full((a.numel() + b.numel(),), -1, dtype=torch.int64, device="cuda")
    beside = torch.full_like(alone, -2)
    other = torch.empty(long.numel() + b.numel(), dtype=torch.int64, device="cuda")
    pm.mul_device(a, b, alone)
    pm.mul_batch([(a, b, beside), (long, b, other)])
    torch.cuda.synchronize()
    assert torch.equal(alone, beside)
