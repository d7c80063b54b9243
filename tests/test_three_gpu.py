"""Products whose transforms have 3 2^k points (up to three quarters of a power
of two): every such length at its edges (exactly full, one limb past it, half an
operand's rows zero or just not), squares, all-ones operands, and batches whose
products share an operand and mix both kinds of length.  Bit-exact against the
CPU oracle, and against the same product in a power of two for the longest."""
import numpy as np
import pytest

import oracle as O
import pi_gb300 as pm
from conftest import rand_limbs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [13, 14, 15, 16, 17, 18, 19, 20])
def test_lengths_at_their_edges(k):
    q = 3 << (k - 2)  # limbs of 3 2^k coefficients
    for la, lb in ((q // 2, q // 2), (q // 2 + 1, q // 2), (q // 2 + 2, q // 2 - 2), (q - q // 3, q // 3), (q // 3 * 2 + 2, 1 + q // 4)):
        a, b = rand_limbs(la, 3 * k + la), rand_limbs(lb, 5 * k + lb)
        assert np.array_equal(pm.mul_mag_ntt(a, b), O.mul_mag_ntt(a, b)), (la, lb)
    a = rand_limbs(q // 2, 7 * k)
    assert np.array_equal(pm.mul_mag_ntt(a, a), O.mul_mag_ntt(a, a))


@pytest.mark.parametrize("k", [13, 17, 18, 21, 22, 23, 24])
def test_all_ones(k):
    """(2^(64 n) - 1)^2 = 2^(128 n) - 2^(64 n + 1) + 1: the largest coefficients."""
    n = 3 << (k - 3)
    ones = np.full(n, (1 << 64) - 1, np.uint64)
    got = pm.mul_mag_ntt(ones, ones.copy())
    want = np.full(2 * n, (1 << 64) - 1, np.uint64)
    want[:n] = 0
    want[0] = 1
    want[n] = (1 << 64) - 2
    assert np.array_equal(got, want)


def test_shared_operands_and_sums():
    import torch

    def dev(x):
        return torch.from_numpy(x.view(np.int64)).cuda()

    def val(t):
        return int.from_bytes(t.cpu().numpy().view(np.uint64).astype("<u8").tobytes(), "little")

    # 3 2^17 coefficients hold 98304 limbs: all of the first group, one of the second too many
    for sizes in ([40000, 45000, 48000], [40000, 45000, 60000]):
        b = dev(rand_limbs(48000, 5))
        ops = [dev(rand_limbs(n, n)) for n in sizes]
        jobs = [(a, b, torch.full((a.numel() + b.numel(),), -1, dtype=torch.int64, device="cuda")) for a in ops]
        torch.cuda.synchronize()
        pm.mul_batch(jobs)
        torch.cuda.synchronize()
        for a, _, o in jobs:
            want = O.mul_mag(a.cpu().numpy().view(np.uint64), b.cpu().numpy().view(np.uint64))
            got = o.cpu().numpy().view(np.uint64)
            assert np.array_equal(got[: want.size], want) and not got[want.size :].any()
        # a1 b + c d in the transform domain, b shared with a product
        c, d = dev(rand_limbs(44000, 8)), dev(rand_limbs(47000, 9))
        a1, a2, e = ops[1], ops[0], torch.empty(0, dtype=torch.int64, device="cuda")
        out = torch.full((max(a1.numel() + b.numel(), c.numel() + d.numel()) + 1,), -1, dtype=torch.int64, device="cuda")
        prod = torch.full((a2.numel() + b.numel(),), -1, dtype=torch.int64, device="cuda")
        torch.cuda.synchronize()
        pm.sum_batch([(a1, b, c, d, out), (a2, b, e, e, prod)])
        torch.cuda.synchronize()
        assert val(out) == val(a1) * val(b) + val(c) * val(d)
        assert val(prod) == val(a2) * val(b)
