"""Products of a long by a short operand, which the engine cuts into segments:
lengths around whole numbers of segments, one-limb and nearly half-length
short operands, both operand orders, all-ones operands (carries through every
window and segment boundary), single calls, batches and batch plans.
Bit-exact against the CPU oracle."""
import numpy as np
import pytest

import oracle as O
import pi_gb300 as pm
from conftest import rand_limbs

pytestmark = pytest.mark.gpu


def _shapes():
    out = [(4096, 1), (100003, 1), (40000, 3), (65536, 8192), (60000, 20000), (30000, 14999), (30000, 15000), (262144, 5001)]
    # k segments of 2^13 points for a 100-limb operand hold k (2^13 - 400) coefficients
    for k in (3, 5, 16):
        n = k * (8192 - 400) // 4 - 100
        out += [(n - 1, 100), (n, 100), (n + 1, 100)]
    return out


@pytest.mark.parametrize("la,lb", _shapes())
def test_uneven_products(la, lb):
    a, b = rand_limbs(la, 3 * la + lb), rand_limbs(lb, 5 * la + 7 * lb)
    want = O.mul_mag(a, b)
    assert np.array_equal(pm.mul_mag_ntt(a, b), want)
    assert np.array_equal(pm.mul_mag_ntt(b, a), want)


@pytest.mark.parametrize("la,lb", [(50000, 1), (50000, 777), (200000, 4096)])
def test_carries_cross_segments(la, lb):
    """(2^(64 la) - 1) (2^(64 lb) - 1) and (2^(64 la) - 1) times one: all-ones windows throughout."""
    a, b = np.full(la, (1 << 64) - 1, np.uint64), np.full(lb, (1 << 64) - 1, np.uint64)
    got = pm.mul_mag_ntt(a, b)
    ia, ib = (1 << (64 * la)) - 1, (1 << (64 * lb)) - 1
    assert int.from_bytes(got.astype("<u8").tobytes(), "little") == ia * ib
    one = np.zeros(lb, np.uint64)
    one[0] = 1
    assert np.array_equal(pm.mul_mag_ntt(a, one)[:la], a)


def test_batches_and_plans_of_uneven_products():
    import torch
    sizes = [(70000, 300), (300, 70000), (5000, 5000), (20000, 2), (70000, 300), (9000, 4000), (700, 600), (150000, 30000)]
    host = [(rand_limbs(la, 11 * i + 1), rand_limbs(lb, 11 * i + 2)) for i, (la, lb) in enumerate(sizes)]
    host.append((host[0][0], host[4][1]))

    def dev(x):
        return torch.from_numpy(x.view(np.int64)).cuda()

    da = {id(x): dev(x) for ab in host for x in ab}
    jobs = [(da[id(a)], da[id(b)], torch.full((a.size + b.size,), -1, dtype=torch.int64, device="cuda")) for a, b in host]
    want = [O.mul_mag(a, b) for a, b in host]

    def check():
        torch.cuda.synchronize()
        for (_, _, o), w in zip(jobs, want):
            got = o.cpu().numpy().view(np.uint64)
            assert np.array_equal(got[: w.size], w) and not got[w.size :].any()
            o.fill_(-1)
        torch.cuda.synchronize()

    torch.cuda.synchronize()
    pm.mul_batch(jobs)
    check()
    plan = pm.BatchPlan([a.size for a, _ in host], [b.size for _, b in host])
    try:
        for _ in range(2):
            plan.run(jobs)
            check()
    finally:
        plan.close()
