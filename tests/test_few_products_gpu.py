"""Few products of up to 2^11 points in a batch take a cluster each, the others of
the batch and larger numbers the persistent kernel: batches of every number
around that bound, with and without products of 2^11 and of 2^12 points, squares,
one-limb and all-ones operands, through the batch call and a replayed plan.
Against Python's integers."""
import numpy as np
import pytest

import pi_gb300 as pm
from conftest import rand_limbs

pytestmark = pytest.mark.gpu

# limbs at the edges of 2^9, 2^10, 2^11 points, and one-limb operands
SHAPES = [(33, 32), (64, 64), (65, 64), (127, 1), (128, 128), (200, 56), (129, 128), (256, 256), (511, 1), (1, 511), (300, 212), (250, 250)]


def _int(x):
    return int.from_bytes(np.ascontiguousarray(x).astype("<u8").tobytes(), "little")


def _dev(x):
    import torch
    return torch.from_numpy(x.view(np.int64)).cuda()


def _batch(shapes, ones):
    import torch
    host, jobs = [], []
    for i, (la, lb) in enumerate(shapes):
        a = np.full(la, (1 << 64) - 1, np.uint64) if ones else rand_limbs(la, 31 * la + i)
        b = np.full(lb, (1 << 64) - 1, np.uint64) if ones else rand_limbs(lb, 17 * lb + 3 * i)
        da = _dev(a)
        sq = i % 5 == 4 and la == lb
        host.append((a, a if sq else b))
        db = da if sq else _dev(b)
        jobs.append((da, db, torch.full((la + lb,), -1, dtype=torch.int64, device="cuda")))
    torch.cuda.synchronize()
    return host, jobs


def _check(host, jobs):
    import torch
    torch.cuda.synchronize()
    for (a, b), (_, _, o) in zip(host, jobs):
        assert _int(o.cpu().numpy().view(np.uint64)) == _int(a) * _int(b), (a.size, b.size)
        o.fill_(-1)
    torch.cuda.synchronize()


@pytest.mark.parametrize("ones", [False, True])
@pytest.mark.parametrize("n", [1, 2, 7, 12, 100, 255, 256, 257])
def test_batches_around_the_bound(n, ones):
    """n products of 2^9 points and more, one or more of 2^11, beside a few of one warp."""
    shapes = [SHAPES[(i * 7 + 6) % len(SHAPES)] for i in range(n)] + [(3, 5), (32, 32), (1, 1)]
    assert any(sum(s) > 256 for s in shapes)
    host, jobs = _batch(shapes, ones)
    pm.mul_batch(jobs)
    _check(host, jobs)


def test_longer_and_shorter_companions():
    for extra in ([], [(600, 300)], [(600, 300), (5000, 4000)], [(5000, 4000), (60000, 10)]):
        host, jobs = _batch(SHAPES + extra, False)
        pm.mul_batch(jobs)
        _check(host, jobs)
    host, jobs = _batch([s for s in SHAPES if sum(s) <= 256], False)
    pm.mul_batch(jobs)
    _check(host, jobs)


def test_plan_of_few_products():
    host, jobs = _batch(SHAPES + [(5000, 4000), (2, 2)], False)
    plan = pm.BatchPlan([a.size for a, _ in host], [b.size for _, b in host])
    try:
        for _ in range(3):
            plan.run(jobs)
            _check(host, jobs)
    finally:
        plan.close()
