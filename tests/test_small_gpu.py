"""Short products at the edges of their forms: the one-warp products (up to 64
limbs in all), the one-CTA transforms of 2^8 .. 2^12 points and the cluster's
of 2^11 .. 2^14, alone and side by side in a batch, with squares, one-limb
operands and all-ones operands (every carry window propagates).  Against
Python's integers."""
import numpy as np
import pytest

import pi_gb300 as pm
from conftest import rand_limbs

pytestmark = pytest.mark.gpu


def _int(x):
    return int.from_bytes(np.ascontiguousarray(x).astype("<u8").tobytes(), "little")


EDGES = [2, 3, 63, 64, 65, 66, 127, 128, 129, 255, 256, 257, 511, 512, 513, 1023, 1024, 1025, 2047, 2048, 2049, 4095, 4096, 4097]


def _shapes():
    out = []
    for n in EDGES:
        out += [(n - n // 2, n // 2), (n - 1, 1), (1, n - 1), (max(1, n // 5), n - max(1, n // 5))]
    return out


def _operands(la, lb, kind):
    if kind == "ones":
        return np.full(la, (1 << 64) - 1, np.uint64), np.full(lb, (1 << 64) - 1, np.uint64)
    return rand_limbs(la, 31 * la + lb), rand_limbs(lb, 17 * la + 3 * lb)


@pytest.mark.parametrize("kind", ["random", "ones"])
def test_lone_products(kind):
    for la, lb in _shapes():
        a, b = _operands(la, lb, kind)
        assert _int(pm.mul_mag_ntt(a, b)) == _int(a) * _int(b), (la, lb)
        assert _int(pm.mul_mag_ntt(a, a)) == _int(a) ** 2, la


@pytest.mark.parametrize("kind", ["random", "ones"])
def test_side_by_side_in_a_batch(kind):
    import torch
    shapes = [s for s in _shapes() if sum(s) <= 1024] * 3
    ops = [_operands(la, lb, kind) for la, lb in shapes]

    def dev(x):
        return torch.from_numpy(x.view(np.int64)).cuda()

    jobs = []
    for i, (a, b) in enumerate(ops):
        da, db = dev(a), dev(b)
        if i % 4 == 3:  # a square
            db, ops[i] = da, (a, a)
        jobs.append((da, db, torch.full((da.numel() + db.numel(),), -1, dtype=torch.int64, device="cuda")))
    torch.cuda.synchronize()
    pm.mul_batch(jobs)
    torch.cuda.synchronize()
    for (a, b), (_, _, o) in zip(ops, jobs):
        assert _int(o.cpu().numpy().view(np.uint64)) == _int(a) * _int(b), (a.size, b.size)
