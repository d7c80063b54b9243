"""The service's HBM budget bounds what its requests really take: scratch of a
group whose products share an operand (and are then not cut into segments)
stays within the budget, and a length no transform holds is refused."""
import ctypes

import numpy as np
import pytest

import oracle as O
import pi_gb300 as pm
from conftest import rand_limbs

pytestmark = pytest.mark.gpu

USED_CURRENT, USED_HIGH = 7, 8  # CU_MEMPOOL_ATTR_USED_MEM_CURRENT, _HIGH


class _Pool:
    """Bytes in use of the device's default memory pool, which holds all scratch."""

    def __init__(self):
        self.cu = ctypes.CDLL("libcuda.so.1")
        self.pool = ctypes.c_void_p()
        assert self.cu.cuDeviceGetDefaultMemPool(ctypes.byref(self.pool), 0) == 0

    def get(self, attr):
        v = ctypes.c_uint64(0)
        assert self.cu.cuMemPoolGetAttribute(self.pool, attr, ctypes.byref(v)) == 0
        return v.value

    def reset_high(self):
        v = ctypes.c_uint64(0)
        assert self.cu.cuMemPoolSetAttribute(self.pool, USED_HIGH, ctypes.byref(v)) == 0


@pytest.mark.parametrize("la,lb", [(1 << 20, 1000), (1000, 1 << 20), (300000, 20000)])
def test_products_that_share_an_operand_stay_within_the_budget(la, lb):
    import torch
    n = 10
    N = 1 << (4 * (la + lb) - 2).bit_length()
    room = 18 * N  # scratch of one such product at full length is 17 to 17.1 N bytes
    a, b = rand_limbs(la, la), rand_limbs(lb, lb + 1)
    want = O.mul_mag(a, b)
    ha, hb = pm.upload(a), pm.upload(b)
    held = pm.service_stats()["bytes_in_use"]
    ballast = pm.upload(np.ones(room // 8, np.uint64))
    torch.cuda.synchronize()
    pool = _Pool()
    pool.reset_high()
    base = pool.get(USED_CURRENT)
    try:
        pm.set_budget(held + n * (8 * (la + lb) + 256) + room)
        # no room beside the ballast: the requests queue up behind the first ones
        reqs = [pm.submit(ha, hb) for _ in range(n)]
        pm.free(ballast)
        for _, t in reqs:
            pm.wait(t)
        got = [pm.download(h) for h, _ in reqs]
        peak = pool.get(USED_HIGH) - base
    finally:
        pm.set_budget(120 << 30)
    for h in [h for h, _ in reqs] + [ha, hb]:
        pm.free(h)
    assert all(np.array_equal(g, want) for g in got)
    assert peak <= room, (peak, room)


def test_a_length_above_2_32_is_refused():
    import torch
    x = torch.empty((1 << 30) + 1, dtype=torch.int64, device="cuda")  # 2^32 + 4 coefficients
    long, short = pm.adopt(x.data_ptr(), x.numel()), pm.adopt(x.data_ptr(), 1000)
    try:
        for p, q in ((long, short), (short, long), (long, long)):
            with pytest.raises(pm.PimulError) as e:
                pm.submit(p, q, pm.OP_MUL)
            assert e.value.code == 1
    finally:
        pm.free(long)
        pm.free(short)
