"""Batched additions and subtractions at the edges of the carry kernels: one
chunk (1024 limbs), look-back over runs of chunks that pass a carry on, and the
lengths around the scanned ones, against Python's integers."""
import numpy as np
import pytest

import pi_gb300 as pm

pytestmark = pytest.mark.gpu


def _t(v, n):
    import torch
    return torch.from_numpy(np.frombuffer(v.to_bytes(8 * n, "little"), dtype="<i8").copy()).cuda()


def _val(t):
    return int.from_bytes(t.cpu().numpy().astype("<i8").tobytes(), "little")


@pytest.mark.parametrize("n", [1, 4, 5, 1023, 1024, 1025, 2048, 511 * 1024, 513 * 1024 + 3, 2048 * 1024, 2048 * 1024 + 1])
def test_carry_through_every_chunk(n):
    import torch
    ones = (1 << (64 * n)) - 1
    mid = ones - (1 << (64 * (n // 2)))  # a zero bit half way up stops the carry
    cases = [(ones, 1, 0), (mid, 1, 0), (1 << (64 * n), 1, 1), (ones, ones, 1), (ones, mid, 1)]
    jobs = [(_t(x, n + 1), _t(y, n + 1), torch.empty(n + 1, dtype=torch.int64, device="cuda"), sub) for x, y, sub in cases]
    torch.cuda.synchronize()
    pm.addsub_batch(jobs)
    torch.cuda.synchronize()
    for (x, y, sub), job in zip(cases, jobs):
        assert _val(job[2]) == (x - y if sub else x + y)
    z = torch.empty(n, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    with pytest.raises(pm.PimulError):
        pm.addsub_batch([(_t(mid, n), _t(ones, n), z, 1)])
