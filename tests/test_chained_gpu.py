"""Products whose operand is the product before, one call after another on a
stream with nothing between them: each call's first kernel may be scheduled
while the last one of the call before still writes its operand.  The same few
buffers are written over many rounds, so a word read too early is another
round's.  Every form of a product takes part: one warp, one CTA, one cluster,
passes of 2^k and of 3 2^k points, segments, and batches; the chains' ends are
compared with the CPU oracle's bit for bit."""
import numpy as np
import pytest

import oracle as O
import pi_gb300 as pm
from conftest import rand_limbs

pytestmark = pytest.mark.gpu

# (limbs of the chained operand, of the constant one): column sums; 2^9, 2^10 points in a CTA; 2^11 .. 2^14 in a
# cluster; 2^15, 2^17, 2^18, 2^19 points in passes; 3 2^13, 3 2^17, 3 2^18 points; 2^13-point segments
CHAINS = [(20, 20), (60, 60), (128, 128), (256, 255), (1000, 1000), (2048, 2048), (4096, 4000), (16384, 16000),
          (32768, 32000), (65536, 65000), (3000, 3100), (45000, 44000), (90000, 90000), (40000, 100), (100, 40000)]


def _chain_host(a, c, rounds):
    la = a.size
    for _ in range(rounds):
        p = np.zeros(a.size + c.size, np.uint64)
        w = O.mul_mag(a, c)
        p[: w.size] = w
        a = p[c.size // 2 : c.size // 2 + la]
    return p


@pytest.mark.parametrize("la,lc", CHAINS)
def test_each_product_feeds_the_next(la, lc):
    import torch
    rounds = 24
    a, c = rand_limbs(la, 3 * la + lc), rand_limbs(lc, 5 * la + 7 * lc)
    want = _chain_host(a, c, rounds)

    def dev(x):
        return torch.from_numpy(x.view(np.int64)).cuda()

    d0, dc = dev(a), dev(c)
    bufs = [torch.full((la + lc,), -1, dtype=torch.int64, device="cuda") for _ in range(2)]
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    for _ in range(4):  # the whole chain again, on buffers that hold its other rounds
        x = d0
        for r in range(rounds):
            out = bufs[r & 1]
            pm.mul_device(x, dc, out, stream=s.cuda_stream)
            x = out[lc // 2 : lc // 2 + la]
    torch.cuda.synchronize()
    assert np.array_equal(out.cpu().numpy().view(np.uint64), want)


def test_each_batch_feeds_the_next():
    import torch
    rounds = 12
    shapes = [s for s in CHAINS if sum(s) <= 40000]
    host = [(rand_limbs(la, 11 * la + lc), rand_limbs(lc, 13 * la + 17 * lc)) for la, lc in shapes]

    def dev(x):
        return torch.from_numpy(x.view(np.int64)).cuda()

    ops = [(dev(a), dev(c)) for a, c in host]
    bufs = [[torch.full((la + lc,), -1, dtype=torch.int64, device="cuda") for la, lc in shapes] for _ in range(2)]
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    for _ in range(3):
        xs = [a for a, _ in ops]
        for r in range(rounds):
            outs = bufs[r & 1]
            pm.mul_batch([(x, c, o) for x, (_, c), o in zip(xs, ops, outs)], stream=s.cuda_stream)
            xs = [o[lc // 2 : lc // 2 + la] for o, (la, lc) in zip(outs, shapes)]
    torch.cuda.synchronize()
    for (a, c), o in zip(host, outs):
        assert np.array_equal(o.cpu().numpy().view(np.uint64), _chain_host(a, c, rounds)), (a.size, c.size)
