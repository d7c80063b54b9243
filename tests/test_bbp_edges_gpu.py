"""BBP terms where the modular power changes its arithmetic: odd moduli around
2^28, 2^30, 2^31 and 2^32, tiny moduli, powers of two times them, and exponents
around whole groups of four bits and past 32 bits.  Against Python's integers."""
import numpy as np
import pytest

import pi_gb300 as pm

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shift", [0, 1, 2])
def test_terms_at_the_edges(shift):
    odd = [3, 5, 7, 9, 93, 255, 1023, 4095, 4097]
    for p in (12, 26, 28, 30, 31, 32):
        odd += [(1 << p) + d for d in (-7, -5, -3, -1, 1, 3, 5, 7)]
    exps = [0, 1, 2, 3, 15, 16, 17, 62, 63, 64, 1000, (1 << 22) - 17, (1 << 26) - 16, (1 << 26) - 15, (1 << 30) - 17, (1 << 30) + 1,
            (1 << 31) - 1, (1 << 31), (1 << 33) + 12345]
    d = [m << shift for m in odd if m << shift < 1 << 34]
    pairs = [(e, x) for e in exps for x in d]
    got = pm.bbp_terms([e for e, _ in pairs], [x for _, x in pairs])
    want = np.array([((pow(16, e, x) << 64) // x) & ((1 << 64) - 1) for e, x in pairs], dtype=np.uint64)
    bad = np.nonzero(got != want)[0]
    assert bad.size == 0, [(pairs[i], int(got[i]), int(want[i])) for i in bad[:4]]
