"""Lone products of 2^13 and 2^14 points: one launch of a sixteen-CTA cluster
where the GPU can place it, the passes where it cannot (forced here by the
environment variable that says so, in a process of its own).  Bit-exact against
the CPU oracle through every entry point that takes a lone product."""
import os
import subprocess
import sys

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

CHILD = r"""
import ctypes, sys
import numpy as np
import torch
sys.path[:0] = [sys.argv[2], sys.argv[2] + "/tests"]
import oracle as O
import pi_gb300 as pm
from conftest import rand_limbs

cluster = sys.argv[1] == "1"
lib = pm.lib()
lib.pimul_stats_get.argtypes = [ctypes.c_int, ctypes.POINTER(ctypes.c_char_p), ctypes.POINTER(ctypes.c_uint64),
                                ctypes.c_void_p, ctypes.c_void_p]
noalloc = lib.pimul_mul_device_noalloc
noalloc.argtypes = [ctypes.c_void_p, ctypes.c_size_t] * 2 + [ctypes.c_void_p] * 2

def launches():
    out = {}
    for k in range(6):
        name, n = ctypes.c_char_p(), ctypes.c_uint64()
        assert lib.pimul_stats_get(k, ctypes.byref(name), ctypes.byref(n), None, None) == 0
        out[name.value.decode()] = n.value
    return out

def check(t, want):
    got = t.cpu().numpy().view(np.uint64)
    assert np.array_equal(got[: want.size], want) and not got[want.size :].any()

for la, lb in ((512, 513), (700, 701), (1024, 1024), (2047, 1), (1025, 1024), (2000, 2000), (2048, 2048), (4000, 96)):
    a, b = rand_limbs(la, la + lb), rand_limbs(lb, 3 * la + lb)
    want, sq = O.mul_mag(a, b), O.mul_mag(a, a)
    lib.pimul_stats_reset()
    assert np.array_equal(pm.mul_mag_ntt(a, b), want)
    n = launches()
    assert (n["small"], n["carry"]) == ((1, 0) if cluster else (0, 1)), (la, lb, n)
    assert np.array_equal(pm.mul_mag_ntt(a, a), sq)
    da, db = (torch.from_numpy(x.view(np.int64)).cuda() for x in (a, b))
    out = torch.full((la + lb,), -1, dtype=torch.int64, device="cuda")
    pm.mul_device(da, db, out)
    torch.cuda.synchronize()
    check(out, want)
    out.fill_(-1)
    torch.cuda.synchronize()
    assert noalloc(da.data_ptr(), la, db.data_ptr(), lb, out.data_ptr(), None) == 0
    torch.cuda.synchronize()
    check(out, want)
print("done")
"""


@pytest.mark.parametrize("cluster", [True, False])
def test_both_forms(cluster):
    env = dict(os.environ)
    env.pop("PIMUL_WIDE_CLUSTERS", None)
    if not cluster:
        env["PIMUL_WIDE_CLUSTERS"] = "0"
    r = subprocess.run([sys.executable, "-c", CHILD, "1" if cluster else "0", ROOT], capture_output=True, text=True, env=env,
                       timeout=300)
    assert r.returncode == 0 and r.stdout.strip().endswith("done"), r.stderr[-2000:]
