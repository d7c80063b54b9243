"""Merged splitting levels at every transform length they run (2^8 .. 2^12
points), against the digits of an independent computation: leaf sizes from two
terms (short transforms, half of a warp idle) to 64, and digit counts that leave
odd last nodes."""
import os

import pytest

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.parametrize("leaf", [2, 4, 8, 12, 16, 24, 32, 48, 64])
@pytest.mark.parametrize("digits", [7_777, 65_537, 99_991])
def test_digits_through_merged_levels(digits, leaf, monkeypatch):
    import pi_gb300 as pm
    with open(os.path.join(HERE, "golden", "pi_digits_100k.txt")) as f:
        ref = f.read().strip()
    monkeypatch.setenv("PIMUL_PI_MERGED_LEVELS", "1")
    s, _ = pm.pi_chudnovsky_batched(digits, leaf)
    assert s == ref[:digits]
