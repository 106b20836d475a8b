"""The radix sort of (high, low) pairs, restated on the host: radix_sort_pairs
(csrc/sort.cu) sorts the two words' bits as one number of low_bits + high_bits, so
a digit may take its low bits from one word and its high bits from the other. The
digits are those of `digits_of`, taken from a key as RadixDigit::of takes them; one
stable pass per digit, least significant first."""
from __future__ import annotations

import numpy as np
import pytest


def digits_of(low_bits, high_bits):
    """(shift, low_mask, up, high_mask) of every pass."""
    out = []
    for b in range(0, low_bits + high_bits, 8):
        if b >= low_bits:
            out.append((32 + b - low_bits, 0xFF, 0, 0))
        else:
            low = min(low_bits - b, 8)
            mask = (1 << low) - 1
            out.append((b, mask, low & 31, 0xFF & ~mask if low < 8 else 0))
    return out


def digit(keys, d):
    shift, low_mask, up, high_mask = d
    low = (keys >> np.uint64(shift)).astype(np.uint32) & np.uint32(low_mask)
    high = ((keys >> np.uint64(32)).astype(np.uint32) << np.uint32(up)) & np.uint32(high_mask)
    return low | high


@pytest.mark.parametrize("low_bits", range(0, 33))
def test_pairs_in_order(low_bits):
    for high_bits in range(0, 33):
        rng = np.random.default_rng(33 * low_bits + high_bits)
        n = 600
        low = rng.integers(0, 1 << low_bits, n, dtype=np.uint64)
        high = rng.integers(0, 1 << high_bits, n, dtype=np.uint64)
        for x, bits in ((low, low_bits), (high, high_bits)):
            x[:3] = (1 << bits) - 1
            x[3:40] >>= np.uint64(bits // 2)
        keys = high << np.uint64(32) | low
        got = keys
        digits = digits_of(low_bits, high_bits)
        assert len(digits) == -(-(low_bits + high_bits) // 8)
        for d in digits:
            v = digit(got, d)
            assert v.max() <= 0xFF
            got = got[np.argsort(v, kind="stable")]
        assert np.array_equal(got, np.sort(keys)), high_bits
