"""Sorts that fit one CTA (sorted in shared memory with one launch) against the CPU oracle — bit exact.

Sizes around every change of launch shape; keys that spread evenly over the bins, that crowd into one or two of them
(the radix way), and whose range straddles a power of two.
"""
import numpy as np
import pytest

import oracle
import thrust_b200 as tb
from util import random_keys, to_device, to_host

pytestmark = pytest.mark.gpu

SIZES = [2, 31, 33, 1023, 1024, 1025, 4607, 4608, 4609, 9215, 9216, 9217]


def _draw(rng, kind, n, dtype):
    dt = np.dtype(dtype)
    k = random_keys(rng, n, dtype)
    if kind == "constant":
        k[:] = k[0]
    elif kind == "few":  # 33 copies of a value and more: over the limit of a bin
        k = k[rng.integers(0, max(1, n // 100), size=n)]
    elif kind == "outlier":  # all but one key share a bin, and differ inside it
        u = np.dtype(f"u{dt.itemsize}")
        raw = rng.integers(0, 200, size=n).astype(u)
        raw[n // 2] = np.iinfo(u).max // 2
        k = raw.view(dtype)
    elif kind == "straddle" and dt.kind in "iu" and dt.itemsize > 2:
        top = 1 << (8 * dt.itemsize - 2)
        k = (top + rng.integers(-3000, 3000, size=n)).astype(dtype)
    return k


@pytest.mark.parametrize("kind", ["uniform", "constant", "few", "outlier", "straddle"])
@pytest.mark.parametrize("dtype", [np.uint8, np.int16, np.int32, np.float32, np.uint64, np.float64])
def test_sort_by_one_cta(cuda_device, dtype, kind):
    chk = oracle.port()
    for n in SIZES:
        rng = np.random.default_rng(7000 + n)
        k = _draw(rng, kind, n, dtype)
        desc = bool(n & 1)
        d = to_device(k)
        tb.sort(d, descending=desc)
        assert to_host(d, dtype).tobytes() == chk.sort(k, desc).tobytes(), n
        for vdtype in (np.uint8, np.uint32, np.uint64):
            v = rng.integers(0, np.iinfo(vdtype).max, size=n, dtype=vdtype)
            dk, dv = to_device(k, offset_elems=1), to_device(v)
            tb.sort_by_key(dk, dv, descending=desc)
            wk, wv = chk.sort_by_key(k, v, desc)
            assert to_host(dk, dtype).tobytes() == wk.tobytes(), (n, vdtype)
            assert to_host(dv, vdtype).tobytes() == wv.tobytes(), (n, vdtype, "values (stability)")
