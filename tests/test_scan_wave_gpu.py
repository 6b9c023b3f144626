"""Scans of inputs whose tiles are all in flight at once — one cluster, or one wave of CTAs — against the CPU oracle,
around every change of kernel: integers bit exact, floats within 1e-5 of the sum of magnitudes."""
import ctypes as C

import numpy as np
import pytest
import torch

import oracle
import thrust_b200 as tb
from thrust_b200 import _capi as capi
from util import to_device, to_host

pytestmark = pytest.mark.gpu


def _edges(bytes_per_elem, sms):
    tile = lambda vecs: 512 * vecs * (16 // bytes_per_elem)
    wave = min(2 * sms, 512)
    marks = [tile(2), tile(8), 16 * tile(2), 16 * tile(8), wave * tile(4), wave * tile(8)]
    return sorted({m + d for m in marks for d in (-1, 0, 1)})


@pytest.mark.parametrize("dtype", [np.int32, np.int64, np.float32, np.float64])
def test_scan_around_every_change_of_kernel(cuda_device, dtype):
    chk = oracle.port()
    rng = np.random.default_rng(11)
    size = np.dtype(dtype).itemsize
    for i, n in enumerate(_edges(size, torch.cuda.get_device_properties(cuda_device).multi_processor_count)):
        x = (rng.uniform(-1, 1, n) if np.dtype(dtype).kind == "f" else rng.integers(-1000, 1000, n)).astype(dtype)
        exclusive, init = bool(i & 1), [None, 7][i % 3 == 0]
        d = to_device(x, offset_elems=i % 4 == 3)
        fn = tb.exclusive_scan if exclusive else tb.inclusive_scan
        got = to_host(fn(d, d, init=init), dtype)  # in place
        if exclusive or init is None:
            want = chk.scan(x, exclusive, init)
        else:
            want = chk.scan(x, False, None) + dtype(init)
        if np.dtype(dtype).kind == "f":
            bound = 1e-5 * (np.abs(x.astype(np.float64)).sum() + abs(init or 0))
            assert np.abs(got.astype(np.float64) - want.astype(np.float64)).max() <= bound, n
        else:
            assert got.tobytes() == want.tobytes(), n


def test_scan_with_a_scratch_for_the_large_tiles_only(cuda_device):
    n = 300 * 8192 + 5
    x = torch.randint(-1000, 1000, (n,), dtype=torch.int32, device=cuda_device)
    out = torch.empty_like(x)
    tiles = -(-n // (512 * 5 * 4))  # the streaming kernel's descriptors: what every size needed at least
    have = C.c_size_t(256 + 8 * tiles)
    temp = torch.empty(have.value, dtype=torch.uint8, device=cuda_device)
    stream = C.c_void_p(torch.cuda.current_stream(cuda_device).cuda_stream)
    for exclusive in (0, 1):
        capi.check(capi.lib.tb200_scan(C.c_void_p(temp.data_ptr()), C.byref(have), C.c_void_p(x.data_ptr()),
                                       C.c_void_p(out.data_ptr()), n, capi.I32, exclusive, None, stream), "scan")
        capi.check(capi.lib.tb200_temp_status(C.c_void_p(temp.data_ptr()), stream), "status")
        want = torch.cumsum(x, 0, dtype=torch.int32)
        assert torch.equal(out, want - x if exclusive else want)


@pytest.mark.parametrize("offset,roundings", [(0, 7), (1, 9)])  # the streaming kernel; pointers that are not aligned
@pytest.mark.parametrize("exclusive", [False, True])
def test_float_prefixes_are_not_rounded_tile_by_tile(cuda_device, exclusive, offset, roundings):
    """Whole numbers below 256: the sums inside a tile are exact (below 2^24), and so are additions to a prefix that is
    carried in 64 bits. What is left is at most five roundings of the sums of up to 32 tiles that join the prefix together
    (a tree), the rounding of the prefix to a float, and that of each addition behind it: prefix + element in the streaming
    kernel, prefix + warp + lane + element in the other. Each is at most 2^-24 of a partial sum, and partial sums of
    positive numbers do not exceed the result by more than these roundings."""
    n = (1 << 27) + 5
    g = torch.Generator(device=cuda_device)
    g.manual_seed(12)
    x = torch.randint(0, 256, (n + offset,), dtype=torch.int32, device=cuda_device, generator=g)[offset:]
    f = torch.empty(n + offset, dtype=torch.float32, device=cuda_device)[offset:]
    f.copy_(x)
    out = torch.empty(n + offset, dtype=torch.float32, device=cuda_device)[offset:]
    want = torch.cumsum(x, 0, dtype=torch.int64) + 1000
    if exclusive:
        want -= x
        tb.exclusive_scan(f, out, init=1000.0)
    else:
        f[0] += 1000
        tb.inclusive_scan(f, out)
    error = ((out.double() - want.double()).abs() / want.double()).max().item()
    assert error <= roundings * 2.0**-24 * (1 + 2.0**-19)


def test_float_scan_beyond_the_largest_float(cuda_device):
    """A prefix that passes the largest float is an infinity for everything behind it, as if it were carried as a float."""
    n = 1 << 24
    x = torch.zeros(n, dtype=torch.float32, device=cuda_device)
    x[1000], x[2_000_000], x[9_000_000] = 3e38, 3e38, -3e38
    got = tb.inclusive_scan(x)
    assert got[999] == 0 and got[1000] == 3e38 and got[1_999_999] == 3e38
    assert torch.isinf(got[2_000_000:9_000_000]).all() and torch.isinf(got[-1])
    x[5] = float("nan")
    assert torch.isnan(tb.inclusive_scan(x)[5:]).all()
