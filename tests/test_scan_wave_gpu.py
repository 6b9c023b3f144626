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
