"""tb200_read_result (status word and result by two copies) and tb200_read_result_in_front (by one)."""
import ctypes as C
import threading

import pytest
import torch

import thrust_b200 as tb
from thrust_b200 import _capi as capi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("at", [0, 8, 240, 248, 512, 1016])  # the scratch begins at 256
@pytest.mark.parametrize("status", [0, capi.ERR_WAIT_TIMEOUT])
def test_read_result(cuda_device, at, status):
    block = torch.zeros(1024, dtype=torch.uint8, device=cuda_device)
    block[256:260].view(torch.int32).fill_(status)
    block[at:at + 8].view(torch.int64).fill_(0x123456789abcdef)
    stream = C.c_void_p(torch.cuda.current_stream(cuda_device).cuda_stream)
    got = C.c_int64(0)
    base = block.data_ptr()
    rc = capi.lib.tb200_read_result(base + 256, base + at, 8, C.byref(got), stream)
    assert rc == status and got.value == 0x123456789abcdef
    assert capi.lib.tb200_temp_status(base + 256, stream) == status


def test_read_result_rejects_bad_arguments(cuda_device):
    got = C.c_int64(0)
    assert capi.lib.tb200_read_result(None, None, 0, None, None) == capi.ERR_INVALID_ARGUMENT
    assert capi.lib.tb200_read_result(256, 256, 17, C.byref(got), None) == capi.ERR_INVALID_ARGUMENT
    assert capi.lib.tb200_read_result(256, None, 8, C.byref(got), None) == capi.ERR_INVALID_ARGUMENT


@pytest.mark.parametrize("status", [0, capi.ERR_WAIT_TIMEOUT])
def test_read_result_in_front(cuda_device, status):
    block = torch.zeros(512, dtype=torch.uint8, device=cuda_device)
    block[256:260].view(torch.int32).fill_(status)
    block[240:248].view(torch.int64).fill_(0x123456789abcdef)
    got = C.c_int64(0)
    stream = C.c_void_p(torch.cuda.current_stream(cuda_device).cuda_stream)
    assert capi.lib.tb200_read_result_in_front(block.data_ptr() + 256, 8, C.byref(got), stream) == status
    assert got.value == 0x123456789abcdef


def test_results_beside_a_scratch_of_the_caller(cuda_device):
    x = torch.arange(100_003, dtype=torch.int32, device=cuda_device) // 3
    temp = torch.empty(1 << 20, dtype=torch.uint8, device=cuda_device)
    out = torch.empty(1, dtype=torch.int32, device=cuda_device)
    total = int(x.sum(dtype=torch.int64)) & 0xFFFFFFFF
    for kwargs in ({}, {"temp": temp}, {"out": out}, {"temp": temp, "out": out}):
        assert tb.reduce(x, **kwargs) & 0xFFFFFFFF == total, kwargs.keys()
    assert int(out) & 0xFFFFFFFF == total
    ones = torch.ones_like(x)
    for t in (None, temp):
        keys, sums, runs = tb.reduce_by_key(x, ones, temp=t)
        assert runs == 33335 and int(sums[:runs].sum()) == x.numel() and torch.equal(keys[:runs], torch.unique(x))
        assert tb.unique_by_key(x, temp=t)[2] == 33335
        assert tb.copy_flagged(x, (x % 2 == 0).to(torch.uint8), temp=t)[1] == int((x % 2 == 0).sum())


def test_read_backs_of_many_threads(cuda_device):
    """Each thread reads results of its own through the slots that all of them share."""
    wrong = []

    def work(i):
        stream = torch.cuda.Stream(cuda_device)
        with torch.cuda.stream(stream):
            x = torch.full((1000 + i,), i + 1, dtype=torch.int32, device=cuda_device)
            for _ in range(200):
                if tb.reduce(x) != (1000 + i) * (i + 1):
                    wrong.append(i)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(12)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
