"""Whole-key sorts of 4- and 8-byte keys that may take the bucket plan (one or two radix passes on the top bits, then
the buckets in shared memory) against the CPU oracle — bit exact, whichever way the device decides.

The inputs reach every decision: buckets that fit after one pass and after two, tiles of whole groups and cut tiles,
keys outside the sampled window, a bucket above the capacity, 64-bit keys whose windows are equal, crowded bins.
"""
import ctypes as C
import threading

import numpy as np
import pytest
import torch

import oracle
import thrust_b200 as tb
from thrust_b200 import _capi as capi
from util import random_keys, to_device, to_host

pytestmark = pytest.mark.gpu

SIZES = [9217, 16385, 100003, 1180003, 4200001]  # one pass, its end for evenly spread keys, two passes


def _keys(rng, kind, n, dtype):
    dt = np.dtype(dtype)
    u = np.dtype(f"u{dt.itemsize}")
    bits = 8 * dt.itemsize
    raw = random_keys(rng, n, u)
    if kind == "window":  # a common prefix above 26 bits (32-bit keys) or 50 bits
        raw = (raw >> u.type(bits - (26 if bits == 32 else 50))) | u.type(1 << (bits - 2))
    elif kind == "outlier":  # too few for the sample to see
        raw >>= u.type(4)
        raw[n // 3] = np.iinfo(u).max
        raw[n // 2] = 0
    elif kind == "heavy":  # one value 12000 times: no bucket of its own
        raw[rng.choice(n, size=min(n // 2, 12000), replace=False)] = raw[0]
    elif kind == "low":  # few distinct prefixes of 40 bits: equal windows, crowded bins
        raw = (raw >> u.type(bits - 20)) << u.type(bits - 20) | random_keys(rng, n, u, bits=6)
    elif kind == "normal":
        f = np.float32 if bits == 32 else np.float64
        raw = rng.standard_normal(n).astype(f).view(u)
    return raw.view(dtype)


@pytest.mark.parametrize("kind", ["uniform", "window", "outlier", "heavy", "low", "normal"])
@pytest.mark.parametrize("dtype", [np.int32, np.float32, np.uint64, np.float64])
def test_bucket_plan(cuda_device, dtype, kind):
    chk = oracle.port()
    for n in SIZES:
        rng = np.random.default_rng(8000 + n)
        k = _keys(rng, kind, n, dtype)
        desc = n == 100003
        v = np.arange(n, dtype=np.uint32)
        dk, dv = to_device(k, offset_elems=n % 3), to_device(v)
        tb.sort_by_key(dk, dv, descending=desc)
        wk, wv = chk.sort_by_key(k, v, desc)
        assert to_host(dk, dtype).tobytes() == wk.tobytes(), n
        assert to_host(dv, np.uint32).tobytes() == wv.tobytes(), (n, "values (stability)")
        d = to_device(k)
        tb.sort(d, descending=desc)
        assert to_host(d, dtype).tobytes() == wk.tobytes(), (n, "keys only")


@pytest.mark.parametrize("vbytes", [1, 2, 8, 16])
@pytest.mark.parametrize("dtype", [np.uint32, np.int64])
def test_bucket_plan_value_widths(cuda_device, dtype, vbytes):
    n = 1500007
    rng = np.random.default_rng(8100)
    k = random_keys(rng, n, dtype)
    v = rng.integers(0, 256, size=(n, vbytes), dtype=np.uint8)
    order = np.argsort(k, kind="stable")
    dk, dv = to_device(k), to_device(v.reshape(-1))
    need = C.c_size_t(0)
    kd = tb.tb200_dtype(dk)
    stream = C.c_void_p(torch.cuda.current_stream(cuda_device).cuda_stream)
    args = (n, kd, vbytes, 0, 0, 8 * k.itemsize, stream)
    capi.check(capi.lib.tb200_radix_sort(None, C.byref(need), None, None, *args), "size")
    temp = torch.empty(need.value, dtype=torch.uint8, device=cuda_device)
    # once with all of the scratch, once with what the byte-wise passes alone need
    for cut in (0, 1 << 19):
        have = C.c_size_t(need.value - cut)
        a, b = dk.clone(), dv.clone()
        capi.check(capi.lib.tb200_radix_sort(C.c_void_p(temp.data_ptr()), C.byref(have), C.c_void_p(a.data_ptr()),
                                             C.c_void_p(b.data_ptr()), *args), "sort")
        capi.check(capi.lib.tb200_temp_status(C.c_void_p(temp.data_ptr()), stream), "status")
        assert to_host(a, dtype).tobytes() == k[order].tobytes(), cut
        assert to_host(b, np.uint8).tobytes() == v[order].tobytes(), cut


def _copies(n, copies, dtype, device):
    g = torch.Generator(device=device)
    g.manual_seed(n + copies)
    info = torch.iinfo(dtype)
    values = torch.randint(info.min, info.max, (max(1, n // copies),), dtype=dtype, device=device, generator=g)
    return values[torch.randint(0, values.numel(), (n,), device=device, generator=g)]


@pytest.mark.parametrize("copies", [2, 5, 16, 60, 150, 400])
@pytest.mark.parametrize("dtype", [torch.int32, torch.int64])
def test_keys_with_copies(cuda_device, dtype, copies):
    for n in (3000, 9000, 700001, 5000011):
        k = _copies(n, copies, dtype, cuda_device)
        v = torch.arange(n, dtype=torch.int32, device=cuda_device)
        want, order = torch.sort(k, stable=True, descending=n == 9000)
        keys = k.clone()
        tb.sort(keys, descending=n == 9000)
        assert torch.equal(keys, want), (n, "keys only")
        tb.sort_by_key(k, v, descending=n == 9000)
        assert torch.equal(k, want), n
        assert torch.equal(v, order.to(torch.int32)), (n, "values (stability)")


@pytest.mark.parametrize("dtype", [torch.int32, torch.int64])
def test_keys_with_copies_are_not_slower_than_byte_wise(cuda_device, dtype):
    """Copies crowd the bins of the tile sort. A scratch without the plan's 512 KiB gives the byte-wise sort."""
    n = 1 << 24
    size = torch.empty(0, dtype=dtype).element_size()
    code = {4: capi.I32, 8: capi.I64}[size]
    stream = C.c_void_p(torch.cuda.current_stream(cuda_device).cuda_stream)
    args = (n, code, 4, 0, 0, 8 * size, stream)
    need = C.c_size_t(0)
    capi.check(capi.lib.tb200_radix_sort(None, C.byref(need), None, None, *args), "size")
    temp = torch.empty(need.value, dtype=torch.uint8, device=cuda_device)

    def device_time(k0, scratch):
        k, v = k0.clone(), torch.arange(n, dtype=torch.int32, device=cuda_device)
        times = []
        for _ in range(6):
            k.copy_(k0)
            begin, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            torch.cuda._sleep(200000)  # the launches are enqueued meanwhile
            begin.record()
            capi.check(capi.lib.tb200_radix_sort(C.c_void_p(temp.data_ptr()), C.byref(C.c_size_t(scratch)),
                                                 C.c_void_p(k.data_ptr()), C.c_void_p(v.data_ptr()), *args), "sort")
            end.record()
            end.synchronize()
            times.append(begin.elapsed_time(end))
        return min(times)

    for copies in (4, 16, 40, 100):
        k0 = _copies(n, copies, dtype, cuda_device)
        assert device_time(k0, need.value) < 1.15 * device_time(k0, need.value - (1 << 19)), copies


@pytest.mark.parametrize("dtype", [np.int32, np.float32, np.uint64])
def test_descending_in_two_passes(cuda_device, dtype):
    n = 4200001
    k = random_keys(np.random.default_rng(8200), n, dtype)
    v = np.arange(n, dtype=np.uint32)
    dk, dv = to_device(k), to_device(v)
    tb.sort_by_key(dk, dv, descending=True)
    wk, wv = oracle.port().sort_by_key(k, v, True)
    assert to_host(dk, dtype).tobytes() == wk.tobytes()
    assert to_host(dv, np.uint32).tobytes() == wv.tobytes()


# What the device decided, as the control block at the start of the scratch holds it: executed passes (word 2), whether
# there is a plan (word 28), window bits (34), tiles (37) and the bits in which the keys of a tile differ (38).
@pytest.mark.parametrize("kind,n,passes,tiles", [
    ("uniform", 100003, 1, None), ("uniform", 4200001, 2, "even"), ("uniform", 3200001, 2, "cut"),
    ("outlier", 4200001, None, None), ("heavy", 4200001, None, None)])
def test_plans_that_the_device_chooses(cuda_device, kind, n, passes, tiles):
    k = _keys(np.random.default_rng(8300), kind, n, np.uint64)
    d = to_device(k)
    need = C.c_size_t(0)
    stream = C.c_void_p(torch.cuda.current_stream(cuda_device).cuda_stream)
    args = (n, capi.U64, 0, 0, 0, 64, stream)
    capi.check(capi.lib.tb200_radix_sort(None, C.byref(need), None, None, *args), "size")
    temp = torch.empty(need.value, dtype=torch.uint8, device=cuda_device)
    capi.check(capi.lib.tb200_radix_sort(C.c_void_p(temp.data_ptr()), C.byref(need), C.c_void_p(d.data_ptr()), None, *args),
               "sort")
    assert to_host(d, np.uint64).tobytes() == np.sort(k).tobytes()
    word = to_host(temp[:160], np.uint32)
    assert bool(word[28]) == (passes is not None)
    if passes is not None:
        assert word[2] == passes
    if tiles == "even":  # groups of 2^g whole buckets
        assert word[38] < word[34] and word[37] & (word[37] - 1) == 0
    elif tiles == "cut":
        assert word[38] == word[34] and word[37] & (word[37] - 1) != 0


def test_sorts_of_several_threads_and_streams_at_once(cuda_device):
    """The kernels of a sort are chained with dependent launches: those of other streams run in between."""
    wrong = []

    def work(i):
        stream = torch.cuda.Stream(cuda_device)
        with torch.cuda.stream(stream):
            g = torch.Generator(device=cuda_device)
            g.manual_seed(i)
            for n in (700_001 + i, 5_000_011, 3000 + i):
                k0 = torch.randint(-2**63, 2**63 - 1, (n,), dtype=torch.int64, device=cuda_device, generator=g)
                want, order = torch.sort(k0, stable=True)
                for _ in range(4):
                    k, v = k0.clone(), torch.arange(n, dtype=torch.int32, device=cuda_device)
                    tb.sort_by_key(k, v)
                    if not (torch.equal(k, want) and torch.equal(v, order.to(torch.int32))):
                        wrong.append((i, n))

    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong


@pytest.mark.parametrize("n,planned", [(237 * 4608, True), (237 * 4608 + 1, False), ((1 << 22) - 1, False), (1 << 22, True)])
def test_plan_is_enqueued_where_there_can_be_one(cuda_device, n, planned):
    """32-bit keys above what one pass can leave and below 2^22: the host knows that there is no plan."""
    k = to_device(random_keys(np.random.default_rng(8400), n, np.uint32))
    want = np.sort(to_host(k, np.uint32))
    stream = C.c_void_p(torch.cuda.current_stream(cuda_device).cuda_stream)
    ms, kinds = (C.c_float * 32)(), (C.c_int * 32)()
    capi.check(capi.lib.tb200_trace_begin(stream), "trace")
    tb.sort(k, key_dtype=capi.U32)
    launches = capi.lib.tb200_trace_end(ms, kinds, 32)
    assert 0 < launches <= 32
    assert (14 in kinds[:launches]) == planned  # the plan's kernels
    assert to_host(k, np.uint32).tobytes() == want.tobytes()
