"""The shared-memory sort in each of its launch shapes (tests/cpp/test_tile_sort.cu), the two largest of which sorts
reach at 280 and 570 million elements only; and sorts of these sizes through the library."""
import subprocess
from pathlib import Path

import pytest
import torch

import thrust_b200 as tb

EXE = Path(__file__).resolve().parent / "cpp" / "bin" / "test_tile_sort"


def _run(what):
    assert EXE.exists(), "tests/cpp/bin/test_tile_sort missing: run __graft_entry__.build()"
    r = subprocess.run([str(EXE), what], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "PASSED" in r.stdout, r.stdout[-2000:] + r.stderr[-2000:]


def test_padding_places():
    _run("places")


@pytest.mark.gpu
def test_tiles_of_every_shape(cuda_device):
    _run("sort")


@pytest.mark.gpu
@pytest.mark.parametrize("descending", [False, True])
@pytest.mark.parametrize("n", [290_000_003, 580_000_001])  # 1024 x 9 and 1024 x 17
def test_large_sorts_with_small_buckets(cuda_device, n, descending):
    g = torch.Generator(device=cuda_device)
    g.manual_seed(n)
    # a range that is no power of two and does not begin at zero: its first and last buckets are partly filled; and
    # thinly spread keys below it, a few hundred to a few thousand to a bucket
    low = 0x10012345
    k = torch.randint(low, 0x7a000000, (n,), dtype=torch.int32, device=cuda_device, generator=g)
    k[: n // 500] = torch.randint(0, low, (n // 500,), dtype=torch.int32, device=cuda_device, generator=g)
    v = torch.arange(n, dtype=torch.int32, device=cuda_device)
    want, order = torch.sort(k, stable=True, descending=descending)
    tb.sort_by_key(k, v, descending=descending)
    assert torch.equal(k, want)
    assert torch.equal(v, order.to(torch.int32))
