"""tb200_read_result: status word and result in one copy (result in front of the scratch) or two."""
import ctypes as C

import pytest
import torch

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
