"""The read-backs of a status word and a result without a GPU: a stand-in for the CUDA runtime's calls records them."""
import subprocess
import sys
from pathlib import Path

import pytest

HERE = Path(__file__).resolve().parent
LIB = HERE.parent / "thrust_b200" / "libthrust_b200.so"

PRELUDE = """
import ctypes as C, threading
fake = C.CDLL(None)
lib = C.CDLL({lib!r})
for f in (lib.tb200_read_result, lib.tb200_read_result_in_front): f.restype = C.c_int
count = lambda name: C.c_size_t.in_dll(fake, name).value
def copies():
    n = count("fake_copies")
    where, size = (C.c_void_p * 1024).in_dll(fake, "fake_from"), (C.c_size_t * 1024).in_dll(fake, "fake_bytes")
    return sorted((where[i], size[i]) for i in range(n))
memory = (C.c_ubyte * 1024)()
base = (C.addressof(memory) + 255) // 256 * 256
scratch = base + 256
def put(at, ctype, value): ctype.from_address(at).value = value
got = C.c_int64(0)
"""


def _run(tmp_path, body):
    fake = tmp_path / "libfake_cudart.so"
    subprocess.run(["gcc", "-shared", "-fPIC", "-O1", "-o", str(fake), str(HERE / "cpp" / "fake_cudart.c")], check=True)
    code = PRELUDE.format(lib=str(LIB)) + body
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=120,
                       env={"PATH": "/usr/bin:/bin", "LD_PRELOAD": str(fake), **_library_path()})
    assert r.returncode == 0, r.stdout + r.stderr


def _library_path():
    import os
    return {k: os.environ[k] for k in ("LD_LIBRARY_PATH",) if k in os.environ}


@pytest.mark.parametrize("gap", [8, 16, 256])
def test_result_close_to_the_scratch_is_copied_by_itself(tmp_path, gap):
    """A result that lies right in front of the scratch may belong to another allocation: no copy spans both."""
    _run(tmp_path, f"""
value = scratch - {gap}
put(value, C.c_int64, 0x123456789abcdef); put(scratch, C.c_int, 3)
assert lib.tb200_read_result(C.c_void_p(scratch), C.c_void_p(value), C.c_size_t(8), C.byref(got), None) == 3
assert got.value == 0x123456789abcdef
assert copies() == [(value, 8), (scratch, 4)], copies()
""")


def test_result_in_front_of_the_scratch_takes_one_copy(tmp_path):
    _run(tmp_path, """
put(scratch - 16, C.c_int64, 77); put(scratch, C.c_int, 0)
assert lib.tb200_read_result_in_front(C.c_void_p(scratch), C.c_size_t(8), C.byref(got), None) == 0
assert got.value == 77 and copies() == [(scratch - 16, 20)], copies()
assert lib.tb200_read_result_in_front(None, C.c_size_t(8), C.byref(got), None) != 0
assert lib.tb200_read_result_in_front(C.c_void_p(scratch), C.c_size_t(17), C.byref(got), None) != 0
assert lib.tb200_read_result_in_front(C.c_void_p(scratch), C.c_size_t(8), None, None) != 0
""")


def test_short_lived_threads_share_the_pinned_page(tmp_path):
    """A pinned allocation per thread, freed when it ends, would make every short-lived thread wait for the whole GPU."""
    _run(tmp_path, """
put(scratch, C.c_int, 5)
def work():
    for _ in range(20): assert lib.tb200_temp_status(C.c_void_p(scratch), None) == 5
for _ in range(3):
    threads = [threading.Thread(target=work) for _ in range(8)]
    for t in threads: t.start()
    for t in threads: t.join()
assert count("fake_host_allocs") <= 1 and count("fake_host_frees") == 0, (count("fake_host_allocs"), count("fake_host_frees"))
lib.tb200_workspace_release_all()
assert count("fake_host_frees") == count("fake_host_allocs")
work()
""")


def test_a_failing_copy_is_reported_and_waited_for(tmp_path):
    _run(tmp_path, """
put(scratch, C.c_int, 0)
C.c_int.in_dll(fake, "fake_fail_copy").value = 1  # the second one
value = scratch - 512 + 64
assert lib.tb200_read_result(C.c_void_p(scratch), C.c_void_p(value), C.c_size_t(8), C.byref(got), None) == 1
assert count("fake_syncs") == 1  # the first may still be on its way to the landing place
assert lib.tb200_temp_status(C.c_void_p(scratch), None) == 0
""")
