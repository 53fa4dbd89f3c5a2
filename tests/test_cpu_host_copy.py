"""copy_to_host against a CUDA runtime of a few calls (tests/hostcopy), whose
copies happen only when they are waited for: bytes, the pinned block's life,
graphs on two devices, and which threads call CUDA."""
import ctypes as C
import subprocess

import numpy as np
import pytest

from plato_b200 import build as b

MB = 1 << 20


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = tmp_path_factory.mktemp("hostcopy") / "libhostcopy.so"
    cmd = [b.nvcc()] + b.NVCC_FLAGS + ["-shared", "--cudart", "none", "-o", str(out), str(b.CSRC / "host_copy.cu"),
                                       str(b.CSRC / "errors.cpp"), str(b.ROOT / "tests/hostcopy/fake_cudart.cpp"),
                                       "-lgomp", "-Xlinker", "-Bsymbolic"]  # these calls, whatever else is loaded
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    lib = C.CDLL(str(out))
    lib.test_copy.argtypes = [C.c_void_p, C.c_void_p, C.c_size_t, C.c_int, C.c_int]
    lib.test_user.restype = C.c_void_p
    lib.test_user_gone.argtypes = [C.c_void_p]
    return lib


def _counts(lib):
    c = (C.c_int * 5)()
    lib.test_counts(c)
    return dict(zip(("allocs", "frees", "events", "foreign", "staged"), c))


def _copy(lib, n, dev=0, fail=-1):
    src = np.random.default_rng(n).integers(0, 256, n, dtype=np.uint8)
    dst = np.zeros(n, np.uint8)
    rc = lib.test_copy(dst.ctypes.data, src.ctypes.data, n, dev, fail)
    if fail < 0:
        assert rc == 0
        np.testing.assert_array_equal(dst, src)
    return rc


def test_the_blocks_life(lib):
    user = lib.test_user()
    before = _counts(lib)
    _copy(lib, 4 * MB)  # goes the plain way: one result of a graph does not pay for the block
    assert _counts(lib) == before
    _copy(lib, MB - 1)  # small: always plain
    assert _counts(lib) == before
    for n in (MB, 4 * MB, 4 * MB + 1, 8 * MB, 9 * MB + 12345, 21 * MB + 4):
        _copy(lib, n)
    c = _counts(lib)
    assert c["allocs"] == before["allocs"] + 1 and c["staged"] > 0
    other = lib.test_user()
    lib.test_user_gone(user)
    assert _counts(lib)["frees"] == before["frees"]
    lib.test_user_gone(other)
    c = _counts(lib)
    assert c["frees"] == c["allocs"] and c["events"] == 0


def test_two_devices_share_the_block(lib):
    user = lib.test_user()
    start = _counts(lib)["allocs"]
    for k in range(12):
        _copy(lib, 5 * MB + k, dev=k & 1)
    c = _counts(lib)
    assert c["allocs"] == start + 1 and c["events"] == 64
    lib.test_user_gone(user)
    assert _counts(lib)["events"] == 0


def test_only_the_caller_calls_cuda(lib):
    user = lib.test_user()
    for _ in range(10):
        _copy(lib, 9 * MB, dev=1)
    assert _counts(lib)["foreign"] == 0
    lib.test_user_gone(user)


@pytest.mark.parametrize("fail", [0, 1, 7, 15, 16, 20, 40])
def test_a_failed_wait_is_an_error(lib, fail):
    user = lib.test_user()
    _copy(lib, 4 * MB)
    assert _copy(lib, 10 * MB, fail=fail) == (3 if fail < 40 else 0)  # PLATO_ECUDA; 10 MB have 40 chunks
    _copy(lib, 10 * MB)  # the block is usable again
    lib.test_user_gone(user)
