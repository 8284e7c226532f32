"""Arrays on their way out of the device: every size class, and indices widened on the way."""
import ctypes as C

import numpy as np
import pytest

from genn_b200 import abi

CHUNK = 512 * 1024


@pytest.fixture(scope="module")
def runner():
    lib = abi.load_library()
    handle = C.c_void_p()
    abi.check(lib.b200_runner_create(0, 1.0, 1, 1, C.byref(handle)))
    yield lib, handle
    abi.check(lib.b200_runner_destroy(handle))


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [np.uint8, np.uint16, np.uint32])
@pytest.mark.parametrize("nbytes", [4, 4096, 262140, 262144, CHUNK - 4, CHUNK + 4, 4 * 1024 * 1024, 33 * CHUNK + 12, 9000004])
def test_pull(runner, dtype, nbytes):
    lib, handle = runner
    want = np.frombuffer(np.random.default_rng(nbytes).bytes(nbytes), dtype=dtype)
    ptr = C.c_void_p()
    abi.check(lib.b200_array_alloc(handle, nbytes, C.byref(ptr)))
    abi.check(lib.b200_array_push(handle, ptr, want.ctypes.data, nbytes))
    got, wide = np.zeros_like(want), np.zeros(want.size, np.uint32)
    abi.check(lib.b200_array_pull(handle, got.ctypes.data, ptr, nbytes))
    abi.check(lib.b200_array_pull_u32(handle, wide.ctypes.data, ptr, want.itemsize, want.size))
    abi.check(lib.b200_array_free(handle, ptr))
    np.testing.assert_array_equal(got, want)
    np.testing.assert_array_equal(wide, want.astype(np.uint32))
