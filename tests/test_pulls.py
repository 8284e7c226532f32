"""Arrays on their way out of the device: every size class, and indices widened on the way."""
import ctypes as C
import mmap
import threading

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


@pytest.mark.gpu
@pytest.mark.parametrize("n", [65536, 65537, 262144, 262145])
def test_a_view_pulled_often_stays_right_and_outlives_its_model(n):
    from genn_b200 import GeNNModel
    m = GeNNModel("float", "views")
    m.dt = 1.0
    pop = m.add_neuron_population("pop", n, "LIF", {"C": 1.0, "TauM": 20.0, "Vrest": -65.0, "Vreset": -70.0, "Vthresh": -50.0, "Ioffset": 0.0,
                                                    "TauRefrac": 2.0}, {"V": -65.0, "RefracTime": 0.0})
    m.build()
    m.load()
    v = pop.vars["V"]
    for i in range(20):
        v.view[...] = np.arange(n, dtype=np.float32) + i
        v.push_to_device()
        v.view[...] = 0.0
        v.pull_from_device()
        np.testing.assert_array_equal(v.view, np.arange(n, dtype=np.float32).reshape(v.view.shape) + i)
    part = v.view.reshape(-1)[1:]
    m.unload()
    del m, pop, v
    np.testing.assert_array_equal(part, np.arange(1, n, dtype=np.float32) + 19)


class _Registered:
    """What the library's page-locking calls were given."""

    def __init__(self):
        self.now, self.ever = {}, []

    def b200_host_register(self, address, nbytes):
        self.now[address] = nbytes
        self.ever.append((address, nbytes))
        return 0

    def b200_host_unregister(self, address):
        del self.now[address]


@pytest.mark.parametrize("n", [65537, 100003, 262144, 1048575])
def test_page_locked_views_lie_in_pages_of_their_own_and_are_unlocked_with_their_memory(n, monkeypatch):
    from genn_b200 import runtime
    from genn_b200.model import Variable
    lib = _Registered()
    monkeypatch.setattr(abi, "load_library", lambda: lib)
    views = []
    for i in range(5):
        v = Variable(f"v{i}", np.float32, None, (1, n))
        v._array = runtime.DeviceArray.__new__(runtime.DeviceArray)
        assert v.view.shape == (1, n) and v.view.dtype == np.float32 and not v.view.any()
        v._array.lock(v.view)
        views.append(v)
    assert len(lib.now) == 5 and len(lib.ever) == 5
    spans = sorted(lib.ever)
    for (a, na), (b, _) in zip(spans, spans[1:] + [(1 << 63, 0)]):
        assert a % mmap.PAGESIZE == 0 and na % mmap.PAGESIZE == 0 and na >= 4 * n and a + na <= b
    for v in views:
        owner = v.view
        while isinstance(owner.base, np.ndarray):
            owner = owner.base
        at, size = v.view.ctypes.data, lib.now[v.view.ctypes.data]
        assert owner.ctypes.data <= at and at + size <= owner.ctypes.data + owner.nbytes
    part = views[0].view.reshape(-1)[10:20]
    held = views[0].view.ctypes.data
    del v, owner, views
    assert list(lib.now) == [held]
    del part
    assert not lib.now and runtime._view_bytes == 0


@pytest.mark.gpu
def test_threads_that_pull_from_one_runner_each_get_their_own(runner):
    """Small arrays, spike lists and the error word pass through one staging buffer of the runner."""
    lib, handle = runner
    wrong, arrays = [], []
    for k in range(4):
        want = np.arange(1000 + 900 * k, dtype=np.uint32) + 100000 * k
        want[0] = want.size - 1         # (as a spike list: the count, then the ids)
        ptr = C.c_void_p()
        abi.check(lib.b200_array_alloc(handle, want.nbytes, C.byref(ptr)))
        abi.check(lib.b200_array_push(handle, ptr, want.ctypes.data, want.nbytes))
        arrays.append((want, ptr))

    def work(k):
        want, ptr = arrays[k]
        n, got, ids, num = want.size, np.zeros_like(want), np.zeros_like(want), C.c_uint32()
        for _ in range(1500):
            got[:] = 0
            abi.check(lib.b200_array_pull(handle, got.ctypes.data, ptr, got.nbytes))
            abi.check(lib.b200_pull_spikes(handle, ptr.value, ptr.value + 4, n - 1, ids.ctypes.data, C.byref(num)))
            abi.check(lib.b200_synchronize(handle))
            if num.value != n - 1 or not np.array_equal(got, want) or not np.array_equal(ids[:n - 1], want[1:]):
                wrong.append(k)
                return

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
