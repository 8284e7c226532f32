"""The recording list (record.cuh) and its decoding, at the sizes where they can go wrong: chunk edges of the listing
kernels, padding bits, rings that start in the middle, batches, more arrays than one launch takes."""
import ctypes as C

import numpy as np
import pytest

from genn_b200 import abi


def _numpy_decode(words, num_neurons, first_row, first_id, start, dt):
    out = []
    for b in range(words.shape[1]):
        bits = np.unpackbits(np.ascontiguousarray(np.roll(words, -first_row, axis=0)[:, b, :]).view(np.uint8), axis=1, bitorder="little")
        step, ids = np.nonzero(bits[:, :num_neurons])
        out.append((start + step * dt, (ids + first_id).astype(np.uint32)))
    return out


@pytest.mark.parametrize("rows,batch,num_neurons,first_row,density", [(1, 1, 1, 0, 1.0), (7, 1, 32, 3, 0.3), (5, 3, 33, 4, 0.2), (20, 2, 95, 0, 0.02),
                                                                      (4, 1, 64, 2, 0.0), (50, 3, 70, 20, 0.03)])
@pytest.mark.parametrize("whole", [False, True])
def test_decoded_spikes_equal_the_unpacked_bits(rows, batch, num_neurons, first_row, density, whole):
    lib = abi.load_library()
    rng = np.random.default_rng(rows * 100 + num_neurons)
    per_row = (num_neurons + 31) // 32
    words = np.where(rng.random((rows, batch, per_row)) < density, rng.integers(1, 2 ** 32, size=(rows, batch, per_row), dtype=np.uint64), 0).astype(np.uint32)
    # the array lies between two others in the list
    base = 11
    flat = np.concatenate([np.full(base, 5, np.uint32), words.reshape(-1), np.full(9, 7, np.uint32)])
    index = np.flatnonzero(flat)
    pairs = np.ascontiguousarray(np.stack([index, flat[index]], axis=1).astype(np.uint32))
    source = (words.ctypes.data, None, 0) if whole else (None, pairs.ctypes.data, len(pairs))
    counts = (C.c_uint64 * batch)()
    args = (*source, base, rows, batch, per_row, first_row, num_neurons, 3, 1.5, 0.1, counts)
    abi.check(lib.b200_decode_recording(*args, None, None))
    got = [(np.empty(n, np.float64), np.empty(n, np.uint32)) for n in counts]
    abi.check(lib.b200_decode_recording(*args, (C.c_void_p * batch)(*[t.ctypes.data for t, _ in got]), (C.c_void_p * batch)(*[i.ctypes.data for _, i in got])))
    for (t, i), (wt, wi) in zip(got, _numpy_decode(words, num_neurons, first_row, 3, 1.5, 0.1)):
        assert np.array_equal(t, wt) and np.array_equal(i, wi)


@pytest.mark.parametrize("whole", [False, True])
def test_a_batch_entry_without_spikes_needs_no_room(whole):
    """Bits beyond the neurons are no spikes: an entry that has nothing else may come without arrays, and those behind it are decoded."""
    lib = abi.load_library()
    words = np.zeros((3, 2, 2), np.uint32)
    words[:, 0, 1] = 1 << 20            # (beyond neuron 39)
    words[:, 1] = 5, 1 << 6
    index = np.flatnonzero(words)
    pairs = np.ascontiguousarray(np.stack([index, words.reshape(-1)[index]], axis=1).astype(np.uint32))
    source = (words.ctypes.data, None, 0) if whole else (None, pairs.ctypes.data, len(pairs))
    counts = (C.c_uint64 * 2)()
    args = (*source, 0, 3, 2, 2, 1, 40, 0, 0.0, 1.0, counts)
    abi.check(lib.b200_decode_recording(*args, None, None))
    assert list(counts) == [0, 9]
    times, ids = np.full(9, -1.0), np.full(9, 99, np.uint32)
    abi.check(lib.b200_decode_recording(*args, (C.c_void_p * 2)(None, times.ctypes.data), (C.c_void_p * 2)(None, ids.ctypes.data)))
    assert np.array_equal(times, np.repeat([0.0, 1.0, 2.0], 3)) and np.array_equal(ids, np.tile([0, 2, 38], 3)) and list(counts) == [0, 9]


@pytest.mark.gpu
@pytest.mark.parametrize("sizes,density", [([1], 1.0), ([4095, 4096, 4097], 0.05), ([16] * 60, 0.5), ([100003], 0.01), ([5000, 0, 37], 0.0)])
def test_the_list_holds_the_non_zero_words_in_order(sizes, density):
    lib = abi.load_library()
    rng = np.random.default_rng(len(sizes))
    h = C.c_void_p()
    abi.check(lib.b200_runner_create(0, 0.1, 0, 1, C.byref(h)))
    flat = np.where(rng.random(sum(sizes)) < density, rng.integers(1, 2 ** 32, size=sum(sizes), dtype=np.uint64), 0).astype(np.uint32)
    ptrs, at = [], 0
    for n in sizes:
        p = C.c_void_p()
        abi.check(lib.b200_array_alloc(h, max(4, 4 * n), C.byref(p)))
        part = np.ascontiguousarray(flat[at:at + n])
        if n:
            abi.check(lib.b200_array_push(h, p, part.ctypes.data, 4 * n))
        ptrs.append(p.value)
        at += n
    index = np.flatnonzero(flat)
    for capacity in (len(flat) + 1, max(1, len(index)), max(1, len(index) - 1)):
        pairs, count = C.c_void_p(), C.c_uint64()
        abi.check(lib.b200_pull_recording(h, len(sizes), (C.c_void_p * len(sizes))(*ptrs), (C.c_uint64 * len(sizes))(*sizes), capacity,
                                          C.byref(pairs), C.byref(count)))
        assert count.value == len(index)
        assert bool(pairs.value) == (len(index) <= capacity)
        if pairs.value and len(index):
            got = np.ctypeslib.as_array((C.c_uint32 * (2 * len(index))).from_address(pairs.value)).reshape(-1, 2)
            assert np.array_equal(got[:, 0], index) and np.array_equal(got[:, 1], flat[index])
    lib.b200_runner_destroy(h)
