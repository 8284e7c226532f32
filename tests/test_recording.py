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


def test_room_for_the_non_zero_words():
    """One in eight of short recordings; a long one asks for no more page-locked memory at first than one in sixteen; never less for
    more words."""
    from genn_b200.runtime import pairs_room
    assert [pairs_room(n) for n in (0, 100, 8192, 313000, 8 << 20, 16 << 20, 250000000)] == [1024, 1024, 1024, 39125, 1 << 19, 1 << 20, 15625000]
    rooms = [pairs_room(n) for n in range(0, 40 << 20, 99991)]
    assert rooms == sorted(rooms)


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


@pytest.mark.gpu
@pytest.mark.parametrize("rate", [1.0, 2.4, 3.4, 5.0])
def test_long_recordings_come_as_pairs_up_to_one_word_in_eight(rate):
    """1.25 M words, of which 3, 7, 10 and 15 % are not zero: fewer than the list has room for at first, more, and too many."""
    from genn_b200 import GeNNModel, init_postsynaptic, init_weight_update
    n, steps = 40000, 1000
    m = GeNNModel("float", "recording")
    m.dt, m.seed = 1.0, 3
    src = m.add_neuron_population("src", n, "Poisson", {"rate": rate}, {"timeStepToSpike": 0.0})
    trg = m.add_neuron_population("trg", 32, "LIF", {"C": 0.25, "TauM": 20.0, "Vrest": -65.0, "Vreset": -70.0, "Vthresh": -50.0, "Ioffset": 0.0, "TauRefrac": 2.0},
                                  {"V": -65.0, "RefracTime": 0.0})
    src.spike_recording_enabled = True
    sg = m.add_synapse_population("syn", "SPARSE", src, trg, init_weight_update("StaticPulseConstantWeight", {"g": 0.0}), init_postsynaptic("DeltaCurr", {}))
    sg.set_sparse_connections(np.arange(n, dtype=np.uint32), np.arange(n, dtype=np.uint32) % 32, presorted=True)
    m.build()
    m.load(num_recording_timesteps=steps)
    rt = m._runtime
    for _ in range(2):
        m.step_time(steps)
        rt.recording_pairs_capacity = None
        m.pull_recording_buffers_from_device()
        times, ids = rt.recorded_spikes("src")[0]
        share = len(rt._rec_pairs) / (steps * n / 32) if rt._rec_pairs is not None else 1.0
        assert (rt._rec_pairs is None) == (rate == 5.0) and (share > 1 / 16) == (rate > 2.0)
        rt.recording_pairs_capacity = 1
        m.pull_recording_buffers_from_device()
        assert rt._rec_pairs is None
        whole = rt.recorded_spikes("src")[0]
        assert np.array_equal(times, whole[0]) and np.array_equal(ids, whole[1]) and len(ids) > 0.8 * n * rate * steps * 1e-3
    m.unload()
