"""The target-resident kernel in windows of steps (resident_window.cuh) against the CPU checker: both reasons for a window, every
connectivity, windows cut short by the end of a call, calls that go on where others ended, spikes from before a call, several
source populations, rates at the ends of the range, and the sizes at which the kernel stops applying."""
import numpy as np
import pytest

from genn_b200 import GeNNModel, init_postsynaptic, init_weight_update
from genn_b200.resolve import resolve
from tests import helpers
from tests.test_gpu_parity import _runtime

pytestmark = pytest.mark.gpu
LIF = {"C": 0.25, "TauM": 20.0, "Vrest": -65.0, "Vreset": -70.0, "Vthresh": -50.0, "Ioffset": 0.1, "TauRefrac": 2.0}
CALLS = (4, 5, 1, 16, 17, 3, 40)


def _sources(m, name, kind, n, rng, rate=60.0):
    if kind == "Poisson":
        return m.add_neuron_population(name, n, "Poisson", {"rate": rate}, {"timeStepToSpike": 0.0})
    trains = [np.sort(rng.integers(0, 90, c)).astype(np.float32) for c in np.arange(n) % 7]
    ends = np.cumsum([len(t) for t in trains]).astype(np.uint32)
    src = m.add_neuron_population(name, n, "SpikeSourceArray", {}, {"startSpike": np.concatenate([[0], ends[:-1]]).astype(np.uint32), "endSpike": ends})
    src.set_extra_global_param("spikeTimes", np.concatenate(trains))
    return src


def _connect(m, name, kind, src, trg, rng, delay, psm=("ExpCurr", {"tau": 4.0}), scale=1.0, k=20):
    ns, nt = src.num_neurons, trg.num_neurons
    if kind == "DENSE":
        sg = m.add_synapse_population(name, "DENSE", src, trg, init_weight_update("StaticPulse", {}, {"g": (scale * rng.uniform(-0.001, 0.006, (ns, nt))).astype(np.float32)}),
                                      init_postsynaptic(*psm))
    else:
        pre, post = np.repeat(np.arange(ns, dtype=np.uint32), k), rng.integers(0, nt, ns * k).astype(np.uint32)
        if kind == "BITMASK":
            sg = m.add_synapse_population(name, "BITMASK", src, trg, init_weight_update("StaticPulseConstantWeight", {"g": 0.02 * scale}), init_postsynaptic(*psm))
        else:
            sg = m.add_synapse_population(name, "SPARSE", src, trg, init_weight_update("StaticPulse", {}, {"g": (scale * rng.uniform(-0.01, 0.06, ns * k)).astype(np.float32)}),
                                          init_postsynaptic(*psm))
        sg.set_sparse_connections(pre, post)
    sg.axonal_delay_steps = delay
    return sg


def _feed(kind, source, pre, post, delay):
    rng = np.random.default_rng(pre + post)
    m = GeNNModel("float", "feed")
    m.dt, m.seed = 1.0, 5
    src = _sources(m, "src", source, pre, rng)
    trg = m.add_neuron_population("trg", post, "LIF", LIF, {"V": rng.uniform(-65, -51, post).astype(np.float32), "RefracTime": 0.0})
    src.spike_recording_enabled = trg.spike_recording_enabled = True
    _connect(m, "syn", kind, src, trg, rng, delay)
    return m


def _late(delay, scale=1.0):
    """A recurrent network whose groups all have one axonal delay; conductances and a source population among them."""
    rng = np.random.default_rng(delay)
    m = GeNNModel("float", "late")
    m.dt, m.seed = 1.0, 9
    src = _sources(m, "src", "Poisson", 70, rng)
    a = m.add_neuron_population("a", 330, "LIF", dict(LIF, Ioffset=0.25), {"V": rng.uniform(-65, -50, 330).astype(np.float32), "RefracTime": 0.0})
    b = m.add_neuron_population("b", 45, "Izhikevich", {"a": 0.02, "b": 0.2, "c": -65.0, "d": 8.0}, {"V": rng.uniform(-65, -55, 45).astype(np.float32), "U": -13.0})
    _connect(m, "sa", "SPARSE", src, a, rng, delay)
    _connect(m, "aa", "SPARSE", a, a, rng, delay, ("ExpCond", {"tau": 5.0, "E": 0.0}), 0.02)
    _connect(m, "ab", "BITMASK", a, b, rng, delay, ("DeltaCurr", {}), 50.0, 10)
    _connect(m, "ba", "DENSE", b, a, rng, delay)
    for p in (src, a, b):
        p.spike_recording_enabled = True
    return m


def _several(delay):
    """Two kinds of sources onto one fused input and another, a population that drives nobody and one that nobody drives."""
    rng = np.random.default_rng(1)
    m = GeNNModel("float", "several")
    m.dt, m.seed = 1.0, 2
    m.fuse_postsynaptic_models = True
    p, q = _sources(m, "p", "Poisson", 129, rng), _sources(m, "q", "SpikeSourceArray", 64, rng)
    idle = _sources(m, "idle", "Poisson", 40, rng)
    trg = m.add_neuron_population("trg", 300, "LIF", LIF, {"V": rng.uniform(-65, -51, 300).astype(np.float32), "RefracTime": 0.0})
    alone = m.add_neuron_population("alone", 33, "LIF", dict(LIF, Ioffset=0.4), {"V": -60.0, "RefracTime": 0.0})
    _connect(m, "s0", "SPARSE", p, trg, rng, delay)
    _connect(m, "s1", "DENSE", q, trg, rng, delay)
    _connect(m, "s2", "BITMASK", p, trg, rng, delay, ("ExpCond", {"tau": 5.0, "E": 0.0}), 0.02)
    for x in (p, q, idle, trg, alone):
        x.spike_recording_enabled = True
    return m


def _check(build, window, ctas=0, calls=CALLS, warps=0, windows=True, patience=None):
    from oracle.oracle import OracleRunner
    net, total = resolve(build()), sum(calls)
    rt, orc, other = _runtime(net, total), OracleRunner(resolve(build()), total), _runtime(resolve(build()), total)
    other.set_option("use_fused", 0)                # (counts the same spikes and events)
    rt.set_option("resident_ctas", ctas)
    rt.set_option("resident_warps", warps)
    rt.set_option("use_windows", windows)
    if patience is not None:
        rt.set_option("resident_patience", patience)
    assert rt.counter("window_steps") == window
    holds = set()
    for r in (rt, other):
        r.set_option("count_events", 1)
    done, seen = 0, {p.name: [] for p in net.pops}
    for n in calls:
        rt.step_time(n)
        other.step_time(n)
        holds.add(rt.counter("resident_hold"))
        for _ in range(n):
            orc.step(1)
            done += 1
            for p in net.pops:
                seen[p.name] += [(done - 1, int(i)) for i in orc.current_spikes(p.name)]
        for p in net.pops:
            assert np.array_equal(np.sort(rt.current_spikes(p.name)), np.sort(orc.current_spikes(p.name))), f"step {done} {p.name}"
            if "V" in p.vars:
                helpers.assert_close(rt.array(f"{p.name}.V")[0], orc.array(f"{p.name}.V")[0], f"step {done} V {p.name}", 1e-5, 5e-6)
        for i in range(len(net.psms)):
            helpers.assert_close(rt.array(f"psm{i}.out_post")[0], orc.array(f"psm{i}.out_post")[0], f"step {done} input {i}", 1e-5, 5e-6)
    assert rt.counter("spikes") == other.counter("spikes") == sum(map(len, seen.values()))
    assert rt.counter("synaptic_events") == other.counter("synaptic_events") > 0
    rt.synchronize()
    rt.pull_recording_buffers()
    for p in net.pops:
        if p.record:
            times, ids = rt.recorded_spikes(p.name)[0]
            got = helpers.sorted_pairs(np.stack([np.rint(times / net.dt).astype(np.uint32), ids], axis=1))
            assert np.array_equal(got, helpers.sorted_pairs(seen[p.name])), f"recorded spikes of {p.name}"
    for r in (rt, other, orc):
        r.close()
    return holds


@pytest.mark.parametrize("delay", [0, 3, 15, 20])
@pytest.mark.parametrize("source", ["Poisson", "SpikeSourceArray"])
@pytest.mark.parametrize("kind", ["SPARSE", "DENSE", "BITMASK"])
def test_sources_ahead_match_the_cpu_checker(kind, source, delay):
    _check(lambda: _feed(kind, source, 131, 300, delay), 16)


@pytest.mark.parametrize("ctas,warps", [(1, 4), (1, 24), (3, 5), (9, 24), (148, 24)])
@pytest.mark.parametrize("kind", ["SPARSE", "DENSE", "BITMASK"])
def test_grids_and_blocks(kind, ctas, warps):
    """All warps read messages, or those without neurons; a warp reads one message or many."""
    _check(lambda: _feed(kind, "Poisson", 33, 65, 1), 16, ctas, (16, 33, 2), warps)


@pytest.mark.parametrize("pre,window", [(2560, 16), (2561, 15), (10240, 4), (10241, 0)])
def test_windows_shrink_as_the_sources_grow(pre, window):
    _check(lambda: _feed("SPARSE", "Poisson", pre, 40, 0), window, calls=(5, 16, 7))


@pytest.mark.parametrize("delay,window", [(2, 0), (3, 4), (6, 7), (15, 16), (16, 0), (19, 10), (20, 7)])
def test_one_axonal_delay_matches_the_cpu_checker(delay, window):
    """Windows of the delay and one step, or of a whole part of that; none where it has no such part of four steps and more."""
    _check(lambda: _late(delay), window, calls=(4, 5, 1, 16, 30))


@pytest.mark.parametrize("delay", [0, 2])
def test_several_sources_and_populations_on_their_own(delay):
    _check(lambda: _several(delay), 16)


@pytest.mark.parametrize("rate", [1e-7, 3.0, 900.0, 2500.0])
def test_rates_at_the_ends_of_the_range(rate):
    """Intervals beyond 2^24 steps, and of less than one."""
    def build():
        rng = np.random.default_rng(4)
        m = GeNNModel("float", "rates")
        m.dt, m.seed = 1.0, 8
        src = _sources(m, "src", "Poisson", 64, rng, rate)
        one = m.add_neuron_population("one", 32, "Poisson", {"rate": 50.0}, {"timeStepToSpike": 0.5})
        trg = m.add_neuron_population("trg", 64, "LIF", LIF, {"V": -60.0, "RefracTime": 0.0})
        _connect(m, "syn", "SPARSE", src, trg, rng, 0, scale=0.1)
        _connect(m, "syn1", "SPARSE", one, trg, rng, 0)
        return m
    _check(build, 16)


def test_windows_and_single_steps_hand_over_to_each_other():
    """Calls of one to three steps go step by step, longer ones in windows, and the option changes the kernel in between."""
    from oracle.oracle import OracleRunner
    net = resolve(_late(7))
    rt, orc = _runtime(net, 100), OracleRunner(resolve(_late(7)), 100)
    for i, n in enumerate((1, 9, 2, 3, 20, 1, 8, 11)):
        rt.set_option("use_windows", 0 if i == 4 else 1)
        assert rt.counter("window_steps") == (0 if i == 4 else 8)
        rt.step_time(n)
        orc.step(n)
        for p in net.pops:
            assert np.array_equal(np.sort(rt.current_spikes(p.name)), np.sort(orc.current_spikes(p.name))), p.name
        helpers.assert_close(rt.array("a.V")[0], orc.array("a.V")[0], "V", 1e-5, 5e-6)
    rt.close()
    orc.close()


@pytest.mark.parametrize("build", [lambda: _late(7), lambda: _feed("SPARSE", "Poisson", 500, 2000, 2)], ids=["late", "feed"])
def test_a_model_built_where_another_of_its_kind_ended(build):
    """Models built and closed one after another get the same memory, and their calls end at the same steps: what an earlier one left
    there is not taken for a word of this one.  (The lists of spikes a call leaves are emptied by one CTA before all fill them.)"""
    from oracle.oracle import OracleRunner
    calls, want = (24, 9, 33), []
    orc = OracleRunner(resolve(build()), sum(calls))
    for n in calls:
        orc.step(n)
        want.append({p.name: np.sort(orc.current_spikes(p.name)) for p in orc.net.pops})
    assert sum(len(v) for v in want[0].values()) > 0
    for _ in range(30):
        rt = _runtime(resolve(build()), sum(calls))
        rt.set_option("resident_ctas", 148)
        assert rt.counter("window_steps") > 0
        for n, spikes in zip(calls, want):
            rt.step_time(n)
            for name, ids in spikes.items():
                assert np.array_equal(np.sort(rt.current_spikes(name)), ids), name
        rt.close()
    orc.close()


@pytest.mark.parametrize("rows", [1, 3, 7, 15, 16, 17])
@pytest.mark.parametrize("build", [lambda: _feed("SPARSE", "Poisson", 131, 300, 2), lambda: _late(15)], ids=["feed", "late"])
def test_recordings_of_fewer_steps_than_a_window(build, rows):
    """A recording holds the last steps of a call, however few: the rows of the steps before, of the same window too, are written over."""
    from oracle.oracle import OracleRunner
    net = resolve(build())
    rt, orc = _runtime(net, rows), OracleRunner(resolve(build()), rows)
    assert rt.counter("window_steps") == 16
    done, seen = 0, {p.name: [] for p in net.pops}
    for n in (21, 16, 37, 64):
        rt.step_time(n)
        for _ in range(n):
            orc.step(1)
            done += 1
            for p in net.pops:
                seen[p.name] += [(done - 1, int(i)) for i in orc.current_spikes(p.name)]
        rt.synchronize()
        rt.pull_recording_buffers()
        for p in net.pops:
            want = [s for s in seen[p.name] if s[0] >= done - rows]
            times, ids = rt.recorded_spikes(p.name)[0]
            got = np.stack([np.rint(times / net.dt).astype(np.uint32), ids], axis=1)
            assert np.array_equal(helpers.sorted_pairs(got), helpers.sorted_pairs(np.array(want, np.int64).reshape(-1, 2))), f"{p.name} after {done} steps"
    assert sum(map(len, seen.values())) > 1000
    rt.close()
    orc.close()


def _busy(kind, delay):
    """Sources of half a spike a step, alone (feed), with a recurrent population (late), or with one that fires as a whole (burst)."""
    rng = np.random.default_rng(delay)
    n = 3000 if kind == "burst" else 200
    m = GeNNModel("float", "busy")
    m.dt, m.seed = 1.0, 23
    src = _sources(m, "in", "Poisson", 300, rng, 600.0)
    trg = m.add_neuron_population("out", n, "LIF", dict(LIF, Ioffset=0.3), {"V": -65.0 if kind == "burst" else rng.uniform(-65, -50, n).astype(np.float32), "RefracTime": 0.0})
    src.spike_recording_enabled = trg.spike_recording_enabled = True
    _connect(m, "syn", "SPARSE", src, trg, rng, delay, scale=1e-4, k=10)
    if kind != "feed":
        _connect(m, "rec", "SPARSE", trg, trg, rng, delay, scale=1e-4, k=10)
    return m


@pytest.mark.parametrize("kind,delay,window", [("feed", 0, 16), ("feed", 5, 16), ("feed", 21, 16), ("late", 15, 16), ("late", 19, 10), ("late", 44, 15), ("burst", 19, 10)])
def test_a_busy_network_leaves_in_the_middle_of_a_call(kind, delay, window):
    """Launches that end early behind a window, the sources of some a window ahead by then, others with spikes that are still on their way
    in messages of one to three windows; the other kernel's share of the call, and this kernel again."""
    holds = _check(lambda: _busy(kind, delay), window, calls=(1, 2, 3, 5, 60, 1, 1, 40, 87), warps=4, patience=1e6 if kind == "burst" else 0)
    assert len(holds) >= 3, holds       # (left more than once)


def test_messages_take_no_more_than_some_spike_queues():
    """They have room for every neuron in every step of a delay, as the queues have, and go back with the rest."""
    n, delay = 20000, 199
    rng = np.random.default_rng(6)
    m = GeNNModel("float", "messages")
    m.dt, m.seed = 1.0, 7
    a = m.add_neuron_population("a", n, "LIF", LIF, {"V": -60.0, "RefracTime": 0.0})
    _connect(m, "aa", "SPARSE", a, a, rng, delay, k=2)
    rt = _runtime(resolve(m), 10)
    assert rt.counter("window_steps") == 10
    queue, size = 4 * n * (delay + 4), rt.counter("resident_message_bytes")
    assert queue < size < 2.5 * queue + 0.25e6 * delay
    rt.step_time(30)
    rt.set_option("use_windows", 0)
    assert rt.counter("resident") == 1 and rt.counter("resident_message_bytes") < size
    rt.set_option("use_resident", 0)
    rt.step_time(5)
    assert rt.counter("resident_message_bytes") == 0
    rt.set_option("use_resident", 1)
    rt.set_option("use_windows", 1)
    assert rt.counter("resident") == 1 and rt.counter("resident_message_bytes") == size
    rt.close()


@pytest.mark.parametrize("windows", [True, False])
@pytest.mark.parametrize("groups,warps", [(64, 2), (32, 1), (63, 2)])
def test_as_many_populations_as_a_block_has_threads(groups, warps, windows):
    """The table of a CTA's warps has an entry more than there are populations; groups without a run of entries onto the last one use it."""
    def build():
        rng = np.random.default_rng(groups)
        m = GeNNModel("float", "many")
        m.dt, m.seed = 1.0, 3
        src = _sources(m, "src", "Poisson", 30, rng, 200.0)
        pops = [m.add_neuron_population(f"p{i}", 1 + (i * 7) % 32, "LIF", LIF, {"V": -56.0, "RefracTime": 0.0}) for i in range(groups - 1)]
        for i, trg in ((0, pops[0]), (1, pops[-2]), (2, pops[-1])):
            _connect(m, f"d{i}", "DENSE", src, trg, rng, 1)
            _connect(m, f"b{i}", "BITMASK", src, trg, rng, 1, k=1)
        return m
    _check(build, 16 if windows else 0, groups, (5, 1, 17, 2), warps, windows)
