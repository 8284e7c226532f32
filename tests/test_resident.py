"""The target-resident time-step path (resident.cu) against the reference's golden vectors and the CPU checker: every grid
size and block size changes which CTA holds a neuron, launches of every length hand over to the other paths, more
spikes than a message head or the delivery list holds, several axonal delays and ring depths in one model."""
import numpy as np
import pytest

from genn_b200 import GeNNModel, abi, init_postsynaptic, init_weight_update
from genn_b200.resolve import resolve
from tests import helpers
from tests.cases import CASES
from tests.test_gpu_parity import _Adapter, _runtime

pytestmark = pytest.mark.gpu
NAMES = ["ff_sparse", "ff_sparse_narrow", "ff_bitmask", "ff_dense", "potjans_mini", "potjans_mini_d1", "cond_delay", "izhikevich", "c1_full"]


def _resident(name, ctas=0, warps=0):
    model, steps, dump_every = CASES[name]()
    net = resolve(model)
    rt = _runtime(net, steps)
    rt.set_option("resident_ctas", ctas)
    rt.set_option("resident_warps", warps)
    assert rt.counter("resident") == 1
    return net, rt, steps, dump_every


@pytest.mark.parametrize("ctas,warps", [(0, 0), (1, 24), (7, 4), (148, 24)])
@pytest.mark.parametrize("name", NAMES)
def test_all_steps_in_one_launch_match_the_reference(name, ctas, warps):
    net, rt, steps, _ = _resident(name, ctas, warps)
    rt.set_option("count_events", 1)
    before = rt.kernel_launches
    rt.step_time(steps)
    rt.synchronize()
    assert rt.kernel_launches == before + 1
    rt.pull_recording_buffers()
    want = helpers.load_golden(name)
    for p in net.pops:
        if p.record:
            times, ids = rt.recorded_spikes(p.name)[0]
            got = helpers.sorted_pairs(np.stack([np.rint(times / net.dt).astype(np.uint32), ids], axis=1))
            assert np.array_equal(got, want[f"spikes_{p.name}"]), f"recorded spikes of {p.name} differ"
    final = helpers.snapshot(_Adapter(rt), net, steps)
    helpers.compare(final, {k: v for k, v in want.items() if k.endswith(f"_{steps}")}, exact_state=False, rtol=1e-5, atol=2e-6)
    assert rt.counter("spikes") == sum(len(want[f"spikes_{p.name}"]) for p in net.pops)
    rt.close()


@pytest.mark.parametrize("name", ["ff_sparse", "ff_bitmask", "potjans_mini", "cond_delay", "izhikevich"])
def test_launches_of_every_length_hand_over_to_the_other_paths(name):
    """Steps on this path alternate with steps on the one-launch-per-kernel path: spike lists, rings and state between
    launches must be what that path expects, and the current spikes those of the reference."""
    net, rt, steps, dump_every = _resident(name)
    chunk = [1, 2, 1, 5, 3, 17, 1, 1, 40]
    spikes = {p.name: [] for p in net.pops}
    done = i = 0
    while done < steps:
        n = min(chunk[i % len(chunk)], steps - done)
        rt.set_option("use_fused", 0 if (i % 3 == 2) else 1)
        rt.step_time(n)
        done += n
        i += 1
        for p in net.pops:
            spikes[p.name] += [(done - 1, int(j)) for j in rt.current_spikes(p.name)]
    want = helpers.load_golden(name)
    for p in net.pops:
        ends = {s for s, _ in spikes[p.name]}
        ref = np.array([q for q in want[f"spikes_{p.name}"] if int(q[0]) in ends]).reshape(-1, 2)
        assert np.array_equal(helpers.sorted_pairs(spikes[p.name]), helpers.sorted_pairs(ref)), p.name
    final = helpers.snapshot(_Adapter(rt), net, steps)
    helpers.compare(final, {k: v for k, v in want.items() if k.endswith(f"_{steps}")}, exact_state=False, rtol=1e-5, atol=2e-6)
    rt.close()


@pytest.mark.parametrize("ctas", [1, 3, 40])
@pytest.mark.parametrize("zero,synapses", [(0, 90), (1, 90), (2, 37), (64, 150), (65, 150), (150, 150)])
def test_heads_and_shares_of_runs_match_the_cpu_checker(zero, synapses, ctas):
    """`zero` synapses of every row have delay 0: no heads, heads of one entry, as many as a run may have, more than that (the
    whole class in front of the update then), nothing else; rows of more than 128 entries are shared out between warps."""
    from oracle.oracle import OracleRunner
    rng = np.random.default_rng(zero + synapses)
    n = 300

    def model():
        m = GeNNModel("float", "heads")
        m.dt = 1.0
        lif = {"C": 0.25, "TauM": 20.0, "Vrest": -65.0, "Vreset": -70.0, "Vthresh": -50.0, "Ioffset": 0.3, "TauRefrac": 2.0}
        pops = [m.add_neuron_population(name, n, "LIF", lif, {"V": v0[name], "RefracTime": 0.0}) for name in "ab"]
        for i, (src, trg) in enumerate(((pops[0], pops[1]), (pops[1], pops[1]))):
            sg = m.add_synapse_population(f"s{i}", "SPARSE", src, trg, init_weight_update("StaticPulseDendriticDelay", {}, {"g": g[i], "d": d}),
                                          init_postsynaptic("ExpCurr", {"tau": 3.0}))
            sg.set_sparse_connections(pre, post[i], presorted=True)
            sg.max_dendritic_delay_timesteps = 5
        return m

    v0 = {name: rng.uniform(-65, -49, n).astype(np.float32) for name in "ab"}
    pre = np.repeat(np.arange(n, dtype=np.uint32), synapses)
    # (equal targets side by side as well: rows are drawn with replacement)
    post = [np.sort(rng.integers(0, n, (n, synapses)), axis=1).astype(np.uint32).ravel() for _ in range(2)]
    d = np.tile(np.where(np.arange(synapses) < zero, 0, 1 + np.arange(synapses) % 4).astype(np.uint8), n)
    g = [rng.uniform(0, 2e-3, n * synapses).astype(np.float32) for _ in range(2)]
    net = resolve(model())
    rt, orc = _runtime(net, 20), OracleRunner(resolve(model()), 20)
    rt.set_option("resident_ctas", ctas)
    assert rt.counter("resident") == 1
    rt.set_option("count_events", 1)
    for steps in (1, 1, 6, 12):
        rt.step_time(steps)
        orc.step(steps)
        for p in net.pops:
            assert np.array_equal(np.sort(rt.current_spikes(p.name)), np.sort(orc.current_spikes(p.name))), p.name
            helpers.assert_close(rt.array(f"{p.name}.V")[0], orc.array(f"{p.name}.V")[0], f"V {p.name}", 1e-5, 2e-6)
    assert rt.counter("spikes") > 0 and rt.counter("synaptic_events") % synapses == 0
    rt.close()
    orc.close()


@pytest.mark.parametrize("kinds", [("ExpCurr", "ExpCond"), ("ExpCond", "ExpCurr"), ("ExpCond", "DeltaCurr"), ("ExpCurr", "ExpCurr", "ExpCond"), ()])
def test_inputs_of_every_kind_match_the_cpu_checker(kinds):
    """LIF neurons with one, two or three unfused inputs (none of them, and the spike sources, have a neuron update of their own),
    spike sources whose trains end, begin late or hold several spikes of one step."""
    from oracle.oracle import OracleRunner
    rng = np.random.default_rng(len(kinds))
    n, k = 100, 40
    trains = [np.sort(rng.integers(0, 30, c)).astype(np.float32) for c in np.arange(n) % 5]
    v0 = rng.uniform(-65, -51, n).astype(np.float32)
    pre, posts = np.repeat(np.arange(n, dtype=np.uint32), k), [rng.integers(0, n, n * k).astype(np.uint32) for _ in kinds]
    weights = [rng.uniform(0, 0.05, n * k).astype(np.float32) for _ in kinds]

    def model():
        m = GeNNModel("float", "inputs")
        m.dt = 1.0
        ends = np.cumsum([len(t) for t in trains]).astype(np.uint32)
        src = m.add_neuron_population("src", n, "SpikeSourceArray", {}, {"startSpike": np.concatenate([[0], ends[:-1]]).astype(np.uint32), "endSpike": ends})
        src.set_extra_global_param("spikeTimes", np.concatenate(trains))
        trg = m.add_neuron_population("trg", n, "LIF", {"C": 0.25, "TauM": 20.0, "Vrest": -65.0, "Vreset": -70.0, "Vthresh": -50.0, "Ioffset": 0.4,
                                                        "TauRefrac": 2.0}, {"V": v0, "RefracTime": 0.0})
        for i, kind in enumerate(kinds):
            params = {"ExpCurr": {"tau": 3.0 + i}, "ExpCond": {"tau": 5.0 + i, "E": 0.0}, "DeltaCurr": {}}[kind]
            g = weights[i] * (0.02 if kind == "ExpCond" else 1.0)
            sg = m.add_synapse_population(f"s{i}", "SPARSE", src, trg, init_weight_update("StaticPulse", {}, {"g": g.astype(np.float32)}), init_postsynaptic(kind, params))
            sg.set_sparse_connections(pre, posts[i])
        if not kinds:       # (a model needs synapses: from the neurons without an input, onto sources that keep none of it)
            sg = m.add_synapse_population("back", "SPARSE", trg, src, init_weight_update("StaticPulse", {}, {"g": np.ones(n * k, np.float32)}), init_postsynaptic("ExpCurr", {"tau": 3.0}))
            sg.set_sparse_connections(pre, rng.integers(0, n, n * k).astype(np.uint32))
        return m

    state = rng.bit_generator.state
    net = resolve(model())
    rng.bit_generator.state = state
    rt, orc = _runtime(net, 40), OracleRunner(resolve(model()), 40)
    assert rt.counter("resident") == 1
    for steps in (1, 2, 7, 30):
        rt.step_time(steps)
        orc.step(steps)
        for p in net.pops:
            assert np.array_equal(np.sort(rt.current_spikes(p.name)), np.sort(orc.current_spikes(p.name))), p.name
        helpers.assert_close(rt.array("trg.V")[0], orc.array("trg.V")[0], "V", 1e-5, 2e-6)
        assert np.array_equal(rt.array("src.startSpike"), orc.array("src.startSpike"))
    rt.close()
    orc.close()


def _mixed():
    """Two populations that all fire at once (more spikes than a message head or the delivery list holds), groups of all
    three connectivities, axonal delays 0, 2 and 5, inputs with and without a ring."""
    rng = np.random.default_rng(3)
    m = GeNNModel("float", "mixed")
    m.dt = 1.0
    lif = {"C": 0.25, "TauM": 20.0, "Vrest": -65.0, "Vreset": -70.0, "Vthresh": -50.0, "Ioffset": 0.5, "TauRefrac": 2.0}
    a = m.add_neuron_population("a", 2500, "LIF", lif, {"V": np.where(rng.random(2500) < 0.9, -50.5, -60.0).astype(np.float32), "RefracTime": 0.0})
    b = m.add_neuron_population("b", 70, "LIF", lif, {"V": rng.uniform(-65, -50, 70).astype(np.float32), "RefracTime": 0.0})
    pre = np.repeat(np.arange(2500, dtype=np.uint32), 3)
    sg = m.add_synapse_population("ab", "SPARSE", a, b, init_weight_update("StaticPulseDendriticDelay", {}, {
        "g": rng.uniform(0, 1e-3, 7500).astype(np.float32), "d": rng.integers(0, 9, 7500).astype(np.uint8)}), init_postsynaptic("ExpCurr", {"tau": 3.0}))
    sg.set_sparse_connections(pre, rng.integers(0, 70, 7500).astype(np.uint32))
    sg.max_dendritic_delay_timesteps = 7        # delays of 7 and 8 steps wrap around
    sg.axonal_delay_steps = 2
    m.add_synapse_population("ba", "DENSE", b, a, init_weight_update("StaticPulse", {}, {"g": rng.uniform(0, 0.01, (70, 2500)).astype(np.float32)}),
                             init_postsynaptic("ExpCurr", {"tau": 5.0}))
    sg = m.add_synapse_population("aa", "BITMASK", a, a, init_weight_update("StaticPulseConstantWeight", {"g": -2e-4}), init_postsynaptic("ExpCurr", {"tau": 5.0}))
    sg.set_sparse_connections(rng.integers(0, 2500, 30000).astype(np.uint32), rng.integers(0, 2500, 30000).astype(np.uint32))
    sg.axonal_delay_steps = 5
    sg = m.add_synapse_population("aa2", "SPARSE", a, a, init_weight_update("StaticPulse", {}, {"g": rng.uniform(0, 1e-3, 7500).astype(np.float32)}),
                                  init_postsynaptic("ExpCurr", {"tau": 5.0}))
    sg.set_sparse_connections(pre, rng.integers(0, 2500, 7500).astype(np.uint32))
    return m


@pytest.mark.parametrize("ctas", [0, 4, 148])
def test_mixed_groups_and_bursts_match_the_cpu_checker(ctas):
    from oracle.oracle import OracleRunner
    net = resolve(_mixed())
    rt, orc = _runtime(net, 50), OracleRunner(resolve(_mixed()), 50)
    rt.set_option("resident_ctas", ctas)
    assert rt.counter("resident") == 1
    done = 0
    for n in (1, 1, 3, 4, 11, 20):
        rt.step_time(n)
        orc.step(n)
        done += n
        for p in net.pops:
            assert np.array_equal(np.sort(rt.current_spikes(p.name)), np.sort(orc.current_spikes(p.name))), f"step {done} {p.name}"
            helpers.assert_close(rt.array(f"{p.name}.V")[0], orc.array(f"{p.name}.V")[0], f"step {done} V {p.name}", 1e-5, 2e-6)
    rt.close()
    orc.close()


def test_pushed_weights_reach_the_private_copy():
    net, rt, steps, _ = _resident("ff_sparse")
    other = _runtime(resolve(CASES["ff_sparse"]()[0]), steps)
    other.set_option("use_fused", 0)
    for r in (rt, other):
        r.step_time(20)
        r.plan.push("syn.g", (net.syn("syn").g * 0.5).astype(np.float32))
        r.step_time(80)
    helpers.assert_close(rt.array("psm0.out_post")[0], other.array("psm0.out_post")[0], "out_post after a weight push", 1e-5, 2e-6)
    rt.close()
    other.close()


def _weights_reduced(ring):
    """A batch-1 network whose weights a custom update halves."""
    rng = np.random.default_rng(5)
    m = GeNNModel("float", "reduced")
    m.dt = 1.0
    lif = {"C": 0.25, "TauM": 20.0, "Vrest": -65.0, "Vreset": -70.0, "Vthresh": -50.0, "Ioffset": 0.3, "TauRefrac": 2.0}
    pops = [m.add_neuron_population(n, 200, "LIF", lif, {"V": rng.uniform(-65, -50, 200).astype(np.float32), "RefracTime": 0.0}) for n in "ab"]
    params = {"g": rng.uniform(0, 2e-3, 4000).astype(np.float32)}
    if ring:
        params["d"] = rng.integers(0, 4, 4000).astype(np.uint8)
    sg = m.add_synapse_population("syn", "SPARSE", *pops, init_weight_update("StaticPulseDendriticDelay" if ring else "StaticPulse", {}, params),
                                  init_postsynaptic("ExpCurr", {"tau": 5.0}))
    sg.set_sparse_connections(np.repeat(np.arange(200, dtype=np.uint32), 20), rng.integers(0, 200, 4000).astype(np.uint32))
    if ring:
        sg.max_dendritic_delay_timesteps = 4
    m.add_custom_update("halved", "train", "SUM", (sg, "g"), broadcast=True, scale=0.5)
    m.build()
    m.load()
    return m


@pytest.mark.parametrize("options", [{}, {"use_resident": 0}], ids=["resident", "grid barrier"])
@pytest.mark.parametrize("ring", [False, True])
def test_weights_changed_by_a_custom_update_reach_the_private_copies(ring, options):
    """The paths that deliver out of private copies against the one that reads the arrays."""
    runs = [(_weights_reduced(ring), o) for o in (options, {"use_fused": 0, "use_tiled": 0})]
    for m, opts in runs:
        for k, v in opts.items():
            m._runtime.set_option(k, v)
        m.step_time(30)
        for _ in range(3):
            m.custom_update("train")
            m.step_time(15)
    got, want = (m._runtime.array("psm0.out_post")[0] for m, _ in runs)
    assert np.abs(want).max() > 0
    helpers.assert_close(got, want, "out_post after custom updates", 1e-5, 2e-6)
    for m, _ in runs:
        m.unload()


def _delivering(seed=8):
    """A batch-1 SPARSE network that fires in every few steps; its weights do not learn."""
    rng = np.random.default_rng(seed)
    m = GeNNModel("float", "delivering")
    m.dt = 1.0
    lif = {"C": 0.25, "TauM": 20.0, "Vrest": -65.0, "Vreset": -70.0, "Vthresh": -50.0, "Ioffset": 0.3, "TauRefrac": 2.0}
    pops = [m.add_neuron_population(n, 200, "LIF", lif, {"V": rng.uniform(-65, -50, 200).astype(np.float32), "RefracTime": 0.0}) for n in "ab"]
    sg = m.add_synapse_population("syn", "SPARSE", *pops, init_weight_update("StaticPulse", {}, {"g": rng.uniform(0, 2e-3, 4000).astype(np.float32)}),
                                  init_postsynaptic("ExpCurr", {"tau": 5.0}))
    sg.set_sparse_connections(np.repeat(np.arange(200, dtype=np.uint32), 20), rng.integers(0, 200, 4000).astype(np.uint32))
    m.build()
    m.load()
    return m, sg


class _Foreign:
    """Device memory of the library's as another one sees it."""

    def __init__(self, pointer, shape):
        self.__cuda_array_interface__ = {"data": (pointer, False), "shape": shape, "typestr": "<f4", "version": 3}


@pytest.mark.parametrize("asked", [False, True])
def test_weights_written_through_the_device_pointer_reach_the_step(asked):
    """By default the next step sees them; a program that asks for the target-resident kernel all the same says when it wrote."""
    import torch
    (m, sg), (other, _) = _delivering(), _delivering()
    other._runtime.set_option("use_fused", 0)
    other._runtime.set_option("use_tiled", 0)
    rt = m._runtime
    assert rt.counter("resident") == 1
    abi.check(rt.lib.b200_array_expose(rt.handle, m.neuron_populations["b"].vars["V"].device_pointer + 256))    # (not an array's first byte)
    m.neuron_populations["b"].vars["V"].device_pointer          # (neuron state is read and written where it lies)
    assert rt.counter("resident") == 1
    if asked:
        rt.set_option("use_resident", 1)
    for x in (m, other):
        x.step_time(30)
    weights = [torch.as_tensor(_Foreign(x.synapse_populations["syn"].vars["g"].device_pointer, sg.vars["g"].shape), device="cuda") for x in (m, other)]
    assert rt.counter("resident") == (1 if asked else 0)
    for _ in range(3):
        for x, w in zip((m, other), weights):
            x._runtime.synchronize()
            w.mul_(0.5)
            torch.cuda.synchronize()
            if asked:
                x._runtime.set_option("rescan_delays", 1)
            x.step_time(15)
    got, want = (x._runtime.array("psm0.out_post")[0] for x in (m, other))
    assert np.abs(want).max() > 0
    helpers.assert_close(got, want, "out_post", 1e-5, 2e-6)
    for x in (m, other):
        x.unload()


def test_messages_of_steps_long_ago_are_not_taken_for_new_ones():
    """Message words carry the last 20 bits of their step.  Four steps on this path, in the first of which every source fires,
    then as many on another as bring the same bits (and the same one of the four message buffers) round again."""
    m = GeNNModel("float", "tags")
    m.dt = 1.0
    lif = {"C": 0.25, "TauM": 20.0, "Vrest": -65.0, "Vreset": -70.0, "Vthresh": -50.0, "Ioffset": 0.0, "TauRefrac": 2.0}
    a = m.add_neuron_population("a", 2368, "LIF", lif, {"V": -40.0, "RefracTime": 0.0})
    b = m.add_neuron_population("b", 2368, "LIF", dict(lif, Vthresh=1000.0), {"V": -65.0, "RefracTime": 0.0})
    for delay in (0, 1):
        sg = m.add_synapse_population(f"syn{delay}", "SPARSE", a, b, init_weight_update("StaticPulseConstantWeight", {"g": 0.1}),
                                      init_postsynaptic("ExpCurr", {"tau": 5.0}))
        sg.set_sparse_connections(np.repeat(np.arange(2368, dtype=np.uint32), 20), np.random.default_rng(delay).integers(0, 2368, 47360).astype(np.uint32))
        sg.axonal_delay_steps = delay
    rt = _runtime(resolve(m), 10)
    rt.set_option("resident_ctas", 148)         # (many CTAs, some of which read before others write)
    assert rt.counter("resident") == 1
    rt.step_time(4)
    assert rt.array("psm0.out_post").max() > 1.0 and rt.array("psm1.out_post").max() > 1.0
    rt.set_option("use_lag", 1)                 # (one of the kernels with a grid barrier; the message buffers stay)
    rt.step_time((1 << 20) - 4)
    rt.set_option("use_resident", 1)
    rt.set_option("count_events", 1)
    rt.step_time(8)
    assert rt.counter("synaptic_events") == 0
    assert rt.array("psm0.out_post").max() < 1e-30 and rt.array("psm1.out_post").max() < 1e-30
    rt.close()


def test_more_events_in_one_launch_than_32_bits_hold():
    """Every neuron of one CTA fires in every step and reaches every neuron through four groups: 4.9e9 events a warp, 1.5e8
    a lane."""
    m = GeNNModel("float", "events")
    m.dt = 1.0
    lif = {"C": 0.25, "TauM": 20.0, "Vrest": -65.0, "Vreset": -70.0, "Vthresh": -50.0, "Ioffset": 50.0, "TauRefrac": 0.0}
    n, groups, steps = 128, 4, 300000
    a = m.add_neuron_population("a", n, "LIF", lif, {"V": -40.0, "RefracTime": 0.0})
    m.fuse_postsynaptic_models = True
    for i in range(groups):
        sg = m.add_synapse_population(f"syn{i}", "BITMASK", a, a, init_weight_update("StaticPulseConstantWeight", {"g": 0.0}),
                                      init_postsynaptic("ExpCurr", {"tau": 5.0}))
        sg.set_sparse_connections(np.repeat(np.arange(n, dtype=np.uint32), n), np.tile(np.arange(n, dtype=np.uint32), n))
    rt = _runtime(resolve(m), 10)
    rt.set_option("resident_ctas", 1)
    rt.set_option("resident_warps", 4)
    assert rt.counter("resident") == 1
    rt.set_option("count_events", 1)
    rt.step_time(1)
    assert rt.counter("spikes") == n and rt.counter("synaptic_events") == 0
    before = rt.kernel_launches
    rt.step_time(steps)
    assert rt.kernel_launches == before + 1
    assert rt.counter("spikes") == n * (steps + 1)
    assert rt.counter("synaptic_events") == groups * n * n * steps
    rt.close()


def _busy(kind, synchronous):
    """Sources that fire in every step, or two populations of which one fires as a whole in some steps."""
    rng = np.random.default_rng(11)
    m = GeNNModel("float", "busy")
    m.dt, m.seed = 1.0, 23
    lif = {"C": 0.25, "TauM": 20.0, "Vrest": -65.0, "Vreset": -70.0, "Vthresh": -50.0, "Ioffset": 0.3, "TauRefrac": 2.0}
    src = m.add_neuron_population("in", 300, "Poisson", {"rate": 600.0 if synchronous else 150.0}, {"timeStepToSpike": 0.0})
    trg = m.add_neuron_population("out", 3000 if synchronous else 200, "LIF", lif,
                                  {"V": -65.0 if synchronous else rng.uniform(-65, -50, 200).astype(np.float32), "RefracTime": 0.0})
    n = trg.num_neurons
    for name, pop, delay in (("syn", src, 0), ("rec", trg, 0)) if kind != "two delays" else (("syn", src, 2), ("rec", trg, 0)):
        pre = np.repeat(np.arange(pop.num_neurons, dtype=np.uint32), 10)
        params = {"g": rng.uniform(0, 1e-5, len(pre)).astype(np.float32)}
        if kind == "rings":
            params["d"] = rng.integers(0, 6, len(pre)).astype(np.uint8)
        sg = m.add_synapse_population(name, "BITMASK" if kind == "bit mask" and pop is src else "SPARSE", pop, trg,
                                      init_weight_update("StaticPulseConstantWeight", {"g": 1e-5}) if kind == "bit mask" and pop is src else
                                      init_weight_update("StaticPulseDendriticDelay" if kind == "rings" else "StaticPulse", {}, params), init_postsynaptic("ExpCurr", {"tau": 5.0}))
        sg.set_sparse_connections(pre, rng.integers(0, n, len(pre)).astype(np.uint32))
        sg.axonal_delay_steps = 3 if kind == "late" else delay
        if kind == "rings":
            sg.max_dendritic_delay_timesteps = 6
    return m


@pytest.mark.parametrize("synchronous", [False, True], ids=["patience 0", "more than the list holds"])
@pytest.mark.parametrize("kind", ["immediate", "late", "rings", "two delays", "bit mask"])
def test_a_busy_network_is_handed_over_and_taken_back(kind, synchronous):
    """Launches that end early, the other kernel's share of their steps, and this kernel again: spikes and state of the CPU
    checker at every end of a call, also where a step that had begun is left to the other kernel."""
    from oracle.oracle import OracleRunner
    net = resolve(_busy(kind, synchronous))
    rt, orc = _runtime(net, 200), OracleRunner(resolve(_busy(kind, synchronous)), 200)
    other = _runtime(resolve(_busy(kind, synchronous)), 200)       # (the same events are counted)
    other.set_option("use_fused", 0)
    for r in (rt, other):
        r.set_option("count_events", 1)
    rt.set_option("resident_warps", 4)          # (few warps: a spike costs the more)
    assert rt.counter("resident") == 1
    rt.set_option("resident_patience", 1e6 if synchronous and kind != "bit mask" else 0)
    holds, done = set(), 0
    for n in (1, 2, 3, 5, 60, 1, 1, 40, 87):
        rt.step_time(n)
        other.step_time(n)
        orc.step(n)
        assert rt.counter("synaptic_events") == other.counter("synaptic_events") and rt.counter("spikes") == other.counter("spikes")
        done += n
        holds.add(rt.counter("resident_hold"))
        for p in net.pops:
            assert np.array_equal(np.sort(rt.current_spikes(p.name)), np.sort(orc.current_spikes(p.name))), f"step {done} {p.name}"
        helpers.assert_close(rt.array("out.V")[0], orc.array("out.V")[0], f"step {done} V", 1e-5, 5e-6)
        for i in range(len(net.psms)):
            helpers.assert_close(rt.array(f"psm{i}.out_post")[0], orc.array(f"psm{i}.out_post")[0], f"step {done} input {i}", 1e-5, 2e-6)
    if (kind, synchronous) in (("two delays", True), ("bit mask", False)):
        assert holds == {0}             # (several delays: lists are worked off one by one; too few spikes for the other path's kernels)
    elif kind == "bit mask":
        assert len(holds) >= 2, holds   # (from call to call)
    else:
        assert len(holds) >= 3, holds   # (left more than once)
    rt.close()
    other.close()
    orc.close()


def test_a_quiet_network_stays():
    net, rt, steps, _ = _resident("potjans_mini")
    for n in (1, 40, 59):
        rt.step_time(n)
    assert rt.counter("resident_hold") == 0
    rt.close()


@pytest.mark.parametrize("kind", ["immediate", "late", "rings", "two delays", "bit mask"])
def test_synapses_changed_between_calls_of_every_length(kind):
    """Weights, then rows, pushed in front of calls of one step and of many: on the other path, on a copy filled again, on a copy
    made again and in the middle of a call, the arrays are those pushed last."""
    net = resolve(_busy(kind, False))
    rt, other = _runtime(net, 10), _runtime(resolve(_busy(kind, False)), 10)
    other.set_option("use_fused", 0)
    other.set_option("use_tiled", 0)
    assert rt.counter("resident") == 1 and rt.counter("resident_builds") == 1
    rng = np.random.default_rng(5)
    g, rows = net.syn("rec").g.copy(), net.syn("rec").row_length.copy()
    for n in (1, 1, 2, 300, 1, 40, 1):
        g = (g * rng.uniform(0.2, 3.0)).astype(np.float32)
        for r in (rt, other):
            r.plan.push("rec.g", g)
            r.step_time(n)
        helpers.assert_close(rt.array("out.V")[0], other.array("out.V")[0], f"V after {n} steps", 1e-5, 5e-6)
    for i in range(len(net.psms)):
        helpers.assert_close(rt.array(f"psm{i}.out_post")[0], other.array(f"psm{i}.out_post")[0], f"input {i}", 1e-5, 2e-6)
    assert rt.counter("resident_builds") == 1, "other weights of the same synapses fill the copy where it lies"
    for n in (1, 2, 600, 1):
        rows = np.minimum(rows, rng.integers(3, 11, len(rows)).astype(np.uint32))
        for r in (rt, other):
            r.plan.push("rec.row_length", rows)
            r.step_time(n)
        helpers.assert_close(rt.array("out.V")[0], other.array("out.V")[0], f"V after {n} steps", 1e-5, 5e-6)
    assert rt.counter("resident") == 1 and 1 < rt.counter("resident_builds") <= 5
    rt.close()
    other.close()


def test_the_private_copy_goes_back_when_the_kernel_is_switched_off():
    import torch
    rng = np.random.default_rng(1)
    m = GeNNModel("float", "memory")
    m.dt = 1.0
    lif = {"C": 0.25, "TauM": 20.0, "Vrest": -65.0, "Vreset": -70.0, "Vthresh": -50.0, "Ioffset": 0.0, "TauRefrac": 2.0}
    a = m.add_neuron_population("a", 40000, "LIF", lif, {"V": -65.0, "RefracTime": 0.0})
    sg = m.add_synapse_population("syn", "SPARSE", a, a, init_weight_update("StaticPulseConstantWeight", {"g": 0.1}), init_postsynaptic("ExpCurr", {"tau": 5.0}))
    pre = np.repeat(np.arange(40000, dtype=np.uint32), 500)
    sg.set_sparse_connections(pre, rng.integers(0, 40000, len(pre)).astype(np.uint32), presorted=True)
    m.build()
    m.load()
    rt = m._runtime
    assert rt.counter("resident") == 1
    size = rt.counter("resident_bytes")
    assert 8 * len(pre) <= size <= 5 * 8 * len(pre)
    rt.synchronize()
    before = torch.cuda.mem_get_info()[0]
    rt.set_option("use_resident", 0)
    rt.step_time(5)
    rt.synchronize()
    assert rt.counter("resident_bytes") == 0
    assert torch.cuda.mem_get_info()[0] - before >= size          # (more than the pool keeps for one allocation)
    rt.set_option("use_resident", 1)
    rt.step_time(5)
    rt.synchronize()
    assert rt.counter("resident_bytes") == size
    m.unload()
