"""Work that programs written against this framework have it do, as timed cases.

Every case is one pass of such a program's inner loop through the public ``GeNNModel`` interface on a
model that stays loaded from pass to pass: step it, and fetch what the program goes on with (membrane
potentials, spikes, weights).  Networks are synthetic, drawn from the case's seed; their shapes are those of
the configurations and tests of this repository (benchmark networks in ``genn_b200.workloads``) or generic.

Kinds of work:

loop         closed-loop control: one time step, then the spikes of that step and the potentials
trial        a stimulus trial: state reset by pushes, many steps driven by given spike trains, recorded spikes
bitmask      fixed binary connectivity (one bit per synapse) with one constant weight, driven by Poisson inputs
dense        a fully connected layer, one copy or a batch of copies of the dynamic state
potjans      the cortical microcircuit (current synapses, heterogeneous dendritic delays, Poisson background)
cond_ei      a balanced network of conductance synapses with an axonal delay
procedural   connectivity regenerated for every spike instead of stored
stdp         batched plasticity: learning steps, then a reduction of the weights over the batch
batch        a recurrent sparse network of given weights run for many inputs at once (batched inference)
load         what every program does first, and parameter sweeps do all the time: build, initialise, read back

A model is closed when its state is dropped (a program that builds many models has to).
"""
import math

import numpy as np

from genn_b200 import GeNNModel, init_postsynaptic, init_sparse_connectivity, init_var, init_weight_update, workloads

LIF = {"C": 0.25, "TauM": 20.0, "Vrest": -65.0, "Vreset": -70.0, "Vthresh": -50.0, "Ioffset": 0.0, "TauRefrac": 2.0}


def listed():
    return [
        # one step of a 1000-neuron Izhikevich network (100 synapses each) between reading sensors and setting motors
        {"name": "loop_1k", "kind": "loop", "neurons": 1000, "degree": 100, "steps": 1},
        # benchmark configuration 1 as trials: 1000 sources at 20 Hz, 10 000 LIF, p = 0.1, 100 ms at 0.1 ms
        {"name": "trial_1k_10k", "kind": "trial", "pre": 1000, "post": 10000, "prob": 0.1, "rate": 20.0, "steps": 1000, "narrow": False},
        # binary connectivity at sizes that fill neither words, warps nor blocks
        {"name": "bitmask_odd", "kind": "bitmask", "pre": 2003, "post": 5009, "prob": 0.1, "rate": 40.0, "steps": 100},
        # a fully connected layer of a network that runs online, one sample at a time
        {"name": "dense_online", "kind": "dense", "pre": 4096, "post": 4096, "batch": 1, "rate": 25.0, "steps": 100},
        # the 8192 x 8192 layer of the dense probe of the benchmark, 2.5 % of the inputs active, 32 samples at once
        {"name": "dense_batch", "kind": "dense", "pre": 8192, "post": 8192, "batch": 32, "rate": 25.0, "steps": 20},
        # the headline network in miniature (the usual size while a model is being developed), potentials only
        {"name": "potjans_tenth", "kind": "potjans", "scale": 0.1, "steps": 100, "record": False},
        # the headline network at full size, 10 ms a pass, spikes recorded and decoded
        {"name": "potjans_full", "kind": "potjans", "scale": 1.0, "steps": 100, "record": True},
        # benchmark configuration 2: 80 000 + 20 000 neurons, in-degree 1000, 1 ms axonal delay
        {"name": "cond_ei_full", "kind": "cond_ei", "scale": 1.0, "steps": 100},
        # benchmark configuration 4: a million neurons whose synapses would not fit many GPUs if they were stored
        {"name": "procedural_1m", "kind": "procedural", "neurons": 1000000, "degree": 1000, "threads": 32, "steps": 10},
        # benchmark configuration 5 at a size that loads quickly: 32 copies, a reduction behind every 100 steps
        {"name": "stdp_batch", "kind": "stdp", "pre": 3000, "post": 3000, "prob": 0.1, "batch": 32, "rate": 25.0, "steps": 100},
        # batched inference through a recurrent sparse network with a high input rate: many events in every step
        {"name": "batch_sparse", "kind": "batch", "neurons": 20000, "prob": 0.05, "batch": 8, "rate": 50.0, "steps": 20, "narrow": True},
        # a sweep's step: 10 M device-drawn synapses with drawn weights, built, initialised and read back
        {"name": "load_sparse", "kind": "load", "pre": 10000, "post": 10000, "prob": 0.1},
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def real(lo, hi):
        return round(math.exp(rng.uniform(math.log(lo), math.log(hi))), 4)

    kind = rng.choice(["loop", "trial", "bitmask", "dense", "potjans", "cond_ei", "procedural", "stdp", "batch", "load"])
    if kind == "loop":
        n = size(100, 20000)
        return {"kind": kind, "neurons": n, "degree": min(n, size(10, 200)), "steps": size(1, 10)}
    if kind == "trial":
        return {"kind": kind, "pre": size(100, 1500), "post": size(300, 10000), "prob": real(0.02, 0.1), "rate": real(5, 50),
                "steps": size(100, 1000), "narrow": rng.random() < 0.5}
    if kind == "bitmask":
        return {"kind": kind, "pre": size(100, 4000), "post": size(200, 10000), "prob": real(0.02, 0.2), "rate": real(10, 80),
                "steps": size(20, 100)}
    if kind == "dense":
        batch = rng.choice([1, 1, 2, 3, 5, 8, 16, 32])
        return {"kind": kind, "pre": size(200, 8192), "post": size(50, 8192), "batch": batch, "rate": real(10, 50), "steps": size(10, 20 if batch > 8 else 100)}
    if kind == "potjans":
        return {"kind": kind, "scale": real(0.03, 1.0), "steps": size(20, 100), "record": rng.random() < 0.5}
    if kind == "cond_ei":
        return {"kind": kind, "scale": real(0.05, 1.0), "steps": size(20, 100)}
    if kind == "procedural":
        return {"kind": kind, "neurons": size(20000, 1000000), "degree": size(100, 1000), "threads": rng.choice([4, 8, 16, 32]), "steps": 10}
    if kind == "stdp":
        return {"kind": kind, "pre": size(300, 3000), "post": size(200, 3000), "prob": real(0.05, 0.1), "batch": rng.choice([1, 2, 4, 8, 16, 32]),
                "rate": real(10, 40), "steps": size(20, 100)}
    if kind == "batch":
        return {"kind": kind, "neurons": size(1000, 20000), "prob": real(0.02, 0.05), "batch": rng.choice([2, 3, 4, 8]), "rate": real(10, 50),
                "steps": size(10, 20), "narrow": rng.random() < 0.5}
    return {"kind": kind, "pre": size(300, 10000), "post": size(300, 10000), "prob": real(0.02, 0.1)}


class State:
    """A loaded model and what the program's loop touches."""

    def __init__(self, case, model, **parts):
        self.case, self.model = case, model
        self.__dict__.update(parts)

    def __del__(self):
        self.model.unload()


def _weight(n_active_inputs, rate, tau, current=0.25):
    """Mean weight with which the mean input current of a neuron is `current` nA (threshold: 0.19 nA)."""
    return current / max(1e-9, n_active_inputs * rate / 1000.0 * tau)


def _ragged(rng, pre, post, prob):
    """(pre, post) pairs row by row, binomial row lengths, targets drawn with replacement."""
    counts = rng.binomial(post, prob, size=pre)
    rows = np.repeat(np.arange(pre, dtype=np.uint32), counts)
    return rows, rng.integers(0, post, size=len(rows), dtype=np.uint32)


def _poisson_to_lif(case, seed, batch, dt):
    m = GeNNModel("float", case["kind"])
    m.dt, m.seed, m.batch_size = dt, seed, batch
    src = m.add_neuron_population("input", case["pre"], "Poisson", {"rate": case["rate"]}, {"timeStepToSpike": 0.0})
    trg = m.add_neuron_population("output", case["post"], "LIF", LIF, {"V": init_var("Uniform", {"min": -65.0, "max": -52.0}), "RefracTime": 0.0})
    return m, src, trg


def _loop(case, seed):
    rng = np.random.default_rng(seed)
    n, k = case["neurons"], case["degree"]
    m = GeNNModel("float", "loop")
    m.dt = 0.5
    pop = m.add_neuron_population("izh", n, "Izhikevich", {"a": 0.02, "b": 0.2, "c": -65.0, "d": 8.0},
                                  {"V": rng.uniform(-70.0, -55.0, n).astype(np.float32), "U": -13.0})
    m.add_current_source("drive", "DC", pop, {"amp": 6.0}, {})
    sg = m.add_synapse_population("rec", "SPARSE", pop, pop,
                                  init_weight_update("StaticPulse", {}, {"g": rng.normal(0.05, 0.02, n * k).astype(np.float32)}),
                                  init_postsynaptic("DeltaCurr", {}))
    sg.set_sparse_connections(np.repeat(np.arange(n, dtype=np.uint32), k), rng.integers(0, n, size=n * k, dtype=np.uint32), presorted=True)
    m.build()
    m.load()
    return State(case, m, pop=pop)


def _trial(case, seed):
    m = workloads.feedforward(seed=seed, num_pre=case["pre"], num_post=case["post"], prob=case["prob"], rate_hz=case["rate"],
                              steps=case["steps"], narrow=case["narrow"])
    src, trg = m.neuron_populations["pre"], m.neuron_populations["post"]
    src.spike_recording_enabled = False
    start = src.vars["startSpike"].init
    m.build()
    m.load(num_recording_timesteps=case["steps"])
    sg = m.synapse_populations["syn"]
    src.vars["startSpike"].view[...] = start
    return State(case, m, src=src, trg=trg, sg=sg)


def _bitmask(case, seed):
    m, src, trg = _poisson_to_lif(case, seed, 1, 1.0)
    rng = np.random.default_rng(seed)
    w = _weight(case["pre"] * case["prob"], case["rate"], 5.0)
    sg = m.add_synapse_population("syn", "BITMASK", src, trg, init_weight_update("StaticPulseConstantWeight", {"g": w}),
                                  init_postsynaptic("ExpCurr", {"tau": 5.0}))
    sg.set_sparse_connections(*_ragged(rng, case["pre"], case["post"], case["prob"]), presorted=True)
    m.build()
    m.load()
    return State(case, m, trg=trg, sg=sg)


def _dense(case, seed):
    m, src, trg = _poisson_to_lif(case, seed, case["batch"], 1.0)
    w = _weight(case["pre"], case["rate"], 5.0)
    sg = m.add_synapse_population("syn", "DENSE", src, trg,
                                  init_weight_update("StaticPulse", {}, {"g": init_var("Uniform", {"min": 0.0, "max": 2.0 * w})}),
                                  init_postsynaptic("ExpCurr", {"tau": 5.0}))
    m.build()
    m.load()
    return State(case, m, trg=trg, sg=sg)


def _room(synapses, sources):
    """Row length that no draw of `synapses` synapses over `sources` rows exceeds."""
    mean = synapses / sources
    return int(mean + 7.0 * math.sqrt(mean) + 16.0)


def _potjans(case, seed):
    m = workloads.potjans(neuron_scale=case["scale"], seed=seed, record=case["record"])
    for sg in m.synapse_populations.values():
        sg.max_connections = _room(sg.connect.params["num"], sg.src.num_neurons)
    m.build()
    m.load(num_recording_timesteps=case["steps"] if case["record"] else None)
    return State(case, m)


def _cond_ei(case, seed):
    m = GeNNModel("float", "cond_ei")
    m.dt, m.seed = 0.1, seed
    lif = {"C": 0.2, "TauM": 20.0, "Vrest": -60.0, "Vreset": -60.0, "Vthresh": -50.0, "Ioffset": 0.35, "TauRefrac": 5.0}
    pops = [m.add_neuron_population(name, int(round(n * case["scale"])), "LIF", lif,
                                    {"V": init_var("Uniform", {"min": -60.0, "max": -50.0}), "RefracTime": 0.0})
            for name, n in (("E", 80000), ("I", 20000))]
    for src, w, tau, erev, degree in ((pops[0], 0.6e-3, 5.0, 0.0, 800), (pops[1], 6.7e-3, 10.0, -80.0, 200)):
        for trg in pops:
            sg = m.add_synapse_population(src.name + trg.name, "SPARSE", src, trg, init_weight_update("StaticPulseConstantWeight", {"g": w}),
                                          init_postsynaptic("ExpCond", {"tau": tau, "E": erev}),
                                          init_sparse_connectivity("FixedNumberPreWithReplacement", {"num": degree}))
            sg.axonal_delay_steps = 10
            sg.max_connections = _room(degree * trg.num_neurons, src.num_neurons)
    m.build()
    m.load()
    return State(case, m)


def _procedural(case, seed):
    n = case["neurons"]
    m = workloads.procedural_stress(num_neurons=n, prob=case["degree"] / n, threads_per_spike=case["threads"], seed=seed)
    m.build()
    m.load()
    m.step_time(100)        # past the start of the run, in which almost nothing fires
    return State(case, m)


def _stdp(case, seed):
    rng = np.random.default_rng(seed)
    m = GeNNModel("float", "stdp")
    m.dt, m.seed, m.batch_size = 1.0, seed, case["batch"]
    src = m.add_neuron_population("input", case["pre"], "Poisson", {"rate": case["rate"]}, {"timeStepToSpike": 0.0})
    lif = dict(LIF, C=0.04 * case["pre"] * case["prob"], Vthresh=-55.0)      # outputs at tens of Hz (workloads.batched_stdp)
    trg = m.add_neuron_population("output", case["post"], "LIF", lif, {"V": init_var("Uniform", {"min": -70.0, "max": -56.0}), "RefracTime": 0.0})
    # every input reaches the same number of outputs
    pre = np.repeat(np.arange(case["pre"], dtype=np.uint32), max(1, int(round(case["post"] * case["prob"]))))
    post = rng.integers(0, case["post"], size=len(pre), dtype=np.uint32)
    g = rng.random(len(pre), dtype=np.float32) * np.float32(0.5)
    sg = m.add_synapse_population("syn", "SPARSE", src, trg,
                                  init_weight_update("STDP", {"tauPlus": 20.0, "tauMinus": 20.0, "Aplus": 0.01, "Aminus": 0.0105,
                                                              "Wmin": 0.0, "Wmax": 1.0}, {"g": g}), init_postsynaptic("ExpCurr", {"tau": 5.0}))
    sg.set_sparse_connections(pre, post, presorted=True)
    m.add_custom_update("mean_g", "gradient", "SUM", (sg, "g"), broadcast=True, scale=1.0 / case["batch"])
    m.build()
    m.load()
    return State(case, m, trg=trg, reduced=m.custom_updates["mean_g"].vars["reduction"])


def _batch(case, seed):
    n = case["neurons"]
    m = GeNNModel("float", "batch")
    m.dt, m.seed, m.batch_size = 1.0, seed, case["batch"]
    m.fuse_postsynaptic_models = True
    m.default_narrow_sparse_ind_enabled = case["narrow"]
    src = m.add_neuron_population("input", n, "Poisson", {"rate": case["rate"]}, {"timeStepToSpike": 0.0})
    trg = m.add_neuron_population("hidden", n, "LIF", LIF, {"V": init_var("Uniform", {"min": -65.0, "max": -52.0}), "RefracTime": 0.0})
    w = _weight(n * case["prob"], case["rate"], 5.0)
    for name, a, mean in (("in", src, w), ("rec", trg, -0.1 * w)):
        m.add_synapse_population(name, "SPARSE", a, trg, init_weight_update("StaticPulse", {}, {"g": init_var("Normal", {"mean": mean, "sd": 0.2 * w})}),
                                 init_postsynaptic("ExpCurr", {"tau": 5.0}), init_sparse_connectivity("FixedProbability", {"prob": case["prob"]}))
    m.build()
    m.load()
    return State(case, m, trg=trg)


class LoadState:
    def __init__(self, case, seed):
        self.case, self.seed = case, seed


PREPARE = {"loop": _loop, "trial": _trial, "bitmask": _bitmask, "dense": _dense, "potjans": _potjans, "cond_ei": _cond_ei,
           "procedural": _procedural, "stdp": _stdp, "batch": _batch, "load": LoadState}


def prepare(case, seed):
    return PREPARE[case["kind"]](case, seed)


def _potentials(model):
    """Every population's membrane potentials, fetched into the model's host copies."""
    out = {}
    for p in model.neuron_populations.values():
        if "V" in p.vars:
            p.vars["V"].pull_from_device()
            out["V_" + p.name] = p.vars["V"].view
    return out


def _counts(pop):
    """Spikes of every neuron in the recorded steps: the rates a program decodes.  (Lists of spikes have no fixed length;
    when each one came is in the potentials that are returned with the counts.)"""
    times, ids = pop.spike_recording_data[0]
    return np.bincount(ids, minlength=pop.num_neurons)


def _run_loop(s):
    s.model.step_time(s.case["steps"])
    fired = np.zeros(s.case["neurons"], dtype=np.uint8)
    fired[s.pop.current_spikes] = 1
    return dict(_potentials(s.model), fired=fired)


def _run_procedural(s):
    s.model.step_time(s.case["steps"])
    out = _potentials(s.model)
    for name, sg in s.model.synapse_populations.items():
        sg.out_post.pull_from_device()
        out["current_" + name] = sg.out_post.view
    return out


def _run_trial(s):
    # back to rest, first spike of every train next, clock at zero
    s.src.vars["startSpike"].push_to_device()
    v, r = s.trg.vars["V"], s.trg.vars["RefracTime"]
    v.view[...] = -65.0
    r.view[...] = 0.0
    s.sg.out_post.view[...] = 0.0
    v.push_to_device()
    r.push_to_device()
    s.sg.out_post.push_to_device()
    s.model.timestep = 0
    s.model.step_time(s.case["steps"])
    s.model.pull_recording_buffers_from_device()
    s.sg.out_post.pull_from_device()
    return dict(_potentials(s.model), current=s.sg.out_post.view, spikes=_counts(s.trg))


def _run_layer(s):
    s.model.step_time(s.case["steps"])
    s.sg.out_post.pull_from_device()
    return dict(_potentials(s.model), current=s.sg.out_post.view)


def _run_network(s):
    s.model.step_time(s.case["steps"])
    if not s.case.get("record"):
        return _potentials(s.model)
    s.model.pull_recording_buffers_from_device()
    out = _potentials(s.model)
    for p in s.model.neuron_populations.values():
        out["spikes_" + p.name] = _counts(p)
    return out


def _run_stdp(s):
    s.model.step_time(s.case["steps"])
    s.model.custom_update("gradient")
    s.reduced.pull_from_device()
    return dict(_potentials(s.model), weights=s.reduced.view)


def _run_load(s):
    case = s.case
    m = GeNNModel("float", "load")
    m.dt, m.seed = 0.1, s.seed
    m.default_narrow_sparse_ind_enabled = True
    pops = [m.add_neuron_population(name, n, "LIF", LIF, {"V": init_var("Normal", {"mean": -58.0, "sd": 5.0}), "RefracTime": 0.0})
            for name, n in (("a", case["pre"]), ("b", case["post"]))]
    sg = m.add_synapse_population("ab", "SPARSE", pops[0], pops[1],
                                  init_weight_update("StaticPulse", {}, {"g": init_var("NormalClipped", {"mean": 0.1, "sd": 0.05, "min": 0.0, "max": 1.0})}),
                                  init_postsynaptic("ExpCurr", {"tau": 5.0}), init_sparse_connectivity("FixedProbability", {"prob": case["prob"]}))
    m.build()
    m.load()
    sg.pull_connectivity_from_device()
    sg.vars["g"].pull_from_device()
    out = dict(_potentials(m), row_lengths=sg.row_lengths, ind=sg.ind, g=sg.vars["g"].view)
    m.unload()
    return out


RUN = {"loop": _run_loop, "trial": _run_trial, "bitmask": _run_layer, "dense": _run_layer, "potjans": _run_network, "cond_ei": _run_network,
       "procedural": _run_procedural, "stdp": _run_stdp, "batch": _run_network, "load": _run_load}


def run(state):
    return RUN[state.case["kind"]](state)


def work(case):
    """Bytes: each synapse that a spike reaches (index, weight, delay as stored), neuron state read and written once a pass.
    Arithmetic: an addition per synaptic event, about 20 operations per neuron and step, and for regenerated or drawn
    synapses about 200 (a share of a Philox block for the gap, one for the weight, a logarithm each, sine and root)."""
    kind, steps = case["kind"], case.get("steps", 1)
    drawn = 0
    if kind == "loop":
        n = case["neurons"]
        events, per_event = 0.005 * n * case["degree"] * steps, 8       # about 10 Hz at 0.5 ms
    elif kind == "trial":
        n = case["pre"] + case["post"]
        events, per_event = case["pre"] * case["rate"] * steps * 1e-4 * case["post"] * case["prob"], 6 if case["narrow"] else 8
    elif kind == "bitmask":
        n = case["pre"] + case["post"]
        events, per_event = case["pre"] * case["rate"] * steps * 1e-3 * case["post"], 0.125
    elif kind == "dense":
        n = (case["pre"] + case["post"]) * case["batch"]
        # a row that several copies need in a step has to be read once
        p = case["rate"] * 1e-3
        rows = case["pre"] * (1.0 - (1.0 - p) ** case["batch"])
        events, per_event = case["pre"] * p * case["batch"] * steps * case["post"], 4.0 * rows / (case["pre"] * p * case["batch"])
    elif kind == "potjans":
        n = sum(int(round(case["scale"] * v)) for v in workloads.POTJANS_NUM.values())
        events, per_event = n * 3.2e-4 * steps * 3870, 7                # about 3.2 Hz at 0.1 ms
    elif kind == "cond_ei":
        n = int(round(100000 * case["scale"]))
        events, per_event = n * 3.0e-4 * steps * 1000, 4                # about 3 Hz at 0.1 ms
    elif kind == "procedural":
        n = case["neurons"]
        events, per_event = n * 0.16 * steps * case["degree"], 0        # as fast as the refractory period allows
        drawn = events
    elif kind == "stdp":
        n = (case["pre"] + case["post"]) * case["batch"]
        synapses = case["pre"] * case["post"] * case["prob"]
        # before-spikes at the input rate (index, weight read and written), after-spikes at about 30 Hz (remap, weight read
        # and written), the reduction over the batch with its write-back
        events, per_event = synapses * case["batch"] * steps * 1e-3 * (case["rate"] + 30.0), 12
        return {"bytes": events * per_event + synapses * (8.0 * case["batch"] + 4.0) + 48.0 * n, "flops": 8.0 * events + synapses * case["batch"] + 20.0 * n * steps}
    elif kind == "batch":
        n = 2 * case["neurons"] * case["batch"]
        fire = case["rate"] * 1e-3
        events = case["neurons"] * case["batch"] * steps * (fire + 0.02) * case["neurons"] * case["prob"]
        # synapse data that several copies need in a step has to be read once
        share = (1.0 - (1.0 - fire) ** case["batch"]) / (fire * case["batch"])
        per_event = (6.0 if case["narrow"] else 8.0) * share
    else:
        n = case["pre"] + case["post"]
        synapses = case["pre"] * case["post"] * case["prob"]
        return {"bytes": 6.0 * synapses + 8.0 * n, "flops": 200.0 * synapses}
    return {"bytes": events * per_event + 48.0 * n, "flops": events + 200.0 * drawn + 20.0 * n * steps}


def tolerance(case):
    """Drawn and stored values are the same bits for every correct implementation.  State sums fp32 inputs in no fixed order
    (about 1e-5), and a potential that stands that close to threshold may cross it a step earlier or later: a neuron or two
    in tens of thousands are then a whole spike apart (20 mV of 60), and so are, for a few steps, the neurons it reaches."""
    if case["kind"] == "load":
        return "exact"
    return {"rel": 3e-3, "max": 0.6, "differ": 2e-3}
