"""DENSE delivery of batched networks against the CPU checker, at the edges of its tiles: columns and sources that fill no
tile, rows of every alignment, more copies than a mask word, more sources than a CTA's window, every source at once."""
import numpy as np
import pytest

from genn_b200 import GeNNModel, init_postsynaptic, init_weight_update
from genn_b200.resolve import resolve
from tests import helpers


def _net(pre, post, batch, rate, weight):
    rng = np.random.default_rng(pre * 31 + post)
    m = GeNNModel("float", "dense_batch")
    m.dt, m.seed, m.batch_size = 1.0, 17, batch
    src = m.add_neuron_population("in", pre, "Poisson", {"rate": rate}, {"timeStepToSpike": 0.0})
    lif = {"C": 1.0, "TauM": 20.0, "Vrest": -65.0, "Vreset": -70.0, "Vthresh": -50.0, "Ioffset": 0.0, "TauRefrac": 2.0}
    trg = m.add_neuron_population("out", post, "LIF", lif, {"V": -65.0, "RefracTime": 0.0})
    wu = (init_weight_update("StaticPulseConstantWeight", {"g": 0.02}) if weight == "constant" else
          init_weight_update("StaticPulse", {}, {"g": rng.uniform(0.0, 4.0 / max(1.0, pre * rate * 1e-3), (pre, post)).astype(np.float32)}))
    sg = m.add_synapse_population("syn", "DENSE", src, trg, wu, init_postsynaptic("ExpCurr", {"tau": 5.0}))
    sg.axonal_delay_steps = 1 if batch == 5 else 0
    return resolve(m)


@pytest.mark.gpu
@pytest.mark.parametrize("pre,post,batch,rate,weight", [
    (1, 1, 2, 900.0, "drawn"), (1023, 129, 3, 100.0, "drawn"), (1024, 127, 32, 50.0, "drawn"), (2049, 260, 5, 30.0, "drawn"),
    (1070, 4, 33, 100.0, "drawn"), (5000, 130, 2, 20.0, "drawn"), (1029, 128, 8, 990.0, "drawn"), (1090, 513, 4, 100.0, "constant"),
    (1025, 1, 2, 100.0, "drawn"), (70001, 5, 3, 3.0, "drawn")])
def test_every_copy_matches_the_cpu_checker(pre, post, batch, rate, weight):
    from genn_b200.runtime import Runtime
    from oracle.oracle import OracleRunner
    rt, orc = Runtime(None, net=_net(pre, post, batch, rate, weight)), OracleRunner(_net(pre, post, batch, rate, weight))
    rt.set_option("count_events", 1)
    events = 0
    for chunk in (1, 2, 7):
        rt.step_time(chunk)
        for _ in range(chunk):
            orc.step(1)
            if batch != 5:
                events += post * sum(len(orc.current_spikes("in", b)) for b in range(batch))
        for name in ("psm0.out_post", "out.V"):
            helpers.assert_close(rt.array(name).reshape(-1), orc.array(name).reshape(-1), f"{name} after {chunk}", 1e-5, 5e-6)
    if batch != 5:
        events -= post * sum(len(orc.current_spikes("in", b)) for b in range(batch))       # (delivered by the next step)
        assert rt.counter("synaptic_events") == events
    rt.close()
    orc.close()
