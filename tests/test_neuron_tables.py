"""GPU: the neuron update of batched networks takes the tables of up to four, in some launches up to eight populations into shared
memory and reads those of more where they lie: state and spikes of the CPU checker at both sides of each line, whatever kernel runs
before it."""
import numpy as np
import pytest

from genn_b200 import GeNNModel, init_postsynaptic, init_weight_update
from genn_b200.resolve import resolve
from tests import helpers

pytestmark = pytest.mark.gpu
LIF = {"C": 1.0, "TauM": 20.0, "Vrest": -65.0, "Vreset": -70.0, "Vthresh": -50.0, "Ioffset": 0.0, "TauRefrac": 2.0}


def _net(groups, size, batch, kind):
    rng = np.random.default_rng(groups * 100 + batch)
    m = GeNNModel("float", "tables")
    m.dt, m.seed, m.batch_size = 1.0, 5, batch
    pre, degree = 40, 9
    src = m.add_neuron_population("in", pre, "Poisson", {"rate": 200.0}, {"timeStepToSpike": 0.0})
    for i in range(groups - 1):
        n = size + 37 * i
        trg = m.add_neuron_population(f"out{i}", n, "LIF", dict(LIF, Ioffset=0.9), {"V": rng.uniform(-65, -50, n).astype(np.float32), "RefracTime": 0.0})
        if kind == "dense":
            m.add_synapse_population(f"syn{i}", "DENSE", src, trg, init_weight_update("StaticPulse", {}, {"g": rng.uniform(0, 0.02, pre * n).astype(np.float32)}),
                                     init_postsynaptic("ExpCurr", {"tau": 5.0}))
            continue
        wu = (init_weight_update("STDP", {"tauPlus": 20.0, "tauMinus": 20.0, "Aplus": 0.01, "Aminus": 0.0105, "Wmin": 0.0, "Wmax": 1.0},
                                 {"g": rng.uniform(0, 0.1, pre * degree).astype(np.float32)}) if kind == "stdp" else
              init_weight_update("StaticPulse", {}, {"g": rng.uniform(0, 0.1, pre * degree).astype(np.float32)}))
        sg = m.add_synapse_population(f"syn{i}", "SPARSE", src, trg, wu, init_postsynaptic("ExpCurr", {"tau": 5.0}))
        sg.set_sparse_connections(np.repeat(np.arange(pre, dtype=np.uint32), degree),
                                  np.concatenate([np.sort(rng.choice(n, degree, replace=False)) for _ in range(pre)]).astype(np.uint32))
    return resolve(m)


@pytest.mark.parametrize("kind", ["dense", "sparse", "stdp"])
@pytest.mark.parametrize("groups,size,batch", [(2, 33, 2), (4, 129, 3), (4, 200, 60), (5, 40, 2), (5, 70, 40), (5, 700, 40), (8, 20, 3), (8, 130, 20), (9, 20, 3)])
def test_populations_at_the_lines_of_the_rule(groups, size, batch, kind):
    from genn_b200.runtime import Runtime
    from oracle.oracle import OracleRunner
    rt, orc = Runtime(None, net=_net(groups, size, batch, kind)), OracleRunner(_net(groups, size, batch, kind))
    fired = 0
    for chunk in (1, 2, 9):
        rt.step_time(chunk)
        orc.step(chunk)
        for name in [n for n in rt.plan.arrays if n.endswith((".out_post", ".V"))]:
            helpers.assert_close(rt.array(name).reshape(-1), orc.array(name).reshape(-1), f"{name} after {chunk}", 1e-5, 2e-5)
        for p in rt.net.pops:
            for b in range(batch):
                got, want = np.sort(rt.current_spikes(p.name, b)), np.sort(orc.current_spikes(p.name, b))
                assert np.array_equal(got, want), f"{p.name} copy {b} after {chunk}"
                fired += len(want)
    assert fired > 0
    rt.close()
    orc.close()
