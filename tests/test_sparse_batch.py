"""SPARSE delivery of batched networks against the CPU checker, at the edges of its rows and buffers: odd sizes, rows shorter
than a lane's four synapses and longer than a piece, every index width, rings of delays, constant weights, several groups
onto one buffer and several buffers, shares with few and with many events."""
import numpy as np
import pytest

from genn_b200 import GeNNModel, init_postsynaptic, init_weight_update
from genn_b200.resolve import resolve
from tests import helpers

LIF = {"C": 1.0, "TauM": 20.0, "Vrest": -65.0, "Vreset": -70.0, "Vthresh": -50.0, "Ioffset": 0.0, "TauRefrac": 2.0}


def _net(pre, post, degree, batch, rate, narrow, delays, constant):
    rng = np.random.default_rng(pre * 31 + post)
    m = GeNNModel("float", "sparse_batch")
    m.dt, m.seed, m.batch_size = 1.0, 17, batch
    m.fuse_postsynaptic_models = True
    m.default_narrow_sparse_ind_enabled = narrow
    src = m.add_neuron_population("in", pre, "Poisson", {"rate": rate}, {"timeStepToSpike": 0.0})
    trgs = [m.add_neuron_population(f"out{i}", post + 7 * i, "LIF", LIF, {"V": -65.0, "RefracTime": 0.0}) for i in range(2)]
    for i, trg in enumerate(trgs):
        n = post + 7 * i
        for part in range(2):       # two groups onto one buffer
            lengths = rng.integers(0, min(n, 2 * degree) + 1, pre)
            lengths[0], lengths[-1] = 0, min(n, 2 * degree)
            pres = np.repeat(np.arange(pre), lengths)
            posts = np.concatenate([np.sort(rng.choice(n, k, replace=False)) for k in lengths]).astype(np.uint32)
            params = {} if constant else {"g": rng.uniform(0.0, 4.0 / max(1.0, pre * rate * 1e-3 * degree / n), len(pres)).astype(np.float32)}
            if delays:
                params["d"] = rng.integers(0, delays, len(pres)).astype(np.uint8)
                wu = init_weight_update("StaticPulseDendriticDelay", {}, params)
            else:
                wu = init_weight_update("StaticPulseConstantWeight", {"g": 1.0 / 64.0}) if constant else init_weight_update("StaticPulse", {}, params)
            sg = m.add_synapse_population(f"syn{i}{part}", "SPARSE", src, trg, wu, init_postsynaptic("ExpCurr", {"tau": 5.0}))
            sg.set_sparse_connections(pres, posts)
            if delays:
                sg.max_dendritic_delay_timesteps = delays
    return resolve(m)


@pytest.mark.gpu
@pytest.mark.parametrize("pre,post,degree,batch,rate,narrow,delays,constant", [
    (5, 3, 1, 2, 500.0, False, 0, False), (301, 250, 30, 3, 50.0, True, 0, False), (97, 5003, 700, 2, 40.0, True, 0, False),
    (2000, 1501, 400, 2, 300.0, False, 0, False), (129, 300, 60, 9, 90.0, True, 5, False), (700, 257, 90, 2, 900.0, True, 0, True)])
def test_every_copy_matches_the_cpu_checker(pre, post, degree, batch, rate, narrow, delays, constant):
    from genn_b200.runtime import Runtime
    from oracle.oracle import OracleRunner
    args = (pre, post, degree, batch, rate, narrow, delays, constant)
    rt, orc = Runtime(None, net=_net(*args)), OracleRunner(_net(*args))
    for chunk in (1, 2, 6):
        rt.step_time(chunk)
        orc.step(chunk)
        for name in [n for n in rt.plan.arrays if n.endswith((".out_post", ".den_delay", ".V"))]:
            helpers.assert_close(rt.array(name).reshape(-1), orc.array(name).reshape(-1), f"{name} after {chunk}", 1e-5, 2e-5)
    assert rt.counter("tiled_ready") == 0
    rt.close()
    orc.close()


@pytest.mark.gpu
@pytest.mark.parametrize("least", [0, 1e9], ids=["shared sums", "row by row"])
@pytest.mark.parametrize("pre,post,degree,batch,rate,narrow,delays,constant", [
    (5, 3, 1, 2, 500.0, False, 0, False), (301, 250, 30, 3, 50.0, True, 0, False), (97, 5003, 700, 2, 40.0, True, 0, False),
    (129, 300, 60, 9, 90.0, True, 5, False), (700, 257, 90, 2, 900.0, True, 0, True)])
def test_either_kernel_matches_the_cpu_checker(pre, post, degree, batch, rate, narrow, delays, constant, least):
    from genn_b200.runtime import Runtime
    from oracle.oracle import OracleRunner
    args = (pre, post, degree, batch, rate, narrow, delays, constant)
    rt, orc = Runtime(None, net=_net(*args)), OracleRunner(_net(*args))
    rt.set_option("scatter_min_spikes", least)
    for chunk in (1, 2, 6):
        assert rt.counter("scatter_armed") == (1 if least == 0 else 0)
        rt.step_time(chunk)
        orc.step(chunk)
        for name in [n for n in rt.plan.arrays if n.endswith((".out_post", ".den_delay", ".V"))]:
            helpers.assert_close(rt.array(name).reshape(-1), orc.array(name).reshape(-1), f"{name} after {chunk}", 1e-5, 2e-5)
    rt.close()
    orc.close()


@pytest.mark.gpu
@pytest.mark.parametrize("pre,rate,armed", [(400, 20.0, 0), (400, 400.0, 1), (4000, 2.0, 0), (4000, 50.0, 1)])
@pytest.mark.parametrize("calls", [[600], [70] * 8])
def test_the_kernel_is_chosen_by_the_spikes_of_the_steps_before(pre, rate, armed, calls):
    """Whatever is assumed of a model at first: one long call, in which the choice may change, or several short ones."""
    from genn_b200.runtime import Runtime
    from oracle.oracle import OracleRunner
    args = (pre, 100, 10, 2, rate, True, 0, False)
    rt, orc = Runtime(None, net=_net(*args)), OracleRunner(_net(*args))
    assert rt.counter("scatter_armed") == (1 if pre == 4000 else 0)
    for n in calls:
        rt.step_time(n)
        rt.synchronize()
        orc.step(n)
    assert rt.counter("scatter_armed") == armed or (len(calls) == 1 and pre == 4000 and not armed)      # (three quiet blocks)
    for name in [n for n in rt.plan.arrays if n.endswith((".out_post", ".V"))]:
        helpers.assert_close(rt.array(name).reshape(-1), orc.array(name).reshape(-1), name, 1e-5, 5e-5)
    rt.close()
    orc.close()
