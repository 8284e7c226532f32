"""The two-phase regeneration of fixed-probability rows against the same rows stored by the initialisation kernels: sub-rows
that overrun what a lane holds, sub-rows shared by fewer lanes than threads, empty ones, targets that divide into no equal
ranges, no autapses, Normal weights and the other draws, batches."""
import numpy as np
import pytest

from genn_b200 import GeNNModel, init_postsynaptic, init_sparse_connectivity, init_var, init_weight_update
from genn_b200.resolve import resolve
from tests import helpers

NORMAL = init_var("Normal", {"mean": 0.01, "sd": 0.004})
UNIFORM = init_var("Uniform", {"min": 0.0, "max": 0.02})


def _net(matrix, n, prob, threads, weights, snippet, batch):
    m = GeNNModel("float", "rows")
    m.dt, m.seed, m.batch_size = 1.0, 91, batch
    lif = {"C": 0.25, "TauM": 20.0, "Vrest": -65.0, "Vreset": -70.0, "Vthresh": -50.0, "Ioffset": 0.0, "TauRefrac": 2.0}
    start = np.random.default_rng(3).uniform(-70.0, -48.0, n).astype(np.float32)       # some fire at once
    pop = m.add_neuron_population("pop", n, "LIF", lif, {"V": start, "RefracTime": 0.0})
    sg = m.add_synapse_population("syn", matrix, pop, pop, init_weight_update("StaticPulse", {}, {"g": weights}),
                                  init_postsynaptic("ExpCurr", {"tau": 5.0}), init_sparse_connectivity(snippet, {"prob": prob}))
    sg.num_threads_per_spike = threads
    return resolve(m)


@pytest.mark.gpu
@pytest.mark.parametrize("n,prob,threads,weights,snippet,batch", [
    (701, 0.3, 1, NORMAL, "FixedProbability", 1), (1501, 0.2, 4, NORMAL, "FixedProbabilityNoAutapse", 1),
    (1503, 0.02, 32, NORMAL, "FixedProbability", 2), (20011, 0.0005, 16, NORMAL, "FixedProbability", 1),
    (20011, 0.002, 32, UNIFORM, "FixedProbabilityNoAutapse", 1), (33, 0.9, 32, NORMAL, "FixedProbability", 3), (1, 0.5, 8, UNIFORM, "FixedProbability", 1)])
def test_regenerated_rows_are_the_stored_ones(n, prob, threads, weights, snippet, batch):
    from genn_b200.runtime import Runtime
    runs = [Runtime(None, net=_net(matrix, n, prob, threads, weights, snippet, batch)) for matrix in ("PROCEDURAL", "SPARSE")]
    for rt in runs:
        rt.set_option("use_fused", 0)
        rt.set_option("count_events", 1)
        rt.step_time(12)
    got, want = ({name: rt.array(name).reshape(-1) for name in ("psm0.out_post", "pop.V")} for rt in runs)
    for name in got:
        helpers.assert_close(got[name], want[name], name, 1e-5, 1e-4)
    assert runs[0].counter("synaptic_events") == runs[1].counter("synaptic_events")
    assert n < 100 or runs[0].counter("synaptic_events") > 0
    for rt in runs:
        rt.close()
