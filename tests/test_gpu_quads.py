"""Plastic networks in quads of mask words (in-degree up to 128) and beside them (more, or mostly one word),
bit for bit the CPU oracle: raster, state, weights and traces; noisy Izhikevich neurons with few arrivals, and LIF
neurons with many, from recurrent synapses, Poisson generators and external spikes."""
import numpy as np
import pytest

import neuronbridge_gb300 as nb
from neuronbridge_gb300 import LearningRule, NetworkDescription, NeuronLayer, float32
from neuronbridge_gb300.workloads import LIF_PARAMS

pytestmark = pytest.mark.gpu

RULE = LearningRule("STDP", {"Max_LTP": float32(0.05), "LTP_tau": float32(16.8), "Max_LTD": float32(0.06),
                             "LTD_tau": float32(33.1)})


def _izhikevich(in_degree, n=90):
    rng = np.random.default_rng(in_degree)
    p = {"a": float32(0.02), "b": float32(0.2), "c": float32(-65.0), "d": float32(8.0), "v0": float32(-65.0),
         "V_th": float32(30.0), "noise_sigma": float32(25.0)}
    tgt = np.repeat(np.arange(n, dtype=np.int32), in_degree)
    src = rng.integers(0, n, len(tgt)).astype(np.int32)
    inh = src >= 0.8 * n
    return NetworkDescription.from_arrays(
        [NeuronLayer("IzhikevichCurrentRK4", n, output=True, parameters=p)], src, tgt, inh.astype(np.int32),
        np.where(inh, 5.0, 6.0 * 30 / in_degree).astype(np.float32), max_weight=np.full(len(tgt), 10.0, np.float32),
        delay=rng.integers(3, 20, len(tgt)).astype(np.int32), synapse_rule=np.where(inh, -1, 0).astype(np.int32),
        rules=[RULE])


def _lif(in_degree, n=90, n_in=20):
    """External spikes and a Poisson generator per neuron besides in_degree - 3 recurrent inputs."""
    rng = np.random.default_rng(in_degree)
    ids = np.arange(n, dtype=np.int32)
    tgt = np.repeat(ids, in_degree - 3)
    src = rng.integers(0, n, len(tgt)).astype(np.int32)
    ext = rng.integers(0, n_in, 2 * n).astype(np.int32)
    layers = [NeuronLayer("TimeDrivenLIF_Voltage_jump", n, output=True, parameters=dict(LIF_PARAMS)),
              NeuronLayer.poisson_rate(n, rate_bias_hz=9000.0, rate_gain_hz_per_current=0.0),
              NeuronLayer.input_spike(n_in)]
    s, t = np.concatenate([src, ids + n, ext + 2 * n]), np.concatenate([tgt, ids, np.repeat(ids, 2)])
    w = np.concatenate([rng.random(len(src)) * 0.5, np.full(n, 0.5), np.full(2 * n, 3.0)]).astype(np.float32)
    inh = (s < n) & (s >= 0.8 * n)
    return NetworkDescription.from_arrays(
        layers, s, t, inh.astype(np.int32), w, max_weight=np.full(len(s), 4.0, np.float32),
        delay=np.concatenate([rng.integers(4, 12, len(src)), np.ones(n), rng.integers(4, 9, 2 * n)]).astype(np.int32),
        synapse_rule=np.where(inh | ((s >= n) & (s < 2 * n)), -1, 0).astype(np.int32), rules=[RULE])


@pytest.mark.parametrize("model", ["izhikevich", "lif"])
@pytest.mark.parametrize("in_degree", [5, 32, 33, 64, 96, 97, 127, 128, 129, 160])
@pytest.mark.parametrize("threads,block_steps", [(256, 0), (32, 2)])
def test_plastic_networks_equal_the_oracle(oracle_lib, model, in_degree, threads, block_steps):
    import oracle

    d = _izhikevich(in_degree) if model == "izhikevich" else _lif(in_degree)
    cfg = nb.SimulationConfig(steps=200, timestep=0.1)
    sim = nb.Simulation(d, cfg, seed=3, threads_per_block=threads, block_steps=block_steps)
    ref = oracle.OracleNet(sim.flat)
    if model == "lif":
        rng = np.random.default_rng(1)
        when, who = np.nonzero(rng.random((300, 20)) < 0.05)
        sim.add_external_spikes(when, who + 180)
        ref.add_external_spikes(when, who + 180)
    sim.run(200).run(100)
    ref.run(300)
    t, i = sim.spike_raster()
    ot, oi = ref.spikes()
    keep = oi < 90
    ot, oi = ot[keep], oi[keep]
    order = np.lexsort((oi, ot))
    assert len(t) > 0 and np.array_equal(t, ot[order]) and np.array_equal(i, oi[order])
    assert np.array_equal(sim.state_field(0), ref.state(0).astype(np.float32))
    assert sim.num_events == ref.num_events
    for a, b in zip(sim.weights().values(), ref.weights()):
        assert np.array_equal(a, b.astype(a.dtype))
