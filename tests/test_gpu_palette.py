"""Static networks with few different weights (codes beside the arrival bits) and with many (records) run the same
dynamics: bit for bit the CPU oracle, for 1 to 6 different (weight, type) pairs, both semantics, in-degrees around the
words of 32 and the quads of four words, and across weights set between run calls."""
import numpy as np
import pytest

import neuronbridge_gb300 as nb
from neuronbridge_gb300 import NetworkDescription, NeuronLayer
from neuronbridge_gb300.workloads import LIF_PARAMS

pytestmark = pytest.mark.gpu


def _network(weights, in_degree, n=70, seed=0, poisson_in=False):
    """n LIF under Poisson drive with `in_degree` recurrent inputs each; synapse k has weights[k % len] (type 1 where
    negative).  poisson_in: the Poisson layer has an input, so it is no generator and is updated like any neuron."""
    rng = np.random.default_rng(seed)
    tgt = np.repeat(np.arange(n, dtype=np.int32), in_degree)
    src = rng.integers(0, n, len(tgt)).astype(np.int32)
    w = np.resize(np.asarray(weights, np.float32), len(tgt))[rng.permutation(len(tgt))]
    ids = np.arange(n, dtype=np.int32)
    s, t = [src, ids + n], [tgt, ids]
    ws, ty, d = [np.abs(w), np.full(n, abs(weights[0]), np.float32)], [(w < 0).astype(np.int32), np.zeros(n, np.int32)], \
        [rng.integers(4, 9, len(tgt)).astype(np.int32), np.ones(n, np.int32)]
    if poisson_in:
        s.append(ids), t.append(ids + n), ws.append(np.full(n, abs(weights[0]), np.float32))
        ty.append(np.zeros(n, np.int32)), d.append(np.full(n, 5, np.int32))
    layers = [NeuronLayer("TimeDrivenLIF_Voltage_jump", n, output=True, parameters=dict(LIF_PARAMS)),
              NeuronLayer.poisson_rate(n, rate_bias_hz=9000.0, rate_gain_hz_per_current=0.0)]
    cat = [np.concatenate(x) for x in (s, t, ty, ws, d)]
    return NetworkDescription.from_arrays(layers, cat[0], cat[1], cat[2], cat[3], delay=cat[4])


def _check(sim, ref):
    t, i = sim.spike_raster()
    ot, oi = ref.spikes()
    keep = oi < 70  # the output layer
    ot, oi = ot[keep], oi[keep]
    order = np.lexsort((oi, ot))
    assert len(t) > 0 and np.array_equal(t, ot[order]) and np.array_equal(i, oi[order])
    assert np.array_equal(sim.state_field(0), ref.state(0).astype(np.float32))
    assert sim.num_events == ref.num_events


@pytest.mark.parametrize("semantics", ["legacy_cpu", "dense"])
@pytest.mark.parametrize("poisson_in", [False, True])
@pytest.mark.parametrize("weights", [(0.5,), (0.5, -2.5), (0.5, -0.5, 0.3), (0.51, 0.23, -1.7, -0.51),
                                     (0.5, 0.4, 0.3, -0.5, -0.4, -0.3)])
@pytest.mark.parametrize("in_degree", [3, 33, 127, 128, 140])
def test_networks_equal_the_oracle(oracle_lib, weights, in_degree, poisson_in, semantics):
    import oracle

    d = _network(weights, in_degree, poisson_in=poisson_in)
    cfg = nb.SimulationConfig(steps=300, timestep=0.1)
    sim = nb.Simulation(d, cfg, semantics=semantics)
    sim.run(300)
    ref = oracle.OracleNet(sim.flat)
    ref.run(300)
    _check(sim, ref)


def test_weights_set_between_calls():
    """A network that starts with two pairs gets a third, a fourth and a fifth, then two again by load of all weights:
    after every change it equals a fresh network with those weights."""
    d = _network((0.5, -2.5), 40)
    cfg = nb.SimulationConfig(steps=100, timestep=0.1)
    sim = nb.Simulation(d, cfg)
    sim.run(100)
    w = d.weight.copy()
    rng = np.random.default_rng(3)
    for value in (0.5, 0.7, 2.5, 0.9, 1.1, 0.7):
        for c in rng.integers(0, len(w), 25):
            sim.set_connection_weight(int(c), value)
            w[c] = value
        _same_as_fresh(sim, d, w, cfg)
    w = np.resize(np.asarray([0.25, 1.5], np.float32), len(w))
    _set_all(sim, w)
    _same_as_fresh(sim, d, w, cfg)


def _set_all(sim, w):
    import ctypes
    from neuronbridge_gb300 import _lib

    w = np.ascontiguousarray(w, np.float32)
    _lib.check(sim.lib.nbg_set_weights(sim._h, w.ctypes.data_as(ctypes.POINTER(ctypes.c_float))))


def test_arrivals_pending_when_the_palette_is_left_and_taken_up_again():
    """Weights that end the palette, and weights that bring it back, between run calls: the arrivals in the delay ring
    are delivered all the same (a network without a palette from the start is the reference)."""
    d = _network((0.5, -2.5), 40)
    cfg = nb.SimulationConfig(steps=50, timestep=0.1)
    few = np.resize(np.asarray([0.5, 2.5, 0.7], np.float32), len(d.weight))
    many = np.resize(np.linspace(0.3, 2.5, 9, dtype=np.float32), len(d.weight))
    sim, ref = nb.Simulation(d, cfg), nb.Simulation(d, cfg, event_log_capacity=1 << 20)  # a log: no palette
    for k, w in enumerate((None, many, few, many)):
        for s in (sim, ref):
            if w is not None:
                _set_all(s, w)
            s.run(50 if k else 300)
    for a, b in zip(sim.spike_raster(), ref.spike_raster()):
        assert len(a) > 0 and np.array_equal(a, b)
    assert np.array_equal(sim.state_field(0), ref.state_field(0)) and sim.num_events == ref.num_events


def _same_as_fresh(sim, d, w, cfg):
    sim.reset()
    sim.run(100)
    other = _network((0.5, -2.5), 40)
    other.weight = w.copy()
    fresh = nb.Simulation(other, cfg)
    fresh.run(100)
    for a, b in zip(sim.spike_raster(), fresh.spike_raster()):
        assert np.array_equal(a, b)
    assert np.array_equal(sim.state_field(0), fresh.state_field(0)) and np.array_equal(sim.weights()["weight"], w)


@pytest.mark.parametrize("inputs,in_degree", [(2, 200), (8, 248), (9, 100), (5, 300), (8, 1100), (40, 100), (300, 20), (784, 0)])
def test_many_generator_inputs_equal_the_oracle(oracle_lib, inputs, in_degree):
    """Several Poisson inputs a neuron in every quad of its mask words (their ranks are mixed with the recurrent ones'), on
    both sides of the rules that choose quads: 8 words or more than 32, 8 inputs."""
    import oracle

    n = 70
    rng = np.random.default_rng(inputs)
    tgt = np.repeat(np.arange(n, dtype=np.int32), in_degree)
    src = rng.integers(0, n, len(tgt)).astype(np.int32)
    gsrc = (n + np.tile(np.arange(inputs), n)).astype(np.int32)
    gtgt = np.repeat(np.arange(n, dtype=np.int32), inputs)
    order = rng.permutation(len(tgt) + len(gtgt))
    layers = [NeuronLayer("TimeDrivenLIF_Voltage_jump", n, output=True, parameters=dict(LIF_PARAMS)),
              NeuronLayer.poisson_rate(inputs, rate_bias_hz=9000.0 / inputs, rate_gain_hz_per_current=0.0)]
    w = np.concatenate([np.resize(np.asarray([0.3, 0.2], np.float32), len(tgt)), np.full(len(gtgt), 0.5, np.float32)])
    delay = np.concatenate([rng.integers(4, 9, len(tgt)), rng.integers(1, 4, len(gtgt))]).astype(np.int32)
    d = NetworkDescription.from_arrays(layers, np.concatenate([src, gsrc])[order], np.concatenate([tgt, gtgt])[order],
                                       np.zeros(len(order), np.int32), w[order], delay=delay[order])
    sim = nb.Simulation(d, nb.SimulationConfig(steps=300, timestep=0.1))
    sim.run(300)
    ref = oracle.OracleNet(sim.flat)
    ref.run(300)
    _check(sim, ref)
