"""Calls on a device without room for their staging: what can be done without it is done, what cannot returns an error, and
the same call works again when there is room."""
import contextlib
import ctypes

import numpy as np
import pytest
import torch

import neuronbridge_gb300 as nb

pytestmark = pytest.mark.gpu

BLOCK = 2 << 20  # the device gives memory out in blocks of 2 MiB


@contextlib.contextmanager
def _leaving(room):
    """All of the device's memory held (none of it touched) but about `room` bytes, straight from the runtime: torch's
    allocator asks for 20 MiB at least."""
    rt = ctypes.CDLL("libcudart.so.13")
    held = []
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    try:
        size = 1 << 40
        while size >= BLOCK:
            p = ctypes.c_void_p()
            if torch.cuda.mem_get_info()[0] >= room + size and rt.cudaMalloc(ctypes.byref(p), ctypes.c_size_t(size)) == 0:
                held.append(p)
            else:
                rt.cudaGetLastError()
                size //= 2
        yield
    finally:
        for p in held:
            rt.cudaFree(p)


def _network(n, in_degree, plastic, delay=3):
    rng = np.random.default_rng(5)
    net = nb.Network()
    if plastic:
        params = {"a": 0.02, "b": 0.2, "c": -65.0, "d": 8.0, "v0": -65.0, "V_th": 30.0, "noise_sigma": 15.0}
        net.add_layer(nb.NeuronLayer("IzhikevichCurrentRK4", n, output=True,
                                     parameters={k: nb.float32(v) for k, v in params.items()}))
        net.add_learning_rule(nb.LearningRule("STDP", {"Max_LTP": nb.float32(0.1), "LTP_tau": nb.float32(20.0),
                                                       "Max_LTD": nb.float32(0.12), "LTD_tau": nb.float32(20.0)}))
    else:
        from neuronbridge_gb300.workloads import LIF_PARAMS

        net.add_layer(nb.NeuronLayer("TimeDrivenLIF_Voltage_jump", n, output=True, parameters=dict(LIF_PARAMS)))
    s = n * in_degree
    extra = {"max_weight": 10.0, "synapse_rule": 0} if plastic else {}
    net.connect(nb.Connection(rng.integers(0, n, s).astype(np.int32), np.repeat(np.arange(n, dtype=np.int32), in_degree),
                              synapse_type=0, weight=rng.random(s).astype(np.float32), delay=delay, **extra))
    return net


@pytest.mark.parametrize("plastic", [True, False])
def test_weights_without_room_for_their_staging(plastic):
    cfg = nb.SimulationConfig(steps=60, timestep=0.1)
    net = _network(50_000, 100, plastic)
    sims = [nb.Simulation(net, cfg, seed=3) for _ in range(2)]
    for s in sims:
        s.run(60)
    want = sims[0].weights()  # gathered on the device, in two chunks
    with _leaving(8 << 20):  # less than the 20 MB of the connection order
        got = sims[1].weights()
    for other in (got, sims[1].weights()):  # the second with room again
        assert want.keys() == other.keys()
        for k in want:
            assert np.array_equal(want[k], other[k]), k


def test_a_delivery_again_after_one_without_room():
    from neuronbridge_gb300 import _lib
    from neuronbridge_gb300.dense import DensePopulations, dense_weights
    from neuronbridge_gb300.workloads import LIF_PARAMS

    n = 8192
    w = dense_weights(n, seed=4)
    layer = nb.NeuronLayer("TimeDrivenLIF_Voltage_jump", 1, parameters=dict(LIF_PARAMS))
    a, b = (DensePopulations(w, layer) for _ in range(2))
    s = (np.random.default_rng(7).random((64, n)) < 0.03).astype(np.uint8)
    want = a.deliver(s)
    with _leaving(0):  # the delivery wants 7.5 MiB
        with pytest.raises(_lib.NbgError):
            b.deliver(s)
        with pytest.raises(_lib.NbgError):  # nor does it launch on what it did not get
            b.deliver(s)
    assert np.array_equal(b.deliver(s), want)


def test_a_ring_that_fits_without_its_padding():
    """In-degree 40 (two mask words a neuron, four with padding) over 4,000 steps of delay: 0.65 GB, 1.29 padded.  The network
    is created where only the former fits, and runs as with the latter."""
    cfg = nb.SimulationConfig(steps=4400, timestep=0.1)
    net = _network(20_000, 40, True, delay=4000)
    with _leaving(1 << 30):
        tight = nb.Simulation(net, cfg, seed=3)
    wide = nb.Simulation(net, cfg, seed=3)
    for s in (tight, wide):
        s.run(4400)
    assert tight.num_events == wide.num_events > 0
    for a, b in zip(tight.spike_raster(), wide.spike_raster()):
        assert len(a) > 0 and np.array_equal(a, b)
    a, b = tight.weights(), wide.weights()
    for k in a:
        assert np.array_equal(a[k], b[k]), k
