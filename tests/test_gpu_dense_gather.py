"""The FP32 dense path (k_dense_gather: spikes ranked into a list, two columns a thread, delivery and update in one
launch) at the edges of its column slices and word chunks, bit for bit: the delivery is the sequential float sum over the
ascending spikes, and steps of the engine equal the CPU oracle."""
import numpy as np
import pytest
import torch

from neuronbridge_gb300 import NeuronLayer
from neuronbridge_gb300.dense import DensePopulations
from neuronbridge_gb300.workloads import LIF_PARAMS

pytestmark = pytest.mark.gpu


def _weights(n):
    g = torch.Generator(device="cuda").manual_seed(n)
    return (torch.randn(n, n, generator=g, device="cuda") / n ** 0.5).cpu().numpy()


def _layer():
    return NeuronLayer("TimeDrivenLIF_Voltage_jump", 1, parameters=dict(LIF_PARAMS))


@pytest.mark.parametrize("n", [128, 384, 512, 640, 1152, 8320])  # one slice, ragged ones, two chunks of spike words
@pytest.mark.parametrize("density", [0.0, 0.03, 1.0])
def test_delivery_is_the_sequential_float_sum(n, density):
    w = _weights(n)
    s = (np.random.default_rng(n).random((64, n)) < density).astype(np.uint8)
    if n > 4096:  # the sums of a few instances are enough at this size
        s[4:] = 0
    eng = DensePopulations(w, _layer(), precision="fp32")
    got = eng.deliver(s)
    eng.close()
    for b in range(64):
        rows = w[np.nonzero(s[b])[0]]
        want = np.cumsum(rows, axis=0, dtype=np.float32)[-1] if len(rows) else np.zeros(n, np.float32)
        assert np.array_equal(got[b], want)
        if n > 4096 and b >= 4:
            break


@pytest.mark.parametrize("n", [128, 640, 1152])
def test_steps_equal_the_oracle(oracle_lib, n):
    import oracle

    w = _weights(n)
    mid, f, ip = _layer().native_params()
    eng = DensePopulations(w, _layer(), precision="fp32", drive_rate_hz=8000.0, drive_weight=0.5, dt=0.1)
    eng.run(100).run(37)
    ref = oracle.OracleDense(64, n, w, f, ip, 8000.0, 0.5, 0.1)
    ref.run(137)
    v, last = eng.state()
    rv, rlast, rs = ref.state()
    assert np.array_equal(eng.spike_counts(), ref.counts()) and eng.spike_counts().sum() > 0
    assert np.array_equal(v.ravel(), rv.astype(np.float32)) and np.array_equal(last.ravel(), rlast)
    assert np.array_equal(eng.spikes().ravel(), rs)


@pytest.mark.parametrize("precision", ["split_bf16", "split_bf16_sync", "fp32"])
@pytest.mark.parametrize("n", [128, 384])
def test_spikes_in_and_out_of_each_layout(precision, n):
    """Out: a neuron spiked at the last step exactly where its LastSpike counter is 0.  In: any non-zero byte is a
    spike, and a delivery leaves the simulation as it was."""
    w = _weights(n)
    eng = DensePopulations(w, _layer(), precision=precision)
    assert not eng.spikes().any()
    total = 0
    for _ in range(30):
        eng.run(5)
        assert np.array_equal(eng.spikes(), (eng.state()[1] == 0).astype(np.uint8))
        total += int(eng.spikes().sum())
    assert total > 0
    s = (np.random.default_rng(n).random((64, n)) < 0.1).astype(np.uint8)
    before = eng.spikes()
    out = eng.deliver(s)
    assert np.array_equal(out, eng.deliver(s * 7)) and np.array_equal(eng.spikes(), before)
    # |error| of a split product: 2^-16 of each weight that is added, and the FP32 sums
    bound = 2.0 ** -15 * (s.astype(np.float64) @ np.abs(w).astype(np.float64)) + 1e-30
    assert (np.abs(out - s.astype(np.float64) @ w.astype(np.float64)) <= bound).all()
