"""The fused tcgen05 dense step at the edges of its tiles (64 post neurons up to 4,864 neurons on 152 SMs, 128 above; one K
chunk a half, more chunks than stages).  The weights are multiples of 1/64 up to 1, so each is one BF16 value and every sum
is exact in FP32: the products' order cannot matter, and the step equals the FP32 path's bit for bit."""
import numpy as np
import pytest

from neuronbridge_gb300 import NeuronLayer
from neuronbridge_gb300.dense import DensePopulations
from neuronbridge_gb300.workloads import LIF_PARAMS

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [128, 256, 896, 1152, 4864, 4992])
def test_fused_step_equals_the_fp32_path(n):
    w = np.random.default_rng(n).integers(-64, 65, (n, n), dtype=np.int8).astype(np.float32) / 64.0
    layer = NeuronLayer("TimeDrivenLIF_Voltage_jump", 1, parameters=dict(LIF_PARAMS))
    out = []
    for precision in ("split_bf16", "fp32"):
        eng = DensePopulations(w, layer, precision=precision, drive_rate_hz=8000.0, drive_weight=0.5, dt=0.1)
        eng.run(100).run(61)
        out.append((*eng.state(), eng.spike_counts(), eng.spikes()))
        eng.close()
    assert out[0][2].sum() > 0
    for a, b in zip(*out):
        assert np.array_equal(a, b)
