"""nbg_poisson_inputs against the PoissonRate hash in numpy, bit for bit, at channel counts that are and are not a
multiple of four, and more steps than the grid has rows."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _hash_uniform01(index, step):
    with np.errstate(over="ignore"):
        x = (index.astype(np.uint32) * np.uint32(747796405) + np.uint32(step + 1) * np.uint32(2891336453)
             + np.uint32(0x9e3779b9))
        x ^= x >> np.uint32(16)
        x *= np.uint32(2246822519)
        x ^= x >> np.uint32(13)
        x *= np.uint32(3266489917)
        x ^= x >> np.uint32(16)
    return (x & np.uint32(0xFFFFFF)).astype(np.float32) / np.float32(0x1000000)


@pytest.mark.parametrize("T,B,C", [(1, 1, 1), (7, 3, 5), (50, 128, 256), (20, 31, 100), (3000, 2, 4), (9, 500, 333)])
def test_inputs_equal_the_hash(T, B, C):
    from neuronbridge_gb300.adjoint import poisson_inputs

    rates = torch.linspace(-50.0, 1200.0, C)
    x = poisson_inputs(rates, T, B, dt=1.0, seed=12345).cpu().numpy()
    r = np.maximum(rates.numpy(), np.float32(0))
    prob = np.minimum(r * np.float32(1.0) * np.float32(0.001), np.float32(1.0))
    idx = np.arange(B * C).reshape(B, C) + 12345
    for t in {0, T // 2, T - 1}:
        assert np.array_equal(x[t], (_hash_uniform01(idx, t) < prob).astype(np.float32))
