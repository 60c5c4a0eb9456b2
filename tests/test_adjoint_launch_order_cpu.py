"""The launches of a backward, recorded by a library that runs nothing.  Which adjoint steps may overlap the launch before
them: a chained step reads W and the forward's record before that launch has ended, so it has to be a step of the same sweep.
And how much of dI an FP32 backward holds at once."""
import pytest
import torch

from neuronbridge_gb300 import adjoint

STEPS = ("nbg_lif_adjoint_step_parts", "nbg_lif_adjoint_step_chained")


class _Recorder:
    def __init__(self):
        self.calls = []

    def __getattr__(self, name):
        def call(*args):
            self.calls.append(name)
            return 1 if name == "nbg_product_tn_split" else 0  # NBG_OK; no sweep: a launch a step
        return call


def _backward(monkeypatch, n, b, steps, segment, record):
    c, o = 8, 3
    monkeypatch.setattr(adjoint, "_stream", lambda: None)
    lib = _Recorder()
    p = adjoint.GradParams(-65.0, -65.0, 10.0, 2, 0)
    x, w_in, w_rec, w_out = (torch.zeros(s) for s in ((steps, b, c), (c, n), (n, n), (n, o)))
    alpha, theta, z, gy = torch.zeros(n), torch.zeros(n), torch.zeros(b, n), torch.zeros(b, o)
    rec = adjoint._record_buffers(steps, b, n, "cpu") if record else None
    ck = torch.zeros(0 if record else -(-steps // segment), b, n)
    adjoint._backward_body(lib, gy, x, w_in, w_rec, w_out, alpha, theta, z, ck, ck.int(), ck, p, segment,
                           adjoint.readout_coefficients(steps, 0.9), rec)
    return [name for name in lib.calls if name != "nbg_lif_adjoint_sweep_work"]


@pytest.mark.parametrize("record", [False, True])
def test_a_chained_step_follows_a_step(monkeypatch, record):
    steps = 7
    order = _backward(monkeypatch, 1280, 128, steps, 3, record)
    chained = [k for k, name in enumerate(order) if name == STEPS[1]]
    assert sum(name in STEPS for name in order) == steps
    # a replayed segment begins anew (7 steps in segments of 3); a recorded run once
    assert len(chained) == steps - (1 if record else 3)
    assert all(order[k - 1] in STEPS for k in chained)


def test_dI_of_a_whole_run_counts_against_the_record_budget(monkeypatch):
    steps, b, n = 7, 4, 20
    products = lambda: _backward(monkeypatch, n, b, steps, 3, True).count("nbg_product_tn")
    assert products() == 2  # W_rec and W_in once
    need = adjoint.record_bytes(steps, b, n) + 8 * steps * b * n
    monkeypatch.setattr(adjoint, "RECORD_BUDGET_BYTES", need)
    assert products() == 2
    monkeypatch.setattr(adjoint, "RECORD_BUDGET_BYTES", need - 1)
    assert products() == 6  # per segment of three steps
    monkeypatch.setattr(adjoint, "RECORD_BUDGET_BYTES", 1 << 60)
    assert not adjoint._whole_dI(1 << 16, 1 << 15, 1) and adjoint._whole_dI((1 << 16) - 1, 1 << 15, 1)


def test_a_run_without_steps_has_no_products(monkeypatch):
    """No step, no term: the gradients stay the zeros that they start from."""
    assert "nbg_product_tn" not in _backward(monkeypatch, 20, 4, 0, 3, True)
