"""The fused adjoint step's two ways to exchange its split-K partials (distributed shared memory, a workspace in global
memory) give the same bits in every output, at the smallest N, an odd multiple of 128 (ragged K split) and above one pipeline."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [512, 640, 1152, 1664])
def test_exchange_through_global_memory_equals_distributed_shared_memory(n):
    from neuronbridge_gb300 import adjoint
    from neuronbridge_gb300.adjoint import _bind, _ptr

    lib = _bind()
    fused = lib.nbg_lif_adjoint_step_fused
    fused.restype, fused.argtypes = ctypes.c_int, lib.nbg_lif_adjoint_step_parts.argtypes[:-3] + [ctypes.c_void_p] * 2
    b, k_cols = 128, 256
    g = torch.Generator(device="cuda").manual_seed(n)
    r = lambda *shape: torch.randn(*shape, generator=g, device="cuda")
    st = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    w = r(n, n) / n ** 0.5
    w_hi, w_lo, d_hi, d_lo = (torch.empty(k, device="cuda", dtype=torch.bfloat16) for k in (n * n, n * n, b * n, b * n))
    assert lib.nbg_adjoint_rec_prepare(_ptr(w), _ptr(w_hi), _ptr(w_lo), n, st) == 0
    d_hi.copy_(r(b * n))
    d_lo.copy_(r(b * n) * 2.0 ** -9)
    g_read, u, vprev = r(b, n), r(b, n), r(b, n)
    s, m = (u > 0.5).float(), (r(b, n) > -1.0).to(torch.uint8)
    alpha, theta = torch.full((n,), 0.9, device="cuda"), torch.full((n,), 0.5, device="cuda")
    acc = [r(b, n) for _ in range(3)]
    p = adjoint.GradParams()
    p.v_rest, p.v_reset, p.slope, p.smooth = 0.0, -0.1, 10.0, 0
    out = []
    for parts in (None, torch.empty(8 * b * n, device="cuda")):
        lam_v, g_theta, g_alpha = (x.clone() for x in acc)
        dI = torch.empty(b, n, device="cuda")
        o = [torch.empty(b * n, device="cuda", dtype=torch.bfloat16) for _ in range(2)]
        t = [torch.zeros(n * k_cols, device="cuda", dtype=torch.bfloat16) for _ in range(2)]
        err = torch.zeros(1, device="cuda", dtype=torch.int32)
        args = [_ptr(w_hi), _ptr(w_lo), _ptr(d_hi), _ptr(d_lo), _ptr(o[0]), _ptr(o[1]), _ptr(g_read), 0.25, _ptr(u), _ptr(s),
                _ptr(m), _ptr(vprev), _ptr(lam_v), _ptr(dI), _ptr(g_theta), _ptr(g_alpha), _ptr(alpha), _ptr(theta),
                ctypes.byref(p), b, n, _ptr(t[0]), _ptr(t[1]), 128, k_cols]
        if parts is None:
            assert fused(*args, _ptr(err), st) == 0
        else:
            assert lib.nbg_lif_adjoint_step_parts(*args, _ptr(parts), _ptr(err), st) == 0
            assert lib.nbg_lif_adjoint_step_parts(*args, None, _ptr(err), st) != 0  # refused, nothing launched
        assert int(err.item()) == 0
        out.append((dI, lam_v, g_theta, g_alpha, *o, *t))
    assert torch.isfinite(out[0][0]).all() and out[0][0].abs().sum() > 0
    for x, y in zip(*out):
        assert torch.equal(x, y)


@pytest.mark.parametrize("n,record", [(128, False), (256, True), (384, True), (512, True), (640, False), (768, False), (896, True), (1024, False), (1152, True)])
def test_sweep_equals_the_steps(monkeypatch, n, record):
    """A segment's steps in one launch against one or two launches each, bit for bit: N below eight K ranges, with two K chunks a CTA, with a last
    CTA of more chunks than pipeline stages (768 and 1152: six, 896: eight), the largest that 152 SMs hold; the whole run or segments of 20 of 47 steps."""
    from neuronbridge_gb300 import adjoint
    from neuronbridge_gb300.adjoint import RecurrentLIF, _bind, poisson_inputs

    torch.manual_seed(0)
    model = RecurrentLIF(n_in=40, n_rec=n, n_out=5, checkpoint=20, seed=11, smooth=False, device="cuda", use_graphs=False,
                         record=record)
    x = poisson_inputs(torch.linspace(50.0, 400.0, 40), 47, 128, dt=1.0, seed=3)
    labels = torch.arange(128, device="cuda") % 5
    assert _bind().nbg_lif_adjoint_sweep_work(128, n) > 0 and _bind().nbg_lif_adjoint_sweep_work(64, n) == 0
    out = []
    for sweep in (True, False):
        monkeypatch.setattr(adjoint, "SWEEP", sweep)
        model.zero_grad(set_to_none=True)
        torch.nn.functional.cross_entropy(model(x), labels).backward()
        out.append([q.grad.clone() for q in model.parameters()])
    assert any(g.abs().sum() > 0 for g in out[0])
    for a, b in zip(*out):
        assert torch.equal(a, b)


def test_sweeps_on_two_streams_of_two_threads():
    """Cooperative launches that do not fit beside one another, on streams of different priority: each gives what it gives
    alone, and none of its bounded waits runs out."""
    import threading

    from neuronbridge_gb300.adjoint import RecurrentLIF, poisson_inputs

    x = poisson_inputs(torch.linspace(50.0, 400.0, 40), 100, 128, dt=1.0, seed=3)
    labels = torch.arange(128, device="cuda") % 5
    models = []
    for _ in range(2):
        torch.manual_seed(0)
        models.append(RecurrentLIF(n_in=40, n_rec=1024, n_out=5, seed=11, smooth=False, device="cuda", use_graphs=False))

    def grads(model):
        model.zero_grad(set_to_none=True)
        torch.nn.functional.cross_entropy(model(x), labels).backward()
        return [q.grad.clone() for q in model.parameters()]

    want = grads(models[0])
    torch.cuda.synchronize()
    out = [None, None]

    def work(k):
        stream = torch.cuda.Stream(priority=-k)
        with torch.cuda.stream(stream):
            out[k] = [grads(models[k]) for _ in range(10)]
            stream.synchronize()

    threads = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for runs in out:
        for got in runs:
            for a, b in zip(got, want):
                assert torch.equal(a, b)


@pytest.mark.parametrize("smooth", [False, True])
def test_recorded_gradients_by_segment(monkeypatch, smooth):
    """A record beside which dI of the whole run does not fit: the gradients of a replayed run, segment by segment, bit for bit."""
    from neuronbridge_gb300 import adjoint
    from neuronbridge_gb300.adjoint import RecurrentLIF, poisson_inputs

    monkeypatch.setattr(adjoint, "RECORD_BUDGET_BYTES", 0)
    x = poisson_inputs(torch.linspace(50.0, 400.0, 30), 47, 20, dt=1.0, seed=3)
    labels = torch.arange(20, device="cuda") % 5
    out = []
    for record in (True, False):
        model = RecurrentLIF(n_in=30, n_rec=150, n_out=5, checkpoint=20, seed=11, smooth=smooth, weight_scale=5.0,
                             use_graphs=False, record=record)
        torch.nn.functional.cross_entropy(model(x), labels).backward()
        out.append([q.grad for q in model.parameters()])
    assert all(g.abs().sum() > 0 for g in out[0][:3])
    for a, b in zip(*out):
        assert torch.equal(a, b)


@pytest.mark.parametrize("smooth", [False, True])
def test_a_run_without_steps(smooth):
    from neuronbridge_gb300.adjoint import RecurrentLIF

    model = RecurrentLIF(n_in=30, n_rec=150, n_out=5, seed=11, smooth=smooth, use_graphs=False)
    y = model(torch.zeros(0, 4, 30, device="cuda"))
    y.sum().backward()
    assert not y.any() and all(not q.grad.any() for q in model.parameters())


@pytest.mark.parametrize("n,steps", [(128, 1), (384, 1), (1024, 1), (256, 30)])
def test_a_sweep_has_no_recurrent_term_at_the_last_step(monkeypatch, n, steps):
    """The sweep's product at the last step runs on a zero operand: with a weight that is not finite it counts as little as in
    the separate steps, which have none.  (One step: finite gradients.  More: NaN in the same places.)"""
    from neuronbridge_gb300 import adjoint
    from neuronbridge_gb300.adjoint import RecurrentLIF, poisson_inputs

    model = RecurrentLIF(n_in=40, n_rec=n, n_out=5, checkpoint=20, seed=11, weight_scale=20.0, use_graphs=False)
    with torch.no_grad():
        model.w_rec[3, 5] = float("inf")
    x = poisson_inputs(torch.linspace(50.0, 400.0, 40), steps, 128, dt=1.0, seed=3)
    labels = torch.arange(128, device="cuda") % 5
    out = []
    for sweep in (True, False):
        monkeypatch.setattr(adjoint, "SWEEP", sweep)
        monkeypatch.setattr(adjoint, "FUSED_STEP", sweep)
        model.zero_grad(set_to_none=True)
        torch.nn.functional.cross_entropy(model(x), labels).backward()
        out.append([q.grad for q in model.parameters()])
    if steps == 1:
        assert all(torch.isfinite(g).all() for g in out[0])
        for a, b in zip(*out):
            assert torch.equal(a, b)
    for a, b in zip(*out):
        assert torch.equal(torch.isnan(a), torch.isnan(b))
