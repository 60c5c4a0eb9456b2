"""The spike-driven forward of a segment (k_lif_fwd_rows: 16-byte columns, or single columns where N or a pointer is not
aligned) against one nbg_lif_forward_step_sparse launch per step fed the ascending FP32 input sum, bit for bit: few and
many spikes a step, no input and every input on, one column group and several, one and several warps."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _rand(shape, seed, normal=False, offset=0):
    n = 1
    for d in shape:
        n *= d
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = (torch.randn if normal else torch.rand)(n + 4, device="cuda", generator=g)
    return x[offset:offset + n].view(shape)


@pytest.mark.parametrize("N,C,offset", [(1, 1, 0), (3, 5, 0), (64, 33, 0), (300, 40, 0), (301, 40, 0), (512, 256, 1),
                                        (1000, 70, 0), (1023, 70, 0), (1024, 256, 0), (2047, 40, 0), (2048, 40, 0),
                                        (64, 4096, 0), (64, 4097, 0)])
@pytest.mark.parametrize("density", [0.02, 1.0])
def test_rows_kernel_equals_per_step_launches(N, C, offset, density):
    from neuronbridge_gb300.adjoint import GradParams, _bind, _SpikeLists, _stream

    lib, st = _bind(), _stream()
    B, L = 3, 11
    w_rec = _rand((N, N), 1, True, offset) * 0.3 if not offset else _rand((N, N), 1, True, offset).mul_(0.3)
    w_in = _rand((C, N), 2, True) * 0.5
    x = (_rand((L, B, C), 3) < density).float() * _rand((L, B, C), 4)
    x[1] = 0.0
    xi = torch.zeros(L, B, N, device="cuda")
    for ch in range(C):  # ascending, one rounding each; a zero input adds a zero
        xi = xi + x[:, :, ch:ch + 1] * w_in[ch]
    alpha = _rand((N,), 5) * 0.1
    theta = _rand((N,), 6) - (0.5 if density == 1.0 else -0.3)  # about every other neuron fires, or a few
    p = GradParams(0.0, 0.0, 10.0, 1, 0)
    c = torch.linspace(0.1, 1.0, L, device="cuda")
    s0 = (_rand((B, N), 7) < 0.3).float()
    out = []
    for form in ("step", "segment", "gather"):
        lists = _SpikeLists(B, N, "cuda")
        v, ref = _rand((B, N), 8).clone(), torch.zeros(B, N, device="cuda", dtype=torch.int32)
        S, U, VP = (torch.zeros((L, B, N), device="cuda") for _ in range(3))
        M = torch.zeros((L, B, N), device="cuda", dtype=torch.uint8)
        z = torch.zeros((B, N), device="cuda")
        lists.load(lib, s0, B, N, st)
        if form == "step":
            for k in range(L):
                lists.step(lib, xi[k], w_rec, v, ref, S[k], U[k], M[k], VP[k], z, float(c[k]), alpha, theta, p, B, N, st)
        elif form == "segment":
            lists.segment(lib, xi, w_rec, v, ref, S, None, U, M, VP, z, c, alpha, theta, p, L, B, N, st)
        else:
            lists.segment_gather(lib, x, w_in, w_rec, v, ref, S, None, U, M, VP, z, c, alpha, theta, p, L, B, N, st)
        torch.cuda.synchronize()
        cnt = lists.cnt[lists.cur].clone()
        idx = torch.cat([lists.idx[lists.cur][b][:int(cnt[b])] for b in range(B)])
        out.append((v, ref, S, U, M, VP, z, cnt, idx))
    if N > 3:
        assert out[0][2].sum() > 0
    for other in out[1:]:
        for a, b in zip(out[0], other):
            assert torch.equal(a, b)


def test_rows_kernel_without_a_record_gives_the_last_spikes():
    from neuronbridge_gb300.adjoint import GradParams, _bind, _SpikeLists, _stream

    lib, st = _bind(), _stream()
    for N in (300, 301):
        B, L = 2, 5
        w, xi = _rand((N, N), 1, True) * 0.3, _rand((L, B, N), 2)
        alpha, theta = torch.full((N,), 0.05, device="cuda"), torch.full((N,), 1.0, device="cuda")
        p = GradParams(0.0, 0.0, 10.0, 2, 0)
        lists = _SpikeLists(B, N, "cuda")
        v, ref = torch.zeros(B, N, device="cuda"), torch.zeros(B, N, device="cuda", dtype=torch.int32)
        last, S = torch.full((B, N), -1.0, device="cuda"), torch.zeros(L, B, N, device="cuda")
        lists.segment(lib, xi, w, v, ref, None, last, None, None, None, None, None, alpha, theta, p, L, B, N, st)
        other = _SpikeLists(B, N, "cuda")
        v2, ref2 = torch.zeros(B, N, device="cuda"), torch.zeros(B, N, device="cuda", dtype=torch.int32)
        other.segment(lib, xi, w, v2, ref2, S, None, None, None, None, None, None, alpha, theta, p, L, B, N, st)
        torch.cuda.synchronize()
        assert torch.equal(last, S[-1]) and torch.equal(v, v2) and S.sum() > 0
