"""FP32 products of the recurrent LIF on the CUDA cores (nbg_product_nt, nbg_product_tn and the steps fused with the
former) at the edges of their tiles, K splits and copy widths.

A product is held to the error bound of its summation: each output is a sum of K rounded-once terms added over chains
and trees of at most K / 32 + 24 additions, so |error| <= (K / 32 + 24) 2^-24 sum |a| |b|.  A fused step must equal the
product followed by the elementwise step bit for bit: the same sums, then the same operations."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


def _lib():
    from neuronbridge_gb300 import _lib as base
    from neuronbridge_gb300.adjoint import _bind, _ptr, _stream

    return _bind(), base.check, _ptr, _stream()


def _randn(*shape, seed=0):
    return torch.randn(*shape, device="cuda", generator=torch.Generator(device="cuda").manual_seed(seed))


def _within_bound(got, a, b, K):
    ref = a.double() @ b.double()
    bound = (K / 32 + 24) * 2.0 ** -24 * (a.abs().double() @ b.abs().double())
    assert ((got.double() - ref).abs() <= bound).all()


@pytest.mark.parametrize("offset", [0, 1])  # 1: operands that are not 16-byte aligned
@pytest.mark.parametrize("M,N,K", [(1, 1, 1), (3, 5, 7), (32, 32, 64), (33, 65, 63), (12, 300, 300), (31, 512, 512),
                                   (64, 1000, 1000), (700, 290, 52), (5, 40, 2100), (130, 1100, 513)])
def test_product_nt_within_its_summation_bound(M, N, K, offset):
    lib, check, ptr, st = _lib()
    a = _randn(M * K + 4, seed=1)[offset:offset + M * K].view(M, K)
    w = _randn(N * K + 4, seed=2)[offset:offset + N * K].view(N, K)
    c = torch.full((M, N), float("nan"), device="cuda")
    check(lib.nbg_product_nt(ptr(a), ptr(w), ptr(c), M, N, K, st))
    _within_bound(c, a, w.t(), K)


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("M,N,K", [(1, 1, 1), (5, 7, 33), (64, 64, 256), (65, 130, 1000), (300, 50, 720),
                                   (512, 512, 8000), (128, 514, 3333)])
def test_product_tn_within_its_summation_bound(M, N, K, offset):
    lib, check, ptr, st = _lib()
    a = _randn(M * K + 4, seed=3)[offset:offset + M * K].view(K, M)
    b = _randn(N * K + 4, seed=4)[offset:offset + N * K].view(K, N)
    split = lib.nbg_product_tn_split(M, N, K)
    part = torch.full((split, M, N), float("nan"), device="cuda")
    out = torch.zeros((M, N), device="cuda")
    check(lib.nbg_product_tn(ptr(a), ptr(b), ptr(part), split, M, N, K, st))
    check(lib.nbg_adjoint_reduce_add(ptr(out), ptr(part), split, M * N, M * N, st))
    _within_bound(out, a.t(), b, K)


@pytest.mark.parametrize("B,N", [(1, 1), (3, 50), (12, 300), (32, 512), (33, 70), (64, 1000), (128, 257), (160, 1024)])
@pytest.mark.parametrize("smooth", [0, 1])
def test_fused_adjoint_steps_equal_product_then_step(B, N, smooth):
    from neuronbridge_gb300.adjoint import GradParams

    lib, check, ptr, st = _lib()
    p = GradParams(-65.0, -65.0, 0.5, 2, smooth)
    w = _randn(N, N, seed=5)
    gr, u, vp = _randn(B, N, seed=6), -60.0 + 5.0 * _randn(B, N, seed=7), -60.0 + 5.0 * _randn(B, N, seed=8)
    s = torch.sigmoid(_randn(B, N, seed=9)) if smooth else (_randn(B, N, seed=9) > 1).float()
    m = (_randn(B, N, seed=10) > -1).to(torch.uint8)
    al, th = torch.full((N,), 0.05, device="cuda"), torch.full((N,), -50.0, device="cuda")
    out = []
    for fused in (False, True):
        lam, gt, ga = (torch.zeros(B, N, device="cuda") for _ in range(3))
        d = [torch.empty(B, N, device="cuda") for _ in range(3)]
        for k in range(3):  # the sweep's first step has no recurrent term
            nxt = d[k - 1] if k else None
            if fused:
                check(lib.nbg_lif_adjoint_step_product(
                    ptr(nxt), ptr(w), ptr(gr), 0.3, ptr(u), ptr(s), ptr(m), ptr(vp), ptr(lam), ptr(d[k]), ptr(gt),
                    ptr(ga), ptr(al), ptr(th), ctypes.byref(p), int(k > 0), B, N, st))
                continue
            ge = torch.empty(B, N, device="cuda")
            if k:
                check(lib.nbg_product_nt(ptr(nxt), ptr(w), ptr(ge), B, N, N, st))
            check(lib.nbg_lif_adjoint_step(ptr(ge) if k else None, ptr(gr), 0.3, ptr(u), ptr(s), ptr(m), ptr(vp),
                                           ptr(lam), ptr(d[k]), ptr(gt), ptr(ga), ptr(al), ptr(th), ctypes.byref(p),
                                           B, N, st))
        out.append(d + [lam, gt, ga])
    for x, y in zip(*out):
        assert torch.equal(x, y)


@pytest.mark.parametrize("B,N", [(1, 3), (12, 300), (40, 512), (33, 70), (160, 1024)])
def test_fused_smooth_forward_equals_product_then_step(B, N):
    from neuronbridge_gb300.adjoint import GradParams

    lib, check, ptr, st = _lib()
    p = GradParams(-65.0, -65.0, 0.5, 2, 1)
    w = 3.0 * _randn(N, N, seed=5) / N ** 0.5
    w_t = torch.empty_like(w)
    check(lib.nbg_transpose(ptr(w), ptr(w_t), N, N, st))
    assert torch.equal(w_t, w.t())
    xi = 3.0 * _randn(3, B, N, seed=6)
    al, th = torch.full((N,), 0.05, device="cuda"), torch.full((N,), -50.0, device="cuda")
    out = []
    for fused in (False, True):
        v, z = torch.full((B, N), -65.0, device="cuda"), torch.zeros(B, N, device="cuda")
        ref = torch.zeros(B, N, device="cuda", dtype=torch.int32)
        S, U, VP = torch.zeros(4, B, N, device="cuda"), torch.empty(3, B, N, device="cuda"), torch.empty(3, B, N, device="cuda")
        M = torch.empty(3, B, N, device="cuda", dtype=torch.uint8)
        for k in range(3):
            if fused:
                check(lib.nbg_lif_forward_step_smooth(
                    ptr(S[k]), ptr(w_t), ptr(xi[k]), ptr(v), ptr(S[k + 1]), ptr(U[k]), ptr(M[k]), ptr(VP[k]), ptr(z),
                    0.3, ptr(al), ptr(th), ctypes.byref(p), int(k > 0), B, N, st))
                continue
            cur = torch.empty(B, N, device="cuda")
            check(lib.nbg_product_nt(ptr(S[k]), ptr(w_t), ptr(cur), B, N, N, st))
            cur.add_(xi[k])
            check(lib.nbg_lif_forward_step(ptr(cur), ptr(v), ptr(ref), ptr(S[k + 1]), ptr(U[k]), ptr(M[k]), ptr(VP[k]),
                                           ptr(z), 0.3, ptr(al), ptr(th), ctypes.byref(p), B, N, st))
        out.append([v, z, S, U, M, VP])
    for x, y in zip(*out):
        assert torch.equal(x, y)


def test_more_row_tiles_than_a_grid_has_rows():
    """2^16 and more tiles of rows: batches and input widths beyond 65,535 tiles run as any other."""
    from neuronbridge_gb300.adjoint import GradParams

    lib, check, ptr, st = _lib()
    r = 65535 * 32 + 40
    x = _randn(r, 3, seed=1)
    t = torch.empty(3, r, device="cuda")
    check(lib.nbg_transpose(ptr(x), ptr(t), r, 3, st))
    assert torch.equal(t, x.t())
    w = torch.eye(3, device="cuda") * 0.5
    c = torch.full((r, 3), float("nan"), device="cuda")
    check(lib.nbg_product_nt(ptr(x), ptr(w), ptr(c), r, 3, 3, st))
    assert torch.equal(c, 0.5 * x)
    # a step of both directions against the product and the plain step
    p = GradParams(-65.0, -65.0, 0.5, 2, 1)
    al, th = torch.full((3,), 0.05, device="cuda"), torch.full((3,), -50.0, device="cuda")
    full = lambda v: torch.full((r, 3), v, device="cuda")
    s, m, u = torch.sigmoid(x), torch.ones(r, 3, device="cuda", dtype=torch.uint8), -60.0 + x
    out = []
    for fused in (False, True):
        v, z, s1, u1, m1, vp1, lam, gt, ga, d = full(-60.0), full(0.0), full(0.0), full(0.0), m.clone(), full(0.0), full(0.1), \
            full(0.0), full(0.0), full(0.0)
        if fused:
            check(lib.nbg_lif_forward_step_smooth(ptr(s), ptr(w), ptr(x), ptr(v), ptr(s1), ptr(u1), ptr(m1), ptr(vp1), ptr(z),
                                                  0.3, ptr(al), ptr(th), ctypes.byref(p), 0, r, 3, st))
            check(lib.nbg_lif_adjoint_step_product(ptr(x), ptr(w), ptr(x), 0.3, ptr(u), ptr(s), ptr(m), ptr(u1), ptr(lam), ptr(d),
                                                   ptr(gt), ptr(ga), ptr(al), ptr(th), ctypes.byref(p), 0, r, 3, st))
        else:
            cur, ref = 0.5 * s + x, torch.zeros(r, 3, device="cuda", dtype=torch.int32)
            check(lib.nbg_lif_forward_step(ptr(cur), ptr(v), ptr(ref), ptr(s1), ptr(u1), ptr(m1), ptr(vp1), ptr(z), 0.3, ptr(al),
                                           ptr(th), ctypes.byref(p), r, 3, st))
            ge = 0.5 * x
            check(lib.nbg_lif_adjoint_step(ptr(ge), ptr(x), 0.3, ptr(u), ptr(s), ptr(m), ptr(u1), ptr(lam), ptr(d), ptr(gt),
                                           ptr(ga), ptr(al), ptr(th), ctypes.byref(p), r, 3, st))
        out.append((v, z, s1, u1, m1, vp1, lam, gt, ga, d))
    for a, b in zip(*out):
        assert torch.equal(a, b)
    rows = 65535 * 64 + 70
    a, b = _randn(1, rows, seed=2), _randn(1, 3, seed=3)
    part, g = torch.empty(rows, 3, device="cuda"), torch.zeros(rows, 3, device="cuda")
    check(lib.nbg_product_tn(ptr(a), ptr(b), ptr(part), 1, rows, 3, 1, st))
    check(lib.nbg_adjoint_reduce_add(ptr(g), ptr(part), 1, rows * 3, rows * 3, st))
    assert torch.equal(g, a.t() * b)


@pytest.mark.parametrize("K", [64, 255, 256, 1000, 1031])
def test_small_product_of_few_and_of_many_outputs(K):
    """The readout's product with the loads of eight terms in flight (fewer than 4,096 outputs, K >= 256) and without: the same
    bits, within the bound of its lanes' chains and their tree."""
    lib, check, ptr, st = _lib()
    a, b = _randn(512, K, seed=1), _randn(K, 10, seed=2)
    out = [torch.full((m, 10), float("nan"), device="cuda") for m in (409, 512)]
    for c in out:
        check(lib.nbg_small_gemm(ptr(a), K, 1, ptr(b), 10, 1, ptr(c), len(c), 10, K, st))
    assert torch.equal(out[0], out[1][:409])
    _within_bound(out[1], a, b, K)


@pytest.mark.parametrize("K", [24, 64, 100, 129, 240, 480, 1000, 2048])
def test_products_are_no_further_from_64_bits_than_the_small_product(K):
    """Error of the norm against 64 bits, of K split over CTAs (12 rows) and not (1,000), and of A^T B, against nbg_small_gemm on
    the same operands: no larger, but for the 2 % that 10^4 to 10^6 outputs leave uncertain (their own spread is below 1 %)."""
    lib, check, ptr, st = _lib()

    def error(got, ref):
        return ((got.double() - ref).norm() / ref.norm()).item()

    def small(a, a_rs, a_cs, b, b_rs, b_cs, M, N):
        c = torch.empty(M, N, device="cuda")
        check(lib.nbg_small_gemm(ptr(a), a_rs, a_cs, ptr(b), b_rs, b_cs, ptr(c), M, N, K, st))
        return c

    for M in (12, 1000):
        a, w = _randn(M, K, seed=1), _randn(1024, K, seed=2)
        ref, c = a.double() @ w.double().t(), torch.empty(M, 1024, device="cuda")
        check(lib.nbg_product_nt(ptr(a), ptr(w), ptr(c), M, 1024, K, st))
        assert error(c, ref) <= 1.02 * error(small(a, K, 1, w, 1, K, M, 1024), ref)
    for M in (50, 512):
        a, b = _randn(K, M, seed=3), _randn(K, 512, seed=4)
        ref, c = a.double().t() @ b.double(), torch.zeros(M, 512, device="cuda")
        split = lib.nbg_product_tn_split(M, 512, K)
        part = torch.empty((split, M, 512), device="cuda")
        check(lib.nbg_product_tn(ptr(a), ptr(b), ptr(part), split, M, 512, K, st))
        check(lib.nbg_adjoint_reduce_add(ptr(c), ptr(part), split, M * 512, M * 512, st))
        assert error(c, ref) <= 1.02 * error(small(a, 1, M, b, 512, 1, M, 512), ref)
