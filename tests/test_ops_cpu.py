"""CPU checks of the op layer: the GEMM addressing emulation that stands in for the tcgen05 kernel, the layout logic
of the pointwise convolutions (NCHW / channels-last in every combination), fused AdamW reference path, losses."""

import math

import numpy as np
import pytest
import torch

from makani_b200.ops import conv as C
from makani_b200.ops.gemm import ACT_DGELU, ACT_GELU, ACT_MULAUX, ACT_NONE, BIAS_ROW, Operand, Output, Tri, gemm
from makani_b200.ops.optim import FusedAdamW
from makani_b200.ops.spectral import expand_weight, fold_weight_grad


def test_emulated_gemm_majors_batches_and_scatter():
    torch.manual_seed(0)
    M, N, K, Z = 5, 7, 6, 3
    a = torch.randn(Z, K, M)          # MN-major A
    b = torch.randn(Z, N, K)          # K-major B
    d = torch.zeros(Z, M, N)
    gemm(M, N, K, Operand(a, ld=M, mn_major=True, zs_lo=K * M), Operand(b, ld=K, zs_lo=N * K), Output(d, rs_lo=N, d_zlo=M * N), zlo_n=Z)
    assert torch.allclose(d, torch.einsum("zkm,znk->zmn", a, b), atol=1e-5)
    # split row / column addressing and accumulate
    d2 = torch.zeros(2, M, 4, N // 1)
    a2 = torch.randn(M * 2, K)
    b2 = torch.randn(N, K)
    out = torch.zeros(M, 2, N)
    gemm(2 * M, N, K, Operand(a2, ld=K), Operand(b2, ld=K), Output(out, rdiv=2, rs_hi=2 * N, rs_lo=N), alpha=2.0)
    assert torch.allclose(out.reshape(2 * M, N), 2.0 * a2 @ b2.t(), atol=1e-5)
    acc = torch.ones(2 * M, N)
    gemm(2 * M, N, K, Operand(a2, ld=K), Operand(b2, ld=K), Output(acc, rs_lo=N), accumulate=True)
    assert torch.allclose(acc, 1.0 + a2 @ b2.t(), atol=1e-5)


def test_emulated_gemm_saved_gelu_derivative_matches_autograd():
    """`preact_deriv` stores d gelu / d pre in the second output; multiplying an upstream gradient by it (ACT_MULAUX)
    gives what autograd gives through gelu, and what ACT_DGELU gives from a saved pre-activation."""
    torch.manual_seed(3)
    M, N, K = 6, 9, 5
    a, b, bias = torch.randn(M, K), torch.randn(N, K), torch.randn(M)
    y, dact, pre = torch.zeros(M, N), torch.zeros(M, N), torch.zeros(M, N)
    gemm(M, N, K, Operand(a, ld=K), Operand(b, ld=K), Output(y, rs_lo=N), bias=bias, bias_mode=BIAS_ROW, act=ACT_GELU,
         preact=dact, preact_deriv=True)
    gemm(M, N, K, Operand(a, ld=K), Operand(b, ld=K), Output(torch.zeros(M, N), rs_lo=N), bias=bias, bias_mode=BIAS_ROW,
         act=ACT_GELU, preact=pre)
    z = (a @ b.t() + bias[:, None]).requires_grad_()
    yr = torch.nn.functional.gelu(z)
    assert torch.allclose(y, yr.detach(), atol=1e-5) and torch.allclose(pre, z.detach(), atol=1e-5)
    # upstream gradient g = u v^T through both backward flavours
    u, v = torch.randn(M, 1), torch.randn(N, 1)
    g = u @ v.t()
    (dz,) = torch.autograd.grad(yr, z, g)
    out1, out2 = torch.zeros(M, N), torch.zeros(M, N)
    gemm(M, N, 1, Operand(u, ld=1), Operand(v, ld=1), Output(out1, rs_lo=N), act=ACT_MULAUX, resid=dact)
    gemm(M, N, 1, Operand(u, ld=1), Operand(v, ld=1), Output(out2, rs_lo=N), act=ACT_DGELU, resid=pre)
    assert torch.allclose(out1, dz, atol=1e-5) and torch.allclose(out2, dz, atol=1e-5)


@pytest.mark.parametrize("x_cl", [False, True])
@pytest.mark.parametrize("out_layout", [C.NCHW, C.CL])
def test_conv_layout_combinations_match_torch(x_cl, out_layout):
    torch.manual_seed(1)
    B, Ci, Co, H, W = 2, 8, 16, 4, 8
    x = torch.randn(B, Ci, H, W)
    if x_cl:
        x = x.contiguous(memory_format=torch.channels_last)
    w = torch.randn(Co, Ci)
    bias = torch.randn(Co)
    res = torch.randn(B, Co, H, W)
    if out_layout == C.CL:
        res = res.contiguous(memory_format=torch.channels_last)
    wq = C.prep_weight(w, torch.float32)
    y, pre = C._conv_fwd(x, wq, Ci, bias, ACT_GELU, res, True, out_layout)
    ref_pre = torch.nn.functional.conv2d(x, w.view(Co, Ci, 1, 1), bias)
    assert C.layout_of(y) == out_layout
    assert torch.allclose(pre, ref_pre, atol=1e-5)
    assert torch.allclose(y, torch.nn.functional.gelu(ref_pre) + res, atol=1e-5)
    # data gradient (with GELU') and weight gradient
    dy = torch.randn(B, Co, H, W)
    if out_layout == C.CL:
        dy = dy.contiguous(memory_format=torch.channels_last)
    aux = torch.randn(B, Ci, H, W)
    if x_cl:
        aux = aux.contiguous(memory_format=torch.channels_last)
    dx = C._conv_dgrad(dy, wq, Ci, act=ACT_DGELU, aux=aux, x_layout=C.layout_of(x))
    xa = aux.clone().requires_grad_()
    torch.nn.functional.gelu(xa).backward(torch.einsum("bohw,oi->bihw", dy, w))
    assert torch.allclose(dx, xa.grad, atol=1e-4)
    dw = C._conv_wgrad(dy, x, splits=3)
    assert torch.allclose(dw, torch.einsum("bohw,bihw->oi", dy, x), atol=1e-4)


def test_spectral_weight_expand_and_fold_are_adjoint():
    torch.manual_seed(2)
    w = torch.randn(3, 5, 4, dtype=torch.complex64)
    wx = expand_weight(w, torch.float32)
    x = torch.randn(6, dtype=torch.complex64)
    l = 2
    xr = torch.cat([x[:3].real, x[:3].imag])
    out = wx[l] @ xr
    ref = torch.einsum("i,io->o", x[:3], w[:, :, l])
    assert torch.allclose(out[:5], ref.real, atol=1e-5) and torch.allclose(out[5:], ref.imag, atol=1e-5)
    g = torch.randn(4, 10, 6)
    dw = fold_weight_grad(g)
    # <expand(w), g> == Re<w, fold(g)> summed over real and imaginary parts
    lhs = (wx * g).sum()
    rhs = (w.real * dw.real + w.imag * dw.imag).sum()
    assert abs(lhs.item() - rhs.item()) < 1e-3


@pytest.mark.parametrize("adamw", [True, False])
def test_fused_adamw_cpu_path_matches_torch(adamw):
    torch.manual_seed(3)
    p1, p2 = torch.randn(7, 3, requires_grad=True), torch.randn(5, requires_grad=True)
    r1, r2 = p1.detach().clone().requires_grad_(), p2.detach().clone().requires_grad_()
    opt = FusedAdamW([p1, p2], lr=1e-2, weight_decay=0.1, adamw=adamw)
    ref = (torch.optim.AdamW if adamw else torch.optim.Adam)([r1, r2], lr=1e-2, weight_decay=0.1)
    for _ in range(3):
        for p, r in ((p1, r1), (p2, r2)):
            g = torch.randn_like(p)
            p.grad, r.grad = g.clone(), g.clone()
        opt.step(); ref.step()
    assert torch.allclose(p1, r1, atol=1e-6) and torch.allclose(p2, r2, atol=1e-6)


def test_complex_modulus_second_moment():
    torch.manual_seed(4)
    p = torch.randn(4, dtype=torch.complex64, requires_grad=True)
    opt = FusedAdamW([p], lr=1e-2, weight_decay=0.0, complex_mode="modulus")
    p.grad = torch.randn(4, dtype=torch.complex64)
    g = p.grad.clone()
    p0 = p.detach().clone()
    opt.step()
    # first step of Adam: update = lr * g / (|g| + eps)
    expect = p0 - 1e-2 * g / (g.abs() + 1e-8)
    assert torch.allclose(p.detach(), expect, atol=1e-5)


def test_lamb_matches_a_direct_restatement():
    import math
    from makani_b200.ops.optim import LAMB
    torch.manual_seed(0)
    ps = [torch.randn(5, 3, requires_grad=True), torch.randn(4, dtype=torch.complex64, requires_grad=True), torch.zeros(3, requires_grad=True)]
    ref = [p.detach().clone() for p in ps]
    opt = LAMB(ps, lr=1e-2, betas=(0.9, 0.95), eps=1e-6, weight_decay=0.1, max_grad_norm=0.5)
    m = [torch.zeros_like(torch.view_as_real(r) if r.is_complex() else r) for r in ref]
    v = [torch.zeros_like(x) for x in m]
    for step in range(1, 4):
        gs = [torch.randn_like(p) for p in ps]
        for p, g in zip(ps, gs):
            p.grad = g.clone()
        opt.step()
        gr = [torch.view_as_real(g) if g.is_complex() else g for g in gs]
        gnorm = math.sqrt(sum(float(g.square().sum()) for g in gr))
        clip = max(1.0, gnorm / 0.5)
        for i, r in enumerate(ref):
            rr = torch.view_as_real(r) if r.is_complex() else r
            g = gr[i] / clip
            m[i] = 0.9 * m[i] + 0.1 * g
            v[i] = 0.95 * v[i] + 0.05 * g * g
            u = (m[i] / (1 - 0.9 ** step)) / ((v[i] / (1 - 0.95 ** step)).sqrt() + 1e-6) + 0.1 * rr
            pn, un = float(rr.norm()), float(u.norm())
            ratio = pn / un if pn > 0 and un > 0 else 1.0
            rr.sub_(1e-2 * ratio * u)
        for p, r in zip(ps, ref):
            a = torch.view_as_real(p.detach()) if p.is_complex() else p.detach()
            b = torch.view_as_real(r) if r.is_complex() else r
            assert torch.allclose(a, b, rtol=1e-5, atol=1e-6)


def test_sync_params_announces_changed_weights(tmp_path):
    """Parameters are written through `.data`, which no version counter shows: what is derived from them must be dropped."""
    import torch.distributed as dist
    from makani_b200.ops import spectral
    from makani_b200.parallel.helpers import sync_params
    dist.init_process_group("gloo", init_method=f"file://{tmp_path}/store", rank=0, world_size=1)
    try:
        before = spectral._WEIGHT_EPOCH
        sync_params(torch.nn.Linear(2, 2))
        assert spectral._WEIGHT_EPOCH > before
    finally:
        dist.destroy_process_group()


@pytest.mark.parametrize("b,l,m,co,ci", [(1, 5, 6, 8, 16), (2, 9, 7, 6, 4)])
def test_planar_spectral_products_emulated(b, l, m, co, ci):
    """The product with planar weights, its adjoint with a residual and the weight gradient, emulated with the kernel's addressing,
    against complex einsum and against the real block form."""
    from makani_b200.ops.spectral import contract, contract_wgrad2, weight_planes
    torch.manual_seed(l)
    keep = (torch.arange(m)[None] <= torch.arange(l)[:, None]).view(1, l, m, 1)
    t2, dt = torch.randn(b, l, m, 2 * ci) * keep, torch.randn(b, l, m, 2 * co) * keep
    w = torch.randn(ci, co, l, dtype=torch.complex64)
    wp = weight_planes(w, torch.float32)
    assert wp.shape == (l, 2, co, ci)
    cplx = lambda t: torch.complex(*t.chunk(2, dim=-1))  # noqa: E731
    parts = lambda z: torch.cat([z.real, z.imag], dim=-1)  # noqa: E731
    y = contract(t2, wp, False)
    torch.testing.assert_close(y, parts(torch.einsum("blmc,col->bmlo", cplx(t2), w)), atol=1e-5, rtol=1e-5)
    torch.testing.assert_close(y, contract(t2, expand_weight(w, torch.float32), False), atol=1e-5, rtol=1e-5)
    res = torch.randn(b, m, l, 2 * ci)
    dx = contract(dt, wp, True, resid=res)
    torch.testing.assert_close(dx, parts(torch.einsum("blmo,col->bmlc", cplx(dt), w.conj())) + res, atol=1e-5, rtol=1e-5)
    # a block of a larger problem: its first order and degree are m0 and l0
    for l0, m0 in ((0, 0), (2, 3)):
        keep = (torch.arange(m)[None] + m0 <= torch.arange(l)[:, None] + l0).view(1, l, m, 1)
        got = contract_wgrad2(dt * keep, t2 * keep, l0, m0)
        ref = torch.einsum("blmo,blmc->loc", cplx(dt * keep), cplx(t2 * keep).conj())
        torch.testing.assert_close(got, torch.stack([ref.real, ref.imag]), atol=1e-5, rtol=1e-5)


@pytest.mark.parametrize("h,w,mmax,analysis", [(3, 64, 33, True), (3, 64, 32, True), (2, 65, 33, False), (2, 72, 37, True), (2, 80, 41, True),
                                               (2, 90, 46, True), (2, 100, 40, False), (2, 100, 41, True), (2, 96, 49, True),
                                               (3, 128, 20, False), (2, 62, 32, False)])
def test_folded_transforms_equal_the_whole_ones(h, w, mmax, analysis):
    """Every plan the rule folds (odd and even halves, all orders or some, the Nyquist order kept or not) against the whole
    matrices; few points, an odd number of them or few orders stay whole."""
    from makani_b200.ops.spectral import SHTPlan, analyse, dft_analysis, dft_synthesis, synthesise
    plan = SHTPlan(h, w, h, mmax, "legendre-gauss", "cpu", torch.float64)
    assert plan.folds_synthesis == (w >= 64) and plan.folds_analysis == analysis
    g = torch.Generator().manual_seed(w)
    x = torch.randn(2, h, w, 8, generator=g, dtype=torch.float64).permute(0, 3, 1, 2)
    t4 = torch.randn(2, h, 2 * mmax, 8, generator=g, dtype=torch.float64)
    pairs = [(analyse(x, plan), dft_analysis(x, plan.f, False, w, plan.k2)),
             (analyse(x, plan, forward=False), dft_analysis(x, plan.gt, True, plan.k2p, plan.k2)),
             (synthesise(t4, plan), dft_synthesis(t4, plan.gt, False, plan.k2p, w)),
             (synthesise(t4, plan, forward=True), dft_synthesis(t4, plan.f, True, w, w))]
    for got, ref in pairs:      # the tables are fp32 numbers of the same angles
        assert got.shape == ref.shape and (got - ref).abs().max() <= 1e-6 * ref.abs().max()
    # rows that mirror each other hold the same numbers
    for (syn, _), table in plan._folded.items():
        a, b = table.reshape(table.shape[0], 2, -1).unbind(1)
        if syn:
            assert torch.equal(a[1:], a[1:].flip(0)) and torch.equal(b[1:], -b[1:].flip(0))
        else:
            r = torch.arange(2 * mmax)
            mirror = w - r + 2 * (r % 2)
            ok = mirror < 2 * mmax
            sign = (1.0 - 2.0 * (r[ok] % 2))[:, None]
            assert torch.equal(a[mirror[ok]], sign * a[ok]) and torch.equal(b[mirror[ok]], -sign * b[ok])


@pytest.mark.parametrize("w,mmax", [(64, 34), (90, 60), (96, 97)])
def test_orders_past_half_the_points_are_transformed_whole(w, mmax):
    """Orders past w / 2 have no mirror among the rows that a folded analysis writes."""
    from makani_b200.ops.gemm import Operand, Output, gemm_fold
    from makani_b200.ops.spectral import SHTPlan, analyse, dft_analysis
    plan = SHTPlan(4, w, 4, mmax, "legendre-gauss", "cpu", torch.float64)
    x = torch.randn(1, 4, w, 8, dtype=torch.float64).permute(0, 3, 1, 2)
    assert torch.equal(analyse(x, plan), dft_analysis(x, plan.f, False, w, plan.k2))
    assert torch.equal(analyse(x, plan, forward=False), dft_analysis(x, plan.gt, True, plan.k2p, plan.k2))
    # and a product that would leave rows of its output unwritten is refused
    table, d = torch.zeros(2 * mmax, w, dtype=torch.float64), torch.zeros(4, 2 * mmax, 8, dtype=torch.float64)
    with pytest.raises(ValueError):
        gemm_fold(2 * mmax, 2 * (w // 4 + 1), 8, w // 2, w, True, table, w // 2, Operand(x, ld=16, mn_major=True, zs_hi=w * 8), 8,
                  Output(d, rs_lo=8, d_zhi=2 * mmax * 8), zhi_n=4)


def test_a_plan_computes_its_angles_once(monkeypatch):
    """Four folded tables and two whole matrices of one transform hold the same cosines: a new grid is prepared in the time it took with
    the whole matrices alone (64 x 128: 4.7 ms, 6.2 with each table's own cosines)."""
    import numpy as np

    from makani_b200.ops.spectral import SHTPlan
    seen = {"cos": 0, "sin": 0}
    for name in seen:
        def count(x, *args, __f=getattr(np, name), __name=name, **kw):
            seen[__name] += np.size(x)
            return __f(x, *args, **kw)
        monkeypatch.setattr(np, name, count)
    h, w, m = 64, 128, 65
    plan = SHTPlan(h, w, h, m, "legendre-gauss", "cpu")
    assert len(plan._folded) == 4
    assert all(n <= 1.5 * m * w for n in seen.values())


@pytest.mark.parametrize("h,w,mmax", [(3, 64, 33), (3, 64, 32), (2, 65, 33), (2, 72, 37), (2, 80, 41), (2, 90, 46), (2, 100, 41), (2, 96, 49),
                                      (2, 128, 20)])
def test_folded_forms_equal_the_whole_ones(h, w, mmax):
    """The folded forms themselves, also where the rule prefers the whole ones."""
    from makani_b200.ops.spectral import SHTPlan, dft_analysis, dft_synthesis, folded_analysis, folded_synthesis
    plan = SHTPlan(h, w, h, mmax, "legendre-gauss", "cpu", torch.float64)
    g = torch.Generator().manual_seed(w)
    t4 = torch.randn(2, h, 2 * mmax, 8, generator=g, dtype=torch.float64)
    x = torch.randn(2, h, w, 8, generator=g, dtype=torch.float64).permute(0, 3, 1, 2)
    pairs = [(folded_synthesis(t4, plan), dft_synthesis(t4, plan.gt, False, plan.k2p, w)),
             (folded_synthesis(t4, plan, forward=True), dft_synthesis(t4, plan.f, True, w, w))]
    if plan.folds_analysis:
        pairs += [(folded_analysis(x, plan), dft_analysis(x, plan.f, False, w, plan.k2)),
                  (folded_analysis(x, plan, forward=False), dft_analysis(x, plan.gt, True, plan.k2p, plan.k2))]
    for got, ref in pairs:      # the tables are fp32 numbers of the same angles
        assert got.shape == ref.shape and (got - ref).abs().max() <= 1e-6 * ref.abs().max()


def test_folding_where_it_pays():
    """Both sides of the rule, at the grids of the recipes and where the folded form was measured to be slower."""
    from makani_b200.ops.gemm import plain_columns
    from makani_b200.ops.spectral import folding_pays
    synthesis = lambda w, m, c: folding_pays(w, w // 2 + 1, 2 * m, m, c)  # noqa: E731
    analysis = lambda w, m, c: folding_pays(2 * m, 2 * (w // 4 + 1), w, w // 2, c)  # noqa: E731
    assert [plain_columns(c) for c in (8, 128, 136, 200, 256, 264, 384, 640, 776)] == [128, 128, 192, 256, 256, 192, 192, 256, 256]
    for args in ((1440, 241, 384), (480, 241, 384), (720, 361, 384), (1440, 64, 136), (1440, 361, 72)):
        assert synthesis(*args)
    for args in ((256, 129, 384), (128, 32, 768), (64, 33, 384), (360, 8, 384), (256, 32, 320)):
        assert not synthesis(*args)
    for args in ((480, 241, 384), (720, 361, 384), (360, 181, 200)):
        assert analysis(*args)
    for args in ((64, 33, 384), (96, 40, 768), (256, 97, 384)):
        assert not analysis(*args)
