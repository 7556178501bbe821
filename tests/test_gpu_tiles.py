"""Tile widths, remainders and the streaming kernels at the sizes where they can go wrong, against plain PyTorch (-m gpu)."""

import pytest
import torch

from makani_b200.ops import _ext
from makani_b200.ops.gemm import (ACT_DGELU, ACT_DRELU, ACT_DSHRINK, ACT_GELU, ACT_MULAUX, ACT_NONE, ACT_RELU, ACT_SHRINK, BIAS_COL,
                                  BIAS_ROW, Operand, Output, Tri, gemm)
from test_gpu_kernels import _dev, _rel, _run_both

pytestmark = pytest.mark.gpu

BF16 = 2.0 ** -8      # spacing of bf16 relative to the value: a rounded result is within half of it of the fp32 one


@pytest.mark.parametrize("pair", [False, True])
@pytest.mark.parametrize("w_mn", [False, True])
@pytest.mark.parametrize("n", [8, 136, 192, 200, 384, 776])
@pytest.mark.parametrize("epi", ["plain", "gelu", "relu", "gelu_pre", "gelu_deriv", "resid", "mul", "dgelu"])
def test_gemm_192_column_tiles(pair, w_mn, n, epi):
    """192-column tiles on single CTAs and pairs, both majors of the weight, every specialised epilogue, N from one vector
    over one tile and its edges to several tiles, ragged rows (many tiles per CTA: test_gemm_many_tiles_per_cta)."""
    dev = _dev()
    k = 520 if pair else 72           # pairs run from K = 512 on, and with fewer where the tiles are many
    m = 128 * 9 + 40
    torch.manual_seed(n + k)
    x = torch.randn(2, m, k, device=dev).to(torch.bfloat16)
    w = (torch.randn(n, k, device=dev) / k ** 0.5).to(torch.bfloat16)
    op = Operand(w.t().contiguous(), ld=n, mn_major=True) if w_mn else Operand(w, ld=k)
    aux = torch.randn(2, m, n, device=dev).to(torch.bfloat16) if epi in ("resid", "mul", "dgelu") else None
    pre = torch.zeros(2, m, n, device=dev, dtype=torch.bfloat16) if epi in ("gelu_pre", "gelu_deriv") else None
    act = {"plain": ACT_NONE, "resid": ACT_NONE, "relu": ACT_RELU, "mul": ACT_MULAUX, "dgelu": ACT_DGELU}.get(epi, ACT_GELU)
    bias = None if epi in ("mul", "dgelu") else torch.randn(n, device=dev)
    d = torch.zeros(2, m, n, device=dev, dtype=torch.bfloat16)
    outs = _run_both(m, n, k, Operand(x, ld=k, zs_lo=m * k), op, Output(d, rs_lo=n, d_zlo=m * n), zlo_n=2, bias=bias,
                     bias_mode=BIAS_COL, act=act, resid=aux, preact=pre, preact_deriv=epi == "gelu_deriv", bn=192)
    for got, ref in outs:
        assert _rel(got, ref) < BF16


@pytest.mark.parametrize("tokens", [64 * 3, 64 * 400 + 8, 128 * 150 * 3])
def test_gemm_one_box_per_tile_over_many_tiles(tokens):
    """Outputs of one 64-column box per tile with a one-slab k loop: the store of a tile must have read its staging box
    before the next tile, which follows at once, is written there."""
    dev = _dev()
    torch.manual_seed(tokens)
    x = torch.randn(tokens, 16, device=dev).to(torch.bfloat16)
    w = torch.randn(16, 16, device=dev).to(torch.bfloat16)
    for _ in range(3):
        d = torch.empty(tokens, 16, device=dev, dtype=torch.bfloat16)
        gemm(tokens, 16, 16, Operand(x, ld=16), Operand(w, ld=16, mn_major=True), Output(d, rs_lo=16))
        assert _rel(d, x.float() @ w.float()) < BF16
    _ext.check_device_errors(dev)


@pytest.mark.parametrize("bn", [0, 128, 192, 256])
@pytest.mark.parametrize("co,ci,t", [(16, 8, 40), (384, 384, 5000), (200, 392, 64 * 9), (768, 384, 20000)])
def test_gemm_chosen_splits(bn, co, ci, t):
    """Weight gradients with the split-k factor left to the launcher; K from under one slab to many per split."""
    dev = _dev()
    torch.manual_seed(co + t)
    dy = torch.randn(t, co, device=dev).to(torch.bfloat16)
    x = torch.randn(t, ci, device=dev).to(torch.bfloat16)
    dw = torch.zeros(co, ci, device=dev)
    gemm(co, ci, t, Operand(dy, ld=co, mn_major=True), Operand(x, ld=ci, mn_major=True), Output(dw, rs_lo=ci), accumulate=True,
         splits=0, bn=bn)
    # fp32 sums of t exact products
    assert _rel(dw, dy.double().t() @ x.double()) < 2.0 ** -24 * max(t, 64) ** 0.5 * 4
    _ext.check_device_errors(dev)


@pytest.mark.parametrize("b", [1, 2, 3])
@pytest.mark.parametrize("i,o,x,y", [(1, 1, 1, 1), (5, 3, 4, 4), (4, 8, 16, 18), (9, 6, 7, 37), (8, 12, 40, 41)])
def test_diagonal_contraction_edges(b, i, o, x, y):
    """Odd and even numbers of modes (8- and 16-byte accesses), channel counts around the four per thread, odd batches."""
    from makani_b200.ops.spectral_modes import contract_diagonal
    dev = _dev()
    g = torch.Generator(dev).manual_seed(i * o + x)
    rnd = lambda *s: torch.randn(*s, dtype=torch.complex64, device=dev, generator=g)  # noqa: E731
    a, w, dy = rnd(b, i, x, y).requires_grad_(), rnd(i, o, x, y).requires_grad_(), rnd(b, o, x, y)
    out = contract_diagonal(a, w)
    got = [out] + list(torch.autograd.grad(out, [a, w], dy))
    ad, wd = a.detach().to(torch.complex128).requires_grad_(), w.detach().to(torch.complex128).requires_grad_()
    r = torch.einsum("bixy,ioxy->boxy", ad, wd)
    ref = [r] + list(torch.autograd.grad(r, [ad, wd], dy.to(torch.complex128)))
    for p, q in zip(got, ref):
        assert _rel(torch.view_as_real(p.detach()), torch.view_as_real(q.detach())) < 2.0 ** -21


@pytest.mark.parametrize("rows,c", [(1, 8), (7, 16), (2049, 24), (5000, 256), (777, 384), (300, 3072), (33, 4104), (100000, 128)])
def test_column_sums(rows, c):
    from makani_b200.ops.norm import row_sums
    dev = _dev()
    x = torch.randn(rows, c, device=dev, generator=torch.Generator(dev).manual_seed(rows)).to(torch.bfloat16)
    got, ref = row_sums(x, c).double(), x.double().sum(0)
    # fp32 summation: error within rows * 2^-24 of the sum of magnitudes, in practice its square root
    assert ((got - ref).abs() <= 2.0 ** -24 * 8 * max(rows, 4) ** 0.5 * x.double().abs().sum(0) / rows ** 0.5 + 1e-6).all()


@pytest.mark.parametrize("ci,co,n", [(8, 3, 2), (64, 5, 32), (72, 16, 34), (136, 8, 64), (12, 4, 30), (16, 4, 33)])
def test_spectral_weight_layouts(ci, co, n):
    """Weight expansion and gradient folding: tile edges in channels and degrees, and the sizes that keep the scalar kernels."""
    from makani_b200.ops.spectral import expand_weight, fold_weight_grad2
    dev = _dev()
    w = torch.randn(ci, co, n, dtype=torch.complex64, device=dev)
    assert torch.equal(expand_weight(w).cpu(), expand_weight(w.cpu()))
    dw = torch.randn(2, n, co, ci, device=dev)
    assert torch.equal(fold_weight_grad2(dw).cpu(), fold_weight_grad2(dw.cpu()))


def test_mlp_without_gradients_equals_training_forward():
    """The forward pass that writes no GELU' gives the same values, in both layouts of the tokens."""
    from makani_b200.models.common.layers import MLP
    from makani_b200.models.networks.afnonet import Mlp
    dev = _dev()
    torch.manual_seed(3)
    m, x = MLP(16, hidden_features=40).to(dev), torch.randn(2, 16, 24, 40, device=dev).to(torch.bfloat16)
    x = x.contiguous(memory_format=torch.channels_last)
    t, z = Mlp(24, hidden_features=96).to(dev), torch.randn(3, 50, 24, device=dev).to(torch.bfloat16)
    for net, inp in ((m, x), (t, z)):
        y = net(inp)
        assert y.requires_grad
        with torch.no_grad():
            assert torch.equal(net(inp), y)
    _ext.check_device_errors(dev)


def test_kept_weights_follow_the_parameter():
    """Expanded weights kept for inference belong to one parameter: not to the next one in the same memory, nor to it once
    it has changed."""
    from makani_b200.ops.spectral import expand_weight
    dev = _dev()
    seen = set()
    for k in range(4):
        w = torch.full((8, 8, 16), complex(k, -k), dtype=torch.complex64, device=dev)
        seen.add(w.data_ptr())
        for _ in range(2):
            assert torch.equal(expand_weight(w, keep=True).cpu(), expand_weight(w.cpu()))
        w.mul_(2.0)
        assert torch.equal(expand_weight(w, keep=True).cpu(), expand_weight(w.cpu()))
        del w
    assert len(seen) < 4      # the allocator did hand out the same memory again


@pytest.mark.parametrize("act", ["none", "gelu"])
@pytest.mark.parametrize("b,c,h,w", [(1, 8, 1, 8), (2, 16, 32, 64), (1, 24, 9, 16), (1, 32, 40, 80), (1, 264, 50, 96), (1, 1024, 20, 40)])
def test_instance_norm_channel_counts(b, c, h, w, act):
    """Channel counts below and above a warp of 16-byte vectors (powers of two and not), fewer tokens than rows in flight."""
    from makani_b200.ops.norm import instance_norm
    dev = _dev()
    g = torch.Generator(dev).manual_seed(c)
    x = (torch.randn(b, h, w, c, device=dev, generator=g) * 1.5 + 0.7).to(torch.bfloat16).permute(0, 3, 1, 2).requires_grad_()
    dy = torch.randn(b, h, w, c, device=dev, generator=g).to(torch.bfloat16).permute(0, 3, 1, 2)
    wt, bs = (torch.rand(c, device=dev, generator=g) + 0.5).requires_grad_(), torch.randn(c, device=dev, generator=g).requires_grad_()
    y = instance_norm(x, wt, bs, 1e-6, act)
    got = [y] + list(torch.autograd.grad(y, [x, wt, bs], dy))
    xd, wd, bd = x.detach().double().requires_grad_(), wt.detach().double().requires_grad_(), bs.detach().double().requires_grad_()
    yr = torch.nn.functional.instance_norm(xd, None, None, wd, bd, True, 0.0, 1e-6)
    yr = torch.nn.functional.gelu(yr) if act == "gelu" else yr
    ref = [yr] + list(torch.autograd.grad(yr, [xd, wd, bd], dy.double()))
    for a, r in zip(got, ref):
        assert _rel(a, r) < BF16


@pytest.mark.parametrize("b,c,h,w", [
    (1, 384, 1, 1), (1, 8, 1, 3),            # fewer rows than threads
    (1, 384, 7, 7), (1, 384, 1, 50), (1, 384, 3, 17),      # a stage of 50 (forward) or 40 and 24 rows (backward): one less, full, one more
    (1, 384, 130, 151),                      # several stages per CTA, the last one ragged
    (3, 8, 61, 67), (1, 16, 300, 301),       # many rows per thread column: sums in two steps
    (2, 1000, 19, 23), (1, 1024, 40, 41),    # fewest rows per stage
    (149, 16, 5, 9),                         # more images than SMs
])
def test_instance_norm_rows_of_the_ring(b, c, h, w):
    """Both passes, with a mean as large as the spread, against float64: statistics to fp32, fields to one rounding to bf16."""
    from makani_b200.ops import _ext
    dev = _dev()
    g = torch.Generator(dev).manual_seed(c + h)
    x, dy = ((torch.randn(b, h, w, c, device=dev, generator=g) + 1.0).bfloat16().permute(0, 3, 1, 2) for _ in range(2))
    wt, bi = (torch.randn(c, device=dev, generator=g) for _ in range(2))
    ext, eps, n = _ext.require(), 1e-2, float(h * w)
    for act in (0, 1):
        y, stats, wf, bf = ext.norm_forward(x, wt, bi, eps, act, n)
        dx, dw, db = ext.norm_backward(x, dy, wf, bf, stats, True, act, n)
        xd, wd, bd = x.double().requires_grad_(), wt.double().requires_grad_(), bi.double().requires_grad_()
        mean = xd.mean((2, 3), keepdim=True)
        rstd = 1.0 / torch.sqrt((xd - mean).square().mean((2, 3), keepdim=True) + eps)
        yd = (xd - mean) * rstd * wd[:, None, None] + bd[:, None, None]
        yd = torch.nn.functional.gelu(yd) if act else yd
        want = torch.autograd.grad(yd, [xd, wd, bd], dy.double())
        assert (stats[..., 0].double() - mean[..., 0, 0]).abs().max() < 1e-5
        assert (stats[..., 1].double() / rstd[..., 0, 0] - 1.0).abs().max() < 1e-5
        # half a unit of 2^-8 per value; GELU is 5.5e-5 off, its derivative 2e-4 times (1 + |x|), at outputs of order 1
        assert (y.double() - yd).norm() < (2.0 ** -8 + (1e-4 if act else 0.0)) * yd.norm() + 1e-6
        scale = (dy.double().norm() * (rstd * wd[:, None, None]).abs().max())      # dx is a difference of terms of this size
        assert (dx.double() - want[0]).norm() < 2.0 ** -8 * want[0].norm() + (2e-3 if act else 1e-5) * scale
        for got, ref, size in ((dw, want[1], (dy.double() * (xd - mean) * rstd)), (db, want[2], dy.double())):
            bound = size.abs().sum((0, 2, 3)).norm()
            assert (got.double() - ref).norm() <= (2e-3 if act else 1e-5) * bound
    _ext.check_device_errors(dev)


@pytest.mark.parametrize("rd,m", [(2, 182), (2, 6), (4, 132), (32, 96), (2, 181), (3, 180)])
@pytest.mark.parametrize("epi", ["plain", "resid", "gelu_pre"])
def test_gemm_split_rows(rd, m, epi):
    """Rows addressed as (r / rd, r % rd): as a dimension of the tensor maps where rd is a power of two that divides the rows,
    by the generic epilogue otherwise."""
    dev = _dev()
    k, n, hi = 72, 136, (m + rd - 1) // rd
    torch.manual_seed(rd * m)
    a, b = torch.randn(3, m, k, device=dev).to(torch.bfloat16), torch.randn(n, k, device=dev).to(torch.bfloat16)
    shape = (rd, 3, hi, n)            # the low part of the row index is the slowest dimension
    lay = dict(rs_lo=3 * hi * n, rdiv=rd, rs_hi=n, d_zlo=hi * n)
    d = torch.zeros(shape, device=dev, dtype=torch.bfloat16)
    aux = torch.randn(shape, device=dev).to(torch.bfloat16) if epi == "resid" else None
    pre = torch.zeros_like(d) if epi == "gelu_pre" else None
    outs = _run_both(m, n, k, Operand(a, ld=k, zs_lo=m * k), Operand(b, ld=k), Output(d, **lay), zlo_n=3, resid=aux, preact=pre,
                     act=ACT_GELU if epi == "gelu_pre" else ACT_NONE)
    for got, ref in outs:
        assert _rel(got, ref) < BF16


@pytest.mark.parametrize("m", [1, 40, 300])
@pytest.mark.parametrize("epi", ["plain", "resid", "fp32"])
def test_gemm_split_rows_of_one(m, epi):
    """rdiv = 1: row r lies at r * rs_hi, and rs_lo, a shorter or a longer distance, is never used."""
    dev = _dev()
    k, n = 72, 136
    torch.manual_seed(m)
    a, b = torch.randn(m, k, device=dev).to(torch.bfloat16), torch.randn(n, k, device=dev).to(torch.bfloat16)
    for lo in (8, 4 * n):
        d = torch.zeros(m, 2 * n, device=dev, dtype=torch.float32 if epi == "fp32" else torch.bfloat16)
        aux = torch.randn(m, 2 * n, device=dev).to(torch.bfloat16) if epi == "resid" else None
        outs = _run_both(m, n, k, Operand(a, ld=k), Operand(b, ld=k), Output(d, rs_lo=lo, rdiv=1, rs_hi=2 * n), resid=aux)
        for got, ref in outs:
            assert _rel(got, ref) < BF16


@pytest.mark.parametrize("z", [1, 2, 91, 800])
@pytest.mark.parametrize("co,ci,k", [(16, 24, 8), (192, 192, 90), (136, 264, 200)])
def test_gemm_batches_summed_inside_tiles(z, co, ci, k):
    """Batches that add into one output: one, a few and many."""
    dev = _dev()
    g = torch.Generator(dev).manual_seed(z + co)
    a = torch.randn(2, z, k, co, device=dev, generator=g).to(torch.bfloat16)
    b = torch.randn(2, z, k, ci, device=dev, generator=g).to(torch.bfloat16)
    d = torch.zeros(2, co, ci, device=dev)
    gemm(co, ci, k, Operand(a, ld=co, mn_major=True, zs_lo=z * k * co, zs_hi=k * co),
         Operand(b, ld=ci, mn_major=True, zs_lo=z * k * ci, zs_hi=k * ci), Output(d, rs_lo=ci, d_zlo=co * ci), zlo_n=2, zhi_n=z,
         accumulate=True, splits=0)
    _ext.check_device_errors(dev)
    assert _rel(d, torch.einsum("lzko,lzki->loi", a.double(), b.double())) < 2.0 ** -24 * max(z * k, 64) ** 0.5 * 4


@pytest.mark.parametrize("nb,bs,hid,bias", [(1, 8, 8, True), (3, 24, 40, True), (8, 96, 96, False), (2, 72, 32, True)])
def test_afno_weight_packing(nb, bs, hid, bias):
    """Packing of both layers' weights and its adjoint against the plain formulation, block sizes around the 32-wide tiles."""
    from makani_b200.ops.afno import _fold, _pack
    dev = _dev()
    g = torch.Generator(dev).manual_seed(bs)
    r = lambda *s: torch.randn(*s, device=dev, generator=g)  # noqa: E731
    ws = (r(2, nb, bs, hid), r(2, nb, hid, bs))
    bz = (r(2, nb, hid), r(2, nb, bs)) if bias else (None, None)
    got, ref = _pack(ws, bz, torch.bfloat16), _pack([w.cpu() for w in ws], [None if b is None else b.cpu() for b in bz], torch.bfloat16)
    for p, q in zip(got[0] + got[1], ref[0] + ref[1]):
        assert (p is None and q is None) or torch.equal(p.cpu(), q)
    dw, db = [r(nb, 2 * hid, 2 * bs), r(nb, 2 * bs, 2 * hid)], [r(nb, 2 * hid), r(nb, 2 * bs)]
    shapes = [(2, nb, bs, hid), (2, nb, hid, bs)]
    got = _fold(dw, db, shapes, (bias, bias))
    ref = _fold([t.cpu() for t in dw], [t.cpu() for t in db], shapes, (bias, bias))
    for p, q in zip(got[0] + got[1], ref[0] + ref[1]):
        assert (p is None and q is None) or torch.equal(p.cpu(), q)


@pytest.mark.parametrize("rows,cols", [(1, 1), (16, 5), (73, 384), (384, 74), (8, 16), (300, 1001)])
def test_convolution_weight_operand(rows, cols):
    from makani_b200.ops.conv import prep_weight
    dev = _dev()
    w = torch.randn(rows, cols, 1, 1, device=dev)
    assert torch.equal(prep_weight(w).cpu(), prep_weight(w.cpu()))


@pytest.mark.parametrize("acc", [False, True])
@pytest.mark.parametrize("m,n,k", [(128, 32, 64), (200, 36, 72), (392, 384, 40), (130, 772, 520)])
def test_gemm_fp32_output(acc, m, n, k):
    """fp32 results stored and added through TMA: half boxes, ragged rows and columns, single CTAs and pairs, added to what
    is there."""
    dev = _dev()
    g = torch.Generator(dev).manual_seed(m + n)
    pad, pm = (n + 7) // 8 * 8, (m + 7) // 8 * 8
    a = torch.randn(5, k, pm, device=dev, generator=g).to(torch.bfloat16)
    b = torch.randn(5, k, pad, device=dev, generator=g).to(torch.bfloat16)
    d = torch.full((5, m, n), 3.0 if acc else float("nan"), device=dev)
    gemm(m, n, k, Operand(a, ld=pm, mn_major=True, zs_hi=k * pm), Operand(b, ld=pad, mn_major=True, zs_hi=k * pad),
         Output(d, rs_lo=n, d_zhi=m * n), zhi_n=5, accumulate=acc)
    _ext.check_device_errors(dev)
    ref = torch.einsum("zkm,zkn->zmn", a[..., :m].double(), b[..., :n].double()) + (3.0 if acc else 0.0)
    assert _rel(d, ref) < 2.0 ** -24 * max(k, 64) ** 0.5 * 4


@pytest.mark.parametrize("b,l,m,co,ci", [(1, 5, 6, 8, 8), (2, 33, 34, 24, 40), (1, 70, 66, 72, 200), (1, 140, 141, 384, 136)])
def test_planar_spectral_products(b, l, m, co, ci):
    """Product with the planar weights, its adjoint (with a residual) and the weight gradient against complex einsum: parts that
    are no whole slabs or tiles, one to three row tiles, orders above the degree skipped."""
    from makani_b200.ops.spectral import contract, contract_wgrad2, weight_planes
    dev = _dev()
    g = torch.Generator(dev).manual_seed(l * ci)
    keep = (torch.arange(m, device=dev)[None] <= torch.arange(l, device=dev)[:, None]).view(1, l, m, 1)
    t2 = (torch.randn(b, l, m, 2 * ci, device=dev, generator=g) * keep).to(torch.bfloat16)
    dt = (torch.randn(b, l, m, 2 * co, device=dev, generator=g) * keep).to(torch.bfloat16)
    w = torch.randn(ci, co, l, dtype=torch.complex64, device=dev, generator=g)
    wp = weight_planes(w)
    wd = torch.complex(wp[:, 0].double(), wp[:, 1].double())                   # [l, co, ci], as rounded
    cplx = lambda t: torch.complex(t[..., : t.shape[-1] // 2].double(), t[..., t.shape[-1] // 2:].double())  # noqa: E731
    parts = lambda z: torch.cat([z.real, z.imag], dim=-1)  # noqa: E731
    y = contract(t2, wp, False)
    assert _rel(y, parts(torch.einsum("blmc,loc->bmlo", cplx(t2), wd))) < BF16
    res = torch.randn(b, m, l, 2 * ci, device=dev, generator=g).to(torch.bfloat16)
    dx = contract(dt, wp, True, resid=res)
    assert _rel(dx, parts(torch.einsum("blmo,loc->bmlc", cplx(dt), wd.conj())) + res.double()) < BF16
    dw = contract_wgrad2(dt, t2)
    ref = torch.einsum("blmo,blmc->loc", cplx(dt), cplx(t2).conj())
    assert _rel(dw, torch.stack([ref.real, ref.imag])) < 2.0 ** -24 * max(b * m, 64) ** 0.5 * 4
    _ext.check_device_errors(dev)


@pytest.mark.parametrize("co", [4, 12, 20])
def test_planar_product_refuses_parts_off_a_vector(co):
    """The adjoint reads the imaginary part of its operand at element co: refused by the host where that is no 16-byte boundary."""
    from makani_b200.ops.spectral import contract
    dev = _dev()
    dt = torch.zeros(1, 6, 7, 2 * co, device=dev, dtype=torch.bfloat16)
    wp = torch.zeros(6, 2, co, 16, device=dev, dtype=torch.bfloat16)
    with pytest.raises(RuntimeError, match="multiples of 8"):
        contract(dt, wp, True)


@pytest.mark.parametrize("z", [1, 7])
@pytest.mark.parametrize("opt", ["bias_row", "bias_col", "relu"])
def test_chosen_splits_leave_the_epilogue_alone(z, opt):
    """splits = 0 with a bias or an activation: applied to each whole product, never to the partial sums of one."""
    dev = _dev()
    m, n, k = 136, 72, 64 * 40
    g = torch.Generator(dev).manual_seed(z)
    a = torch.randn(z, k, m, device=dev, generator=g).to(torch.bfloat16)
    b = torch.randn(z, k, n, device=dev, generator=g).to(torch.bfloat16)
    bias = None if opt == "relu" else torch.randn(m if opt == "bias_row" else n, device=dev, generator=g) * 100
    d = torch.zeros(m, n, device=dev)
    gemm(m, n, k, Operand(a, ld=m, mn_major=True, zs_hi=k * m), Operand(b, ld=n, mn_major=True, zs_hi=k * n), Output(d, rs_lo=n), zhi_n=z,
         accumulate=True, splits=0, bias=bias, bias_mode=BIAS_ROW if opt == "bias_row" else BIAS_COL,
         act=ACT_RELU if opt == "relu" else ACT_NONE)
    _ext.check_device_errors(dev)
    ref = torch.einsum("zkm,zkn->zmn", a.double(), b.double())
    ref = torch.relu(ref) if opt == "relu" else ref + (bias[:, None] if opt == "bias_row" else bias[None, :]).double()
    # fp32 sums of k exact products, truncated by the tensor core at every 16 of them
    assert _rel(d, ref.sum(0)) < 2.0 ** -24 * (k / 16)


@pytest.mark.parametrize("sign", ["zero_mean", "one_signed"])
@pytest.mark.parametrize("co,ci,t", [(16, 16, 4096), (64, 64, 115200), (384, 768, 200000), (384, 384, 1038240), (768, 3072, 16200)])
def test_chosen_splits_keep_the_sums_short(sign, co, ci, t):
    """The tensor core truncates its running sum at every 16 products: the chosen factor gives chains no longer, and sums no less
    exact, than twice as many 128 x 256 tiles as SMs would."""
    dev = _dev()
    g = torch.Generator(dev).manual_seed(co)
    rnd = lambda *s: torch.randn(*s, device=dev, generator=g)  # noqa: E731
    dy, x = (rnd(t, co), rnd(t, ci)) if sign == "zero_mean" else (rnd(t, co).abs(), rnd(t, ci).abs())
    dy, x = dy.to(torch.bfloat16), x.to(torch.bfloat16)
    ref = torch.zeros(co, ci, dtype=torch.float64, device=dev)
    for p, q in zip(dy.split(131072), x.split(131072)):
        ref += p.double().t() @ q.double()
    tiles = ((co + 127) // 128) * ((ci + 255) // 256)
    sms = torch.cuda.get_device_properties(dev).multi_processor_count
    err = {}
    for splits in (0, min((t + 63) // 64, (2 * sms + tiles - 1) // tiles)):
        dw = torch.zeros(co, ci, device=dev)
        gemm(co, ci, t, Operand(dy, ld=co, mn_major=True), Operand(x, ld=ci, mn_major=True), Output(dw, rs_lo=ci), accumulate=True,
             splits=splits)
        err[splits] = _rel(dw, ref)
    _ext.check_device_errors(dev)
    chosen, least = err.pop(0), next(iter(err))
    # (the order of the fp32 additions between the chains differs from run to run: 2^-24 each, at random)
    assert chosen <= err[least] * 1.02 + 2.0 ** -24
    assert chosen <= t / least / 16 * 2.0 ** -23 + 2.0 ** -23


@pytest.mark.parametrize("sign", ["zero_mean", "one_signed"])
def test_batches_into_one_output_keep_their_own_sums(sign):
    """A batch is summed by itself and added in fp32: the tensor core's truncation does not grow with the number of batches."""
    dev = _dev()
    z, k, n = 91, 90, 192
    g = torch.Generator(dev).manual_seed(5)
    a, b = (torch.randn(z, k, n, device=dev, generator=g) for _ in range(2))
    a, b = (a.abs(), b.abs()) if sign == "one_signed" else (a, b)
    a, b = a.to(torch.bfloat16), b.to(torch.bfloat16)
    d = torch.zeros(n, n, device=dev)
    gemm(n, n, k, Operand(a, ld=n, mn_major=True, zs_hi=k * n), Operand(b, ld=n, mn_major=True, zs_hi=k * n), Output(d, rs_lo=n), zhi_n=z,
         accumulate=True, splits=0)
    _ext.check_device_errors(dev)
    # k / 16 truncations per batch, then z roundings of 2^-24 at random
    assert _rel(d, torch.einsum("zko,zki->oi", a.double(), b.double())) < (k / 16) * 2.0 ** -24 + 2.0 ** -24 * z ** 0.5 / 4


def _spectral_layer(dev, seed=3):
    from makani_b200.models.common.spectral_convolution import SpectralConv
    from makani_b200.sht import InverseRealSHT, RealSHT
    torch.manual_seed(seed)
    fwd = RealSHT(17, 32, lmax=16, mmax=17, grid="equiangular").to(dev)
    inv = InverseRealSHT(17, 32, lmax=16, mmax=17, grid="equiangular").to(dev)
    m = SpectralConv(fwd, inv, 16, 16, operator_type="dhconv").to(dev)
    x = torch.randn(1, 17, 32, 16, device=dev).to(torch.bfloat16).permute(0, 3, 1, 2)
    return m, x


def _count_expansions(monkeypatch):
    from makani_b200.ops import spectral
    made, real = [], spectral._planes
    monkeypatch.setattr(spectral, "_planes", lambda w, dtype: made.append(1) or real(w, dtype))
    return made


def test_captured_pass_expands_its_own_weights(monkeypatch):
    """A pass captured after eager ones, then weights that change and an eager pass that drops the kept expansion: the replay
    reads the new weights, from memory of its own; and what a capture made serves no eager pass."""
    dev = _dev()
    m, x = _spectral_layer(dev)
    made = _count_expansions(monkeypatch)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.no_grad(), torch.cuda.stream(side):
        m(x)
        m(x)
        assert len(made) == 1                                  # kept between eager passes of one stream
        side.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=side):
            y = m(x)[0]
        assert len(made) == 2
        for k in range(3):
            m.weight.copy_(torch.randn_like(m.weight))
            want = m(x)[0].clone()
            junk = [torch.randn_like(m.weight) for _ in range(4)]       # the dropped expansion's memory is handed out again
            g.replay()
            assert torch.equal(y, want), k
            del junk
        assert len(made) == 5
        m.weight.data.mul_(2.0)
        from makani_b200.ops.spectral import note_weights_changed
        note_weights_changed()
        want = m(x)[0]
        g.replay()
        assert torch.equal(y, want)
    torch.cuda.synchronize()
    _ext.check_device_errors(dev)


def test_kept_weights_serve_one_stream(monkeypatch):
    """An expansion may still be in flight on the stream that makes it: another stream makes its own."""
    dev = _dev()
    m, x = _spectral_layer(dev)
    made = _count_expansions(monkeypatch)
    with torch.no_grad():
        a = m(x)[0]
        torch.cuda.synchronize()
        side = torch.cuda.Stream()
        with torch.cuda.stream(side):
            b = m(x)[0]
        torch.cuda.synchronize()
    assert len(made) == 2 and torch.equal(a, b)


def test_launch_count_counts_launches():
    dev = _dev()
    n = _ext.launch_count()
    _ext.require().stream_state(dev.index)
    assert _ext.launch_count() == n


def test_recorded_passes_share_one_expansion(monkeypatch):
    """The steps of a roll-out share one expansion, which goes with the last of their graphs; weights changed in place, announced or
    not once the graphs are gone, or a new parameter in the same memory, are expanded anew."""
    from makani_b200.ops import spectral
    dev = _dev()
    m, x = _spectral_layer(dev)
    made = _count_expansions(monkeypatch)

    def rollout(steps, inp=x):
        y = inp
        for _ in range(steps):
            y = m(y)[0]
        return y

    y = rollout(3)
    assert len(made) == 1
    g = torch.autograd.grad(y.float().square().mean(), m.weight)[0]
    assert len(spectral._RECORDED) == 1 and next(iter(spectral._RECORDED.values()))[1]() is None      # nothing outlives the graph
    monkeypatch.setattr(spectral, "_RECORDED", type(spectral._RECORDED)())
    real = spectral._kept
    with monkeypatch.context() as mp:
        mp.setattr(spectral, "_kept", lambda w, dtype, make, keep, share: real(w, dtype, make, False, False))
        y2 = rollout(3)
        g2 = torch.autograd.grad(y2.float().square().mean(), m.weight)[0]
    assert torch.equal(y, y2) and torch.equal(g, g2)
    del y, y2
    a = rollout(1)
    with torch.no_grad():
        m.weight.mul_(1.5)                  # while a graph lives: the version shows it
    b = rollout(1)
    assert not torch.equal(a, b)
    del a, b
    m.weight.data.mul_(0.5)                 # unannounced: with no graph alive nothing is kept that this could make stale
    got = rollout(1)
    spectral.note_weights_changed()
    with torch.no_grad():
        assert torch.equal(got, m(x)[0])
    del got
    seen = set()
    for k in range(4):                      # new parameters, one after the other in the same memory
        m.weight = torch.nn.Parameter(torch.full_like(m.weight.detach(), complex(k, -k)))
        seen.add(m.weight.data_ptr())
        got = rollout(1)
        with torch.no_grad():
            spectral.note_weights_changed()
            assert torch.equal(got, m(x)[0]), k
        del got
    _ext.check_device_errors(dev)


def test_captured_training_shares_inside_the_capture(monkeypatch):
    """Two forward passes, their backward pass and an update in one graph: one expansion per replay, of that replay's weights."""
    dev = _dev()
    m, x = _spectral_layer(dev)
    made = _count_expansions(monkeypatch)

    def step():
        y = m(m(x)[0])[0]
        g = torch.autograd.grad(y.float().square().mean(), m.weight)[0]
        with torch.no_grad():
            m.weight.add_(g, alpha=-10.0)
        return y

    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    start = m.weight.detach().clone()
    with torch.cuda.stream(side):
        want = [step().detach().clone() for _ in range(4)]
        assert len(made) == 4
        with torch.no_grad():
            m.weight.copy_(start)
        side.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            y = step()
        assert len(made) == 5
        for k in range(4):
            graph.replay()
            assert _rel(y, want[k]) < 1e-6, k
        assert _rel(want[3], want[0]) > 1e-3
    torch.cuda.synchronize()
    _ext.check_device_errors(dev)


@pytest.mark.parametrize("shift", [1, 4, 8])
def test_linear_bias_alone_trains(shift):
    """A linear layer with a frozen weight on inputs without gradient: its bias trains also where the gradient handed in is no
    multiple of 16 bytes into its storage."""
    from makani_b200.ops.linear import linear_lastdim
    dev = _dev()
    x = torch.randn(3, 50, 24, device=dev).to(torch.bfloat16)
    w, b = torch.randn(16, 24, device=dev), torch.zeros(16, device=dev, requires_grad=True)
    dy = torch.randn(3 * 50 * 16 + shift, device=dev).to(torch.bfloat16)[shift:].view(3, 50, 16)
    g, = torch.autograd.grad(linear_lastdim(x, w, b), b, dy)
    assert _rel(g, dy.double().sum((0, 1))) < 2.0 ** -22


@pytest.mark.parametrize("rows,c", [(1, 8), (2049, 24), (5000, 256), (16200, 768), (33, 4104), (1000003, 16), (115200, 384)])
def test_column_sums_repeat_themselves(rows, c):
    """One fixed order of the additions: the same bits on every call, whatever else keeps the SMs busy."""
    from makani_b200.ops.norm import row_sums
    dev = _dev()
    x = (torch.randn(rows, c, device=dev, generator=torch.Generator(dev).manual_seed(c)) * 1e3).to(torch.bfloat16)
    first = row_sums(x, c)
    side, busy = torch.cuda.Stream(), torch.randn(4096, 4096, device=dev)
    for k in range(8):
        with torch.cuda.stream(side):
            busy = torch.sin(busy)
        assert torch.equal(row_sums(x, c), first), k
    torch.cuda.synchronize()


def test_afno_bias_gradients_repeat_themselves():
    from makani_b200.models.networks.afnonet import AFNO2D
    dev = _dev()
    torch.manual_seed(2)
    m = AFNO2D(128, num_blocks=4).to(dev)
    x, dy = (torch.randn(2, 24, 48, 128, device=dev).to(torch.bfloat16) for _ in range(2))
    grads = [torch.autograd.grad(m(x), [m.b1, m.b2], dy) for _ in range(6)]
    for g in grads[1:]:
        assert torch.equal(g[0], grads[0][0]) and torch.equal(g[1], grads[0][1])


def test_column_sums_of_no_rows():
    from makani_b200.ops.norm import row_sums
    assert torch.equal(row_sums(torch.empty(0, 16, device=_dev(), dtype=torch.bfloat16), 16).cpu(), torch.zeros(16))


@pytest.mark.parametrize("k", [40, 136, 264, 384])
@pytest.mark.parametrize("n", [384, 72, 520])
@pytest.mark.parametrize("epi", ["plain", "gelu", "resid", "mul", "dgelu", "gelu_pre", "gelu_deriv", "fp32"])
def test_gemm_many_tiles_per_cta(k, n, epi):
    """At least four tiles per CTA and per pair: every operand buffer, staging box and accumulator is used again and again.  Short
    k loops run on single CTAs, 264 and 384 on pairs; one 64-column box per warp, ragged columns, ragged rows."""
    dev = _dev()
    z, m = 4, 128 * 150 + 40
    g = torch.Generator(dev).manual_seed(k + n)
    rnd = lambda *s: torch.randn(*s, device=dev, generator=g)  # noqa: E731
    x, w = rnd(z, m, k).to(torch.bfloat16), (rnd(n, k) / k ** 0.5).to(torch.bfloat16)
    aux = rnd(z, m, n).to(torch.bfloat16) if epi in ("resid", "mul", "dgelu") else None
    bias = rnd(n) if epi in ("plain", "gelu", "resid", "gelu_pre", "gelu_deriv") else None
    act = {"resid": ACT_NONE, "plain": ACT_NONE, "fp32": ACT_NONE, "mul": ACT_MULAUX, "dgelu": ACT_DGELU}.get(epi, ACT_GELU)
    acc = x.double() @ w.double().t() + (bias.double() if bias is not None else 0.0)
    leaf = (aux if epi == "dgelu" else acc).double().requires_grad_()
    slope, = torch.autograd.grad(torch.nn.functional.gelu(leaf).sum(), leaf)
    second = acc if epi == "gelu_pre" else slope
    ref = {"plain": lambda: acc, "fp32": lambda: acc, "resid": lambda: acc + aux.double(), "mul": lambda: acc * aux.double(),
           "dgelu": lambda: acc * slope}.get(epi, lambda: torch.nn.functional.gelu(acc))()
    for _ in range(3):
        d = torch.full((z, m, n), float("nan"), device=dev, dtype=torch.float32 if epi == "fp32" else torch.bfloat16)
        pre = torch.full_like(d, float("nan")) if epi in ("gelu_pre", "gelu_deriv") else None
        gemm(m, n, k, Operand(x, ld=k, zs_lo=m * k), Operand(w, ld=k), Output(d, rs_lo=n, d_zlo=m * n), zlo_n=z, bias=bias,
             bias_mode=BIAS_COL, act=act, resid=aux, preact=pre, preact_deriv=epi == "gelu_deriv")
        # on the GPU and in full: one element of one tile counts.  bf16 rounding is half of BF16 of a value; the fp32 sum behind it and
        # the kernel's GELU (a polynomial and tanh.approx, 2^-10) add less than as much
        for got, want in ((d, ref), (pre, second)):
            if got is not None:
                scale = want.square().mean().sqrt()
                tol = 2.0 ** -18 if epi == "fp32" else BF16
                assert ((got.double() - want).abs() <= tol * (want.abs() + scale)).all()
    _ext.check_device_errors(dev)


@pytest.mark.parametrize("b,l,m,co,ci", [(1, 240, 241, 256, 256), (2, 210, 211, 200, 136), (1, 202, 203, 256, 184), (1, 208, 209, 248, 384)])
def test_planar_weight_gradient_on_pairs(b, l, m, co, ci):
    """More than one row tile with little padding and 200 orders or more: the planar weight gradient runs on CTA pairs, with the
    negated segment, degree-limited k ranges and, for 136 to 192 and 384 columns, a pair's half of one and a half boxes."""
    from makani_b200.ops.spectral import contract_wgrad2
    dev = _dev()
    g = torch.Generator(dev).manual_seed(l)
    keep = (torch.arange(m, device=dev)[None] <= torch.arange(l, device=dev)[:, None]).view(1, l, m, 1)
    t2 = (torch.randn(b, l, m, 2 * ci, device=dev, generator=g) * keep).to(torch.bfloat16)
    dt = (torch.randn(b, l, m, 2 * co, device=dev, generator=g) * keep).to(torch.bfloat16)
    cplx = lambda t: torch.complex(t[..., : t.shape[-1] // 2].double(), t[..., t.shape[-1] // 2:].double())  # noqa: E731
    ref = torch.einsum("blmo,blmc->loc", cplx(dt), cplx(t2).conj())
    ref = torch.stack([ref.real, ref.imag])
    for _ in range(2):
        got = contract_wgrad2(dt, t2)
        assert _rel(got, ref) < 2.0 ** -24 * (b * m) ** 0.5 * 4
        assert (got.double() - ref).abs().max() < 2.0 ** -16 * ref.abs().max()
    _ext.check_device_errors(dev)


@pytest.mark.parametrize("m,n,k,zlo,zhi,groups", [
    (8, 8, 1, 1, 1, False),             # one token, the smallest operands
    (72, 40, 63, 2, 1, False),          # part of one slab, batches that add up
    (136, 384, 1000, 1, 1, False),      # two row blocks, two column tiles that take the slabs in turn
    (384, 768, 30001, 1, 1, False),     # three row blocks on single CTAs, many splits, a ragged last slab
    (768, 384, 65537, 1, 1, False),     # CTA pairs
    (520, 256, 4097, 3, 1, False),      # pairs with a padded row block, batches
    (192, 192, 91, 8, 45, True),        # one vector per group, summed over the other batch index
])
def test_row_sums_beside_the_weight_gradient(m, n, k, zlo, zhi, groups):
    from makani_b200.ops.gemm import Operand, Output, gemm
    g = torch.Generator(device="cuda").manual_seed(m + k)
    # one-signed, so that nothing cancels
    a = (torch.rand(zhi, zlo, k, m, device="cuda", generator=g) + 0.5).bfloat16()
    b = torch.randn(zhi, zlo, k, n, device="cuda", generator=g).bfloat16()
    outs = zlo if groups else 1

    def run(sums):
        d = torch.zeros(outs, m, n, device="cuda")
        done = gemm(m, n, k, Operand(a, ld=m, mn_major=True, zs_lo=k * m, zs_hi=zlo * k * m),
                    Operand(b, ld=n, mn_major=True, zs_lo=k * n, zs_hi=zlo * k * n),
                    Output(d, rs_lo=n, d_zlo=m * n if groups else 0), zlo_n=zlo, zhi_n=zhi, accumulate=True, splits=0, row_sums=sums)
        return d, done

    sums, again = (torch.full((outs, m), float("nan"), device="cuda") for _ in range(2))
    d, done = run(sums)
    _, _ = run(again)
    plain, _ = run(None)
    assert done and torch.equal(sums, again)
    # a lane adds up to four tokens of every 64 one after the other, then some 64 partial sums: each step rounds to 2^-24
    ref = a.double().sum(dim=(0, 2) if groups else (0, 1, 2)).reshape(outs, m)
    steps = 4 * -(-k // 64) + 64
    assert ((sums.double() - ref).abs() <= steps * 2.0 ** -24 * ref).all()
    # the gradient itself: the same chains, added up in another order
    assert (d - plain).norm() <= 1e-6 * plain.norm() + 1e-12


@pytest.mark.parametrize("b,h,w,mmax,c", [
    (1, 2, 64, 33, 8),          # half a tile of rows, one vector of channels, the mirror boxes at row 1
    (2, 3, 72, 36, 136),        # the Nyquist order left out, a ragged second column tile
    (1, 5, 90, 46, 64),         # an odd number of pairs of points
    (1, 4, 65, 20, 16),         # an odd number of longitudes
    (1, 3, 248, 125, 200),      # rows past the middle in the last box
    (1, 80, 480, 241, 384),     # pairs of CTAs, several tiles per pair
    (1, 7, 1440, 241, 72),      # few of the orders: the analysis stays whole
])
def test_folded_transforms(b, h, w, mmax, c):
    from makani_b200.ops.spectral import SHTPlan, analyse, synthesise
    dev = _dev()
    plan = SHTPlan(h, w, h, mmax, "legendre-gauss", dev)
    g = torch.Generator(dev).manual_seed(w)
    t4 = torch.randn(b, h, 2 * mmax, c, device=dev, generator=g).to(torch.bfloat16)
    td, f, gt = t4.double(), plan.f.double(), plan.gt[:, :plan.k2].double()
    pairs = [(synthesise(t4, plan).permute(0, 2, 3, 1), gt @ td), (synthesise(t4, plan, forward=True).permute(0, 2, 3, 1), f.t() @ td)]
    assert torch.equal(synthesise(t4, plan), synthesise(t4, plan))      # rows written twice are written with the same bits
    if w % 8 == 0:
        x = torch.randn(b, h, w, c, device=dev, generator=g).to(torch.bfloat16).permute(0, 3, 1, 2)
        xd = x.permute(0, 2, 3, 1).double()
        pairs += [(analyse(x, plan), f @ xd), (analyse(x, plan, forward=False), gt.t() @ xd)]
        assert torch.equal(analyse(x, plan), analyse(x, plan))
    # bf16 outputs; the whole matrices round the same angles to bf16, a few entries to the other neighbour
    for got, ref in pairs:
        assert got.shape == ref.shape and _rel(got, ref) < BF16
    _ext.check_device_errors(dev)


@pytest.mark.parametrize("what", ["conv_weight", "conv_bias", "conv_residual", "mlp_weight", "linear_weight", "linear_bias", "token_mlp_weight",
                                  "norm_weight_cl", "norm_bias_cl", "norm_weight_nchw", "afno_weight", "afno_bias"])
def test_host_tensors_beside_cuda_activations_are_refused(what):
    from makani_b200.ops.afno import afno_filter_stacked
    from makani_b200.ops.conv import conv1x1, mlp2
    from makani_b200.ops.linear import linear_lastdim, mlp2_lastdim
    from makani_b200.ops.norm import instance_norm
    dev = _dev()
    x = torch.randn(1, 16, 8, 16, device=dev).bfloat16().contiguous(memory_format=torch.channels_last)
    tok = torch.randn(32, 16, device=dev).bfloat16()
    on = lambda *shape, host=False: torch.randn(*shape, device="cpu" if host else dev)  # noqa: E731
    planes = torch.randn(1, 8, 8, 16, device=dev).bfloat16()
    calls = {
        "conv_weight": lambda: conv1x1(x, on(16, 16, 1, 1, host=True)),
        "conv_bias": lambda: conv1x1(x, on(16, 16, 1, 1), on(16, host=True)),
        "conv_residual": lambda: conv1x1(x, on(16, 16, 1, 1), None, x.cpu()),
        "mlp_weight": lambda: mlp2(x, on(32, 16, 1, 1), on(32), on(16, 32, 1, 1, host=True), on(16)),
        "linear_weight": lambda: linear_lastdim(tok, on(16, 16, host=True)),
        "linear_bias": lambda: linear_lastdim(tok, on(16, 16), on(16, host=True)),
        "token_mlp_weight": lambda: mlp2_lastdim(tok, on(32, 16, host=True), on(32), on(16, 32), on(16)),
        "norm_weight_cl": lambda: instance_norm(x, on(16, host=True), on(16)),
        "norm_bias_cl": lambda: instance_norm(x, on(16), on(16, host=True)),
        "norm_weight_nchw": lambda: instance_norm(x.contiguous(), on(16, host=True), on(16)),
        "afno_weight": lambda: afno_filter_stacked(planes, on(2, 2, 8, 8, host=True), None, on(2, 2, 8, 8), None, (0, 1, 7), 3, 0.0),
        "afno_bias": lambda: afno_filter_stacked(planes, on(2, 2, 8, 8), on(2, 2, 8, host=True), on(2, 2, 8, 8), None, (0, 1, 7), 3, 0.0),
    }
    with pytest.raises(RuntimeError):
        calls[what]()


def test_bf16_weights_of_linear_layers_are_not_copied():
    dev = _dev()
    x, w = torch.randn(64, 24, device=dev).bfloat16(), torch.randn(16, 24, device=dev).bfloat16()
    y, wq, _ = _ext.require().conv_forward(x, w, None, None, 0, -1, False)
    assert wq.data_ptr() == w.data_ptr() and _rel(y, x.double() @ w.double().t()) < BF16
    wt = torch.randn(24, 16, device=dev).bfloat16().t()      # strided: a copy, as ever
    assert _rel(_ext.require().conv_forward(x, wt, None, None, 0, -1, False)[0], x.double() @ wt.double().t()) < BF16


@pytest.mark.parametrize("rows,mirror,pairs,n,k,z", [
    (64, 64, False, 8, 16, 3),           # the last box of sums holds one row
    (65, 65, False, 72, 40, 2),          # no row is its own mirror
    (90, 90, False, 136, 46, 2),
    (126, 126, False, 264, 8, 1),        # the computed rows end with a box
    (480, 480, False, 384, 241, 5),      # CTA pairs
    (66, 64, True, 16, 32, 2),           # all orders
    (64, 64, True, 8, 32, 1),            # all but the last
    (92, 90, True, 72, 45, 3),           # an odd number of points in each half
    (450, 480, True, 136, 240, 2),
])
def test_folded_products_write_every_row_once(rows, mirror, pairs, n, k, z):
    """Rows past the middle are differences of the rows before it, whatever the table holds there: each row is written once."""
    from makani_b200.ops.gemm import gemm_fold, pad_to
    dev = _dev()
    g = torch.Generator().manual_seed(rows + n)
    m, part = (2 * (mirror // 4 + 1) if pairs else mirror // 2 + 1), pad_to(k, 64)
    table = torch.randint(-1, 2, (rows, 2 * part), generator=g).float()
    table[m:] = 97.0
    b = torch.randint(-1, 2, (z, k, 2, n), generator=g).float()
    b[:, :, :, ::3] = 0.0      # columns of zeros
    out = []
    for d in ("cpu", dev, dev, dev):
        dt = torch.float32 if d == "cpu" else torch.bfloat16
        y = torch.full((z, rows, n), float("nan"), device=d, dtype=dt)
        gemm_fold(rows, m, n, k, mirror, pairs, table.to(d, dt), part, Operand(b.to(d, dt), ld=2 * n, mn_major=True, zs_hi=k * 2 * n), n,
                  Output(y, rs_lo=n, d_zhi=rows * n), zhi_n=z)
        out.append(y)
    # whole numbers: the products and sums are exact, the results rounded once
    assert torch.equal(out[1].cpu(), out[0].to(torch.bfloat16))
    assert all(torch.equal(y.view(torch.int16), out[1].view(torch.int16)) for y in out[2:])
    _ext.check_device_errors(dev)


@pytest.mark.parametrize("n", [4, 60, 73, 131, 256 + 1, 764])
@pytest.mark.parametrize("kind", ["plain", "relu", "row_bias", "preact", "resid", "mulaux", "fp32", "split_rows"])
def test_ragged_widths_leave_the_columns_behind_them_alone(n, kind):
    """A product into the first n columns of a wider matrix, whole vectors and the columns of a partial one."""
    dev = _dev()
    g = torch.Generator(dev).manual_seed(n)
    t, k, z = 300, 72, 2
    ld = -(-n // 8) * 8 + 8
    dt = torch.float32 if kind == "fp32" else torch.bfloat16
    x, w = (torch.randn(*s, device=dev, generator=g).bfloat16() for s in ((z, t, k), (n, k)))
    y, pre = (torch.full((z, t, ld), 7.0, device=dev, dtype=dt) for _ in range(2))
    r, bias = torch.randn(z, t, ld, device=dev, generator=g).bfloat16(), torch.randn(t, device=dev, generator=g)
    kw = {"relu": dict(act=ACT_RELU), "row_bias": dict(bias=bias, bias_mode=BIAS_ROW), "preact": dict(act=ACT_GELU, preact=pre),
          "resid": dict(resid=r), "mulaux": dict(act=ACT_MULAUX, resid=r)}.get(kind, {})
    out = Output(y, rs_lo=t // 2 * ld, rs_hi=ld, rdiv=2, d_zlo=t * ld) if kind == "split_rows" else Output(y, rs_lo=ld, d_zlo=t * ld)
    gemm(t, n, k, Operand(x, ld=k, zs_lo=t * k), Operand(w, ld=k), out, zlo_n=z, **kw)
    a = x.double() @ w.double().t()
    ref = {"relu": a.clamp(min=0), "row_bias": a + bias[:, None], "preact": torch.nn.functional.gelu(a, approximate=_ext.gelu_approximation()),
           "resid": a + r[..., :n], "mulaux": a * r[..., :n], "split_rows": torch.cat([a[:, 0::2], a[:, 1::2]], 1)}.get(kind, a)
    assert _rel(y[..., :n], ref) < BF16 and (y[..., n:] == 7.0).all()
    if kind == "preact":
        assert _rel(pre[..., :n], a) < BF16 and (pre[..., n:] == 7.0).all()
    _ext.check_device_errors(dev)


@pytest.mark.parametrize("n", [4, 60, 73, 131, 250, 764])
@pytest.mark.parametrize("kind", ["plain", "gelu", "preact", "deriv", "resid", "mulaux"])
def test_column_bias_over_ragged_widths(n, kind):
    dev = _dev()
    g = torch.Generator(dev).manual_seed(n)
    t, k, ld, z = 300, 72, -(-n // 8) * 8 + 8, 2
    x, w = (torch.randn(*s, device=dev, generator=g).bfloat16() for s in ((z, t, k), (z, n, k)))
    bias = torch.zeros(z, ld, device=dev)
    bias[:, :n] = torch.randn(z, n, device=dev, generator=g)
    y, pre = (torch.full((z, t, ld), 7.0, device=dev, dtype=torch.bfloat16) for _ in range(2))
    r = torch.randn(z, t, ld, device=dev, generator=g).bfloat16()
    kw = {"gelu": dict(act=ACT_GELU), "preact": dict(act=ACT_GELU, preact=pre), "deriv": dict(act=ACT_GELU, preact=pre, preact_deriv=True),
          "resid": dict(resid=r), "mulaux": dict(act=ACT_MULAUX, resid=r)}.get(kind, {})
    gemm(t, n, k, Operand(x, ld=k, zs_lo=t * k), Operand(w, ld=k, zs_lo=n * k), Output(y, rs_lo=ld, d_zlo=t * ld), zlo_n=z, bias=bias,
         bias_mode=BIAS_COL, bias_zs=ld, **kw)
    a = (x.double() @ w.double().transpose(1, 2) + bias[:, None, :n].double()).requires_grad_(True)
    h = torch.nn.functional.gelu(a, approximate=_ext.gelu_approximation())
    ref = {"plain": a, "resid": a + r[..., :n], "mulaux": a * r[..., :n]}.get(kind, h)
    assert _rel(y[..., :n], ref) < BF16 and (y[..., n:] == 7.0).all()
    if kind == "preact":
        assert _rel(pre[..., :n], a) < BF16 and (pre[..., n:] == 7.0).all()
    if kind == "deriv":
        assert _rel(pre[..., :n], torch.autograd.grad(h.sum(), a)[0]) < BF16 and (pre[..., n:] == 7.0).all()
    _ext.check_device_errors(dev)


def test_column_bias_over_ragged_widths_leaves_through_tma():
    """764 of 768 columns take about the time of 768; element by element they took 3.3 times as long."""
    dev = _dev()
    x, w, b = torch.randn(115200, 384, device=dev).bfloat16(), torch.randn(768, 384, device=dev).bfloat16(), torch.randn(768, device=dev)
    y = torch.empty(115200, 768, device=dev, dtype=torch.bfloat16)

    def best(n):
        out = []
        for _ in range(8):
            t0, t1 = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            t0.record()
            gemm(115200, n, 384, Operand(x, ld=384), Operand(w, ld=384), Output(y, rs_lo=768), bias=b, bias_mode=BIAS_COL)
            t1.record()
            torch.cuda.synchronize()
            out.append(t0.elapsed_time(t1))
        return min(out)

    assert best(764) < 2.0 * best(768)


def test_folded_products_with_a_narrow_last_tile_keep_their_ctas_together():
    """136 of 256 columns: CTAs that met only the tiles of 8 columns ran ahead, and shared lines left L2 half by half (150 us, 256
    channels 106)."""
    from makani_b200.ops.spectral import SHTPlan, folded_synthesis
    dev = _dev()
    plan = SHTPlan(8, 1440, 8, 64, "legendre-gauss", dev)

    def best(c):
        t4, out = torch.randn(1, 721, 128, c, device=dev).bfloat16(), []
        for _ in range(8):
            t0, t1 = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            t0.record()
            folded_synthesis(t4, plan)
            t1.record()
            torch.cuda.synchronize()
            out.append(t0.elapsed_time(t1))
        return min(out)

    assert best(136) < 1.15 * best(256)


@pytest.mark.parametrize("b,taken", [(1024, True), (1025, False)])
def test_row_sums_of_very_many_batches_are_a_pass_of_their_own(b, taken):
    """Four partial sums per row and batch: past 4096 adding them up takes longer than reading the matrix once more."""
    from makani_b200.ops.conv import _conv_wgrad
    dev = _dev()
    g = torch.Generator(dev).manual_seed(b)
    dy, x = (torch.randint(-1, 2, (b, 8, 8, 64), device=dev, generator=g).bfloat16().permute(0, 3, 1, 2) for _ in range(2))
    d, sums = torch.zeros(64, 64, device=dev), torch.empty(64, device=dev)
    assert gemm(64, 64, 64, Operand(dy, ld=64, mn_major=True, zs_lo=64 * 64), Operand(x, ld=64, mn_major=True, zs_lo=64 * 64), Output(d, rs_lo=64),
                zlo_n=b, accumulate=True, splits=0, row_sums=sums) == taken
    dw, db = _conv_wgrad(dy, x, bias=True)
    assert torch.equal(db, dy.float().sum((0, 2, 3)))
    assert torch.equal(dw, torch.einsum("bohw,bihw->oi", dy.float(), x.float()))


@pytest.mark.parametrize("m,n,k,zlo", [
    (1120, 384, 4097, 1),       # CTA pairs, the second of the last pair without rows
    (1096, 40, 513, 2),         # the same, ragged, batches that add up
    (768, 384, 65537, 1),       # one token in the last slab
    (384, 768, 30001, 1),       # single CTAs, many splits
    (520, 256, 4097, 3),
])
def test_row_sums_count_every_token_once(m, n, k, zlo):
    """Whole numbers whose sums fp32 holds: exact in any order.  The last token of a batch weighs more than any other."""
    dev = _dev()
    g = torch.Generator(dev).manual_seed(k)
    a = torch.randint(0, 4, (zlo, k, m), device=dev, generator=g).bfloat16()
    a[:, -1] = torch.randint(100, 256, (zlo, m), device=dev, generator=g).bfloat16()
    b = torch.randint(-1, 2, (zlo, k, n), device=dev, generator=g).bfloat16()
    d, sums = torch.zeros(m, n, device=dev), torch.full((m,), float("nan"), device=dev)
    assert gemm(m, n, k, Operand(a, ld=m, mn_major=True, zs_lo=k * m), Operand(b, ld=n, mn_major=True, zs_lo=k * n), Output(d, rs_lo=n),
                zlo_n=zlo, accumulate=True, splits=0, row_sums=sums)
    assert torch.equal(sums.double(), a.double().sum((0, 1)))
    assert torch.equal(d.double(), (a.double().transpose(1, 2) @ b.double()).sum(0))
    _ext.check_device_errors(dev)


def test_activations_in_the_epilogue_cost_about_as_much_as_none():
    """Each activation has a loop of its own: asked for at run time, the derivatives took 1.4 to 2.1 times as long as a saved one."""
    dev = _dev()
    m, k, n = 115200, 384, 768
    x, w, r = torch.randn(m, k, device=dev).bfloat16(), torch.randn(n, k, device=dev).bfloat16(), torch.randn(m, n, device=dev).bfloat16()
    y = torch.empty_like(r)

    def best(**kw):
        out = []
        for _ in range(8):
            t0, t1 = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            t0.record()
            gemm(m, n, k, Operand(x, ld=k), Operand(w, ld=k), Output(y, rs_lo=n), **kw)
            t1.record()
            torch.cuda.synchronize()
            out.append(t0.elapsed_time(t1))
        return min(out)

    saved = best(act=ACT_MULAUX, resid=r)
    for act in (ACT_DRELU, ACT_DSHRINK):
        assert best(act=act, resid=r) < 1.25 * saved
    assert best(act=ACT_DGELU, resid=r) < 1.6 * saved
    assert best(act=ACT_SHRINK, act_param=0.1) < 1.6 * best()


def test_norm_of_a_field_off_a_16_byte_boundary():
    """The channels-last kernels load whole 16-byte vectors; elsewhere the field is copied first, and the kernels themselves refuse it."""
    from makani_b200.ops.norm import instance_norm
    dev = _dev()
    b, c, h, w = 2, 16, 6, 8
    x = torch.randn(b * h * w * c + 1, device=dev).bfloat16()[1:].view(b, h, w, c).permute(0, 3, 1, 2)
    assert x.data_ptr() % 16 and x.is_contiguous(memory_format=torch.channels_last)
    wt, bi = torch.randn(c, device=dev), torch.randn(c, device=dev)
    ref = torch.nn.functional.instance_norm(x.double(), None, None, wt.double(), bi.double(), eps=1e-6)
    assert _rel(instance_norm(x, wt, bi, 1e-6), ref) < BF16
    with pytest.raises(RuntimeError, match="invalid argument"):
        _ext.require().norm_forward(x, wt, bi, 1e-6, 0, float(h * w))


@pytest.mark.parametrize("b,l,m,co,ci", [
    (1, 296, 5, 8, 8),            # as few channels as there are, orders in part of one slab
    (1, 80, 81, 136, 72),         # second tiles of 8 outputs and 8 inputs
    (1, 28, 64, 200, 328),        # a slab that is full, more orders than degrees
    (1, 20, 21, 384, 384),        # whole tiles
    (1, 132, 66, 128, 200),       # two slabs, the second of two orders
    (1, 196, 197, 256, 64),       # four slabs
    (2, 80, 81, 136, 72), (1, 82, 83, 136, 72), (1, 8, 9, 16, 16),      # two samples, degrees off four, few tiles: planes and their re-layout
])
def test_spectral_weight_gradient_in_its_own_layout(b, l, m, co, ci):
    """Against complex float64 and against the planes with their re-layout; every element written (memory full of NaN before)."""
    from makani_b200.ops.spectral import contract_wgrad2, fold_weight_grad2, weight_gradient
    dev = _dev()
    g = torch.Generator(dev).manual_seed(l + co)
    keep = (torch.arange(m, device=dev)[None] <= torch.arange(l, device=dev)[:, None]).view(1, l, m, 1)
    t2, dt = ((torch.randn(b, l, m, 2 * c, device=dev, generator=g) * keep).to(torch.bfloat16) for c in (ci, co))
    cplx = lambda t: torch.complex(t[..., : t.shape[-1] // 2].double(), t[..., t.shape[-1] // 2:].double())  # noqa: E731
    ref = torch.einsum("blmo,blmc->col", cplx(dt), cplx(t2).conj())
    full = torch.full((ci, co, l), float("nan"), dtype=torch.complex64, device=dev)
    del full      # the next tensor of this size takes its place
    got = weight_gradient(dt, t2)
    bound = 2.0 ** -24 * max(b * m, 64) ** 0.5 * 4      # fp32 sums of up to b m products, truncated every 16
    assert got.shape == ref.shape and _rel(torch.view_as_real(got), torch.view_as_real(ref)) < bound
    assert _rel(torch.view_as_real(got), torch.view_as_real(fold_weight_grad2(contract_wgrad2(dt, t2)))) < bound
    _ext.check_device_errors(dev)


@pytest.mark.parametrize("n,epi", [(264, "plain"), (264, "resid"), (264, "mul"), (200, "gelu_deriv"), (776, "plain"), (328, "gelu_deriv")])
def test_narrow_last_column_tile_over_many_rows(n, epi):
    """Many rows and an even number of column tiles, the last one narrow: the grid has no factor in common with them, every tile is still met."""
    dev = _dev()
    g = torch.Generator(dev).manual_seed(n)
    m, k = 256 * 148 + 40, 72
    x, w = torch.randn(m, k, device=dev, generator=g).to(torch.bfloat16), (torch.randn(n, k, device=dev, generator=g) * k ** -0.5).to(torch.bfloat16)
    aux = torch.randn(m, n, device=dev, generator=g).to(torch.bfloat16) if epi in ("resid", "mul") else None
    pre = torch.full((m, n), float("nan"), device=dev, dtype=torch.bfloat16) if epi == "gelu_deriv" else None
    d = torch.full((m, n), float("nan"), device=dev, dtype=torch.bfloat16)
    gemm(m, n, k, Operand(x, ld=k), Operand(w, ld=k), Output(d, rs_lo=n), resid=aux, preact=pre, preact_deriv=pre is not None,
         act={"mul": ACT_MULAUX, "gelu_deriv": ACT_GELU}.get(epi, ACT_NONE))
    z = (x.double() @ w.double().t())
    if epi == "gelu_deriv":
        z.requires_grad_()
        y = torch.nn.functional.gelu(z)
        (dy,) = torch.autograd.grad(y.sum(), z)
        assert _rel(pre, dy) < BF16
    else:
        y = z if aux is None else (z + aux.double() if epi == "resid" else z * aux.double())
    assert _rel(d, y.detach()) < BF16
    _ext.check_device_errors(dev)


@pytest.mark.parametrize("l,m,h,n", [(129, 130, 216, 48), (240, 241, 240, 136), (256, 9, 520, 200), (257, 20, 208, 72)])
def test_triangular_rows_on_one_pair(l, m, h, n):
    """Row-triangular products whose rows one CTA pair covers (and one more row than that): zeros below the first valid row, also for
    batches that have none in the first half of the pair, and nothing left unwritten."""
    dev = _dev()
    g = torch.Generator(dev).manual_seed(l)
    hp = (h + 7) // 8 * 8
    keep = (torch.arange(l, device=dev)[None] >= torch.arange(m, device=dev)[:, None])[..., None]
    table = torch.randn(m, l, hp, device=dev, generator=g).mul(keep).to(torch.bfloat16)
    table[..., h:] = 0
    x = torch.randn(m, h, n, device=dev, generator=g).to(torch.bfloat16)
    d = torch.full((m, l, n), float("nan"), device=dev, dtype=torch.bfloat16)
    gemm(l, n, h, Operand(table, ld=hp, zs_hi=l * hp), Operand(x, ld=n, mn_major=True, zs_hi=h * n), Output(d, rs_lo=n, d_zhi=l * n), zhi_n=m,
         tri=Tri(rmin_a=1))
    ref = torch.einsum("mlh,mhn->mln", table[..., :h].double(), x.double())
    assert _rel(d, ref) < BF16 and bool((d[~keep.expand_as(d)] == 0).all())
    _ext.check_device_errors(dev)


@pytest.mark.parametrize("b,c,t", [(75, 256, 3000), (1, 24, 100), (1, 48, 100), (2, 72, 3360), (1, 64, 32400), (1, 96, 1800), (1, 128, 3601), (3, 192, 700), (1, 16, 18000),
                                   (1, 1024, 333), (2, 384, 6720)])
def test_instance_norm_with_statistics_of_two_devices(b, c, t):
    """The exchange form of the four kernels on one of two halves of a field, at rows of threads that fill no whole warps (and some that do): the other
    half's sums are in place and all flags set before the launches, so that nothing waits.  Against float64 of the whole field."""
    dev = _dev()
    g = torch.Generator(dev).manual_seed(c + t)
    ext, eps, n = _ext.require(), 1e-2, float(2 * t)
    x, dy = ((torch.randn(2, b, t, c, device=dev, generator=g) + 0.5).bfloat16() for _ in range(2))
    wt, bi = (torch.randn(c, device=dev, generator=g) for _ in range(2))
    # flags[8] that are waited for | counters of the waits | launches done | signals[8]
    ctrl = torch.zeros(32, dtype=torch.int32, device=dev)
    ctrl[:8] = 1000
    at = ctrl.data_ptr()
    bumped, done, signals = at + 32, at + 36, at + 64
    sync = [1, 1, done, at, bumped, 0, bumped, 2, 0, 0, 0, 0, 0, 2, signals, signals + 4] + [0] * 6 + [0] * 9
    segments, copy = torch.zeros(2, b, c, 2, device=dev), torch.zeros(b, c, 2, device=dev)
    xd, wd, bd = x.double().requires_grad_(), wt.double().requires_grad_(), bi.double().requires_grad_()
    mean = xd.mean((0, 2), keepdim=True)
    rstd = 1.0 / torch.sqrt((xd - mean).square().mean((0, 2), keepdim=True) + eps)
    for act in (0, 1):
        yd = (xd - mean) * rstd * wd + bd
        yd = torch.nn.functional.gelu(yd) if act else yd
        (want,) = torch.autograd.grad(yd, xd, dy.double(), retain_graph=True)
        stats = torch.empty(b, c, 2, device=dev)

        def other(a0, a1):
            """The second device's sums"""
            segments[1] = torch.stack([a0[1], a1[1]], -1).float()

        def both(run):
            segments[0] = copy[:] = float("nan")
            sums = torch.zeros(b, c, 2, device=dev)
            run(sums)
            assert torch.equal(sums, segments[0]) and torch.equal(sums, copy)

        dsts, srcs = [segments[0].data_ptr(), copy.data_ptr()], [segments[0].data_ptr(), segments[1].data_ptr()]
        other(x.double().sum(2), x.double().square().sum(2))
        both(lambda sums: ext.inorm_cl_sums(x[0], None, None, None, None, sums, None, None, b, c, 0, 0, sync, dsts))
        y, dx = torch.full_like(x[0], float("nan")), torch.full_like(x[0], float("nan"))
        ext.inorm_cl_apply(x[0], None, y, wt, bi, segments[0], stats, b, c, n, eps, act, 0, sync, srcs)
        assert (stats[..., 0].double() - mean[0, :, 0]).abs().max() < 1e-5
        assert (stats[..., 1].double() / rstd[0, :, 0] - 1.0).abs().max() < 1e-5
        # half a unit of 2^-8 per value; GELU is 5.5e-5 off, its derivative 2e-4 times (1 + |x|), at outputs of order 1
        assert (y.double() - yd[0]).norm() < (2.0 ** -8 + (1e-4 if act else 0.0)) * yd[0].norm() + 1e-6
        pre = ((xd - mean) * rstd * wd + bd).detach().requires_grad_()
        (slope,) = torch.autograd.grad(torch.nn.functional.gelu(pre).sum() if act else pre.sum(), pre)
        gd = (dy.double() * slope)
        other(gd.sum(2), (gd * (xd - mean) * rstd).sum(2).detach())
        dw, db = torch.zeros(c, device=dev), torch.zeros(c, device=dev)
        both(lambda sums: ext.inorm_cl_sums(x[0], dy[0], wt, bi, stats, sums, dw, db, b, c, act, 1, sync, dsts))
        ext.inorm_cl_apply(x[0], dy[0], dx, wt, bi, segments[0], stats, b, c, n, 0.0, act, 1, sync, srcs)
        scale = dy.double().norm() * (rstd * wd).abs().max()      # dx is a difference of terms of this size
        assert (dx.double() - want[0]).norm() < 2.0 ** -8 * want[0].norm() + (2e-3 if act else 1e-5) * scale
        for got, term in ((db, gd[0]), (dw, (gd * (xd - mean) * rstd)[0].detach())):
            assert (got.double() - term.sum((0, 1))).norm() <= (2e-3 if act else 1e-5) * term.abs().sum((0, 1)).norm()
    assert int(ctrl[8]) == 8 and int(ctrl[9]) == 0 and ctrl[16:18].tolist() == [8, 8]      # every launch counted and signalled once
    _ext.check_device_errors(dev)


@pytest.mark.parametrize("b,c,h,w", [(1, 24, 10, 10), (8, 72, 80, 84), (1, 64, 180, 180), (2, 96, 30, 60), (8, 128, 1, 3601), (1, 192, 100, 181), (1, 8, 97, 192),
                                     (75, 384, 50, 60), (149, 128, 60, 128)])
def test_instance_norm_rows_that_fill_no_whole_warps(b, c, h, w):
    """The last two: shares of an image in several waves of CTAs."""
    dev = _dev()
    g = torch.Generator(dev).manual_seed(c + h)
    x, dy = (torch.randn(b, h, w, c, device=dev, generator=g).bfloat16().permute(0, 3, 1, 2) for _ in range(2))
    wt, bi = (torch.randn(c, device=dev, generator=g) for _ in range(2))
    ext = _ext.require()
    y, stats, wf, bf = ext.norm_forward(x, wt, bi, 1e-2, 0, float(h * w))
    dx, dw, db = ext.norm_backward(x, dy, wf, bf, stats, True, 0, float(h * w))
    xd, wd, bd = x.double().requires_grad_(), wt.double().requires_grad_(), bi.double().requires_grad_()
    yd = torch.nn.functional.instance_norm(xd, None, None, wd, bd, True, 0.0, 1e-2)
    want = torch.autograd.grad(yd, [xd, wd, bd], dy.double())
    # half a unit of 2^-8 per value, sums of fp32
    assert (y.double() - yd).norm() < 2.0 ** -8 * yd.norm()
    assert (dx.double() - want[0]).norm() < 2.0 ** -8 * want[0].norm() + 1e-5 * dy.double().norm()
    xh = torch.nn.functional.instance_norm(x.double(), eps=1e-2)
    for got, ref, term in ((dw, want[1], dy.double() * xh), (db, want[2], dy.double())):
        assert (got.double() - ref).norm() <= 1e-5 * term.abs().sum((0, 2, 3)).norm()
    _ext.check_device_errors(dev)


@pytest.mark.parametrize("co,ci", [(8, 8), (600, 1008), (1544, 1576), (2056, 1288)])
def test_gradients_are_added_to_zero_at_any_size(co, ci):
    """Cleared by blocks for four per SM (up to some 10 MB) and by four vectors of a thread: weight gradients that start in memory full of NaN."""
    dev = _dev()
    g = torch.Generator(dev).manual_seed(co)
    ext = _ext.require()
    x, dy = (torch.randn(2, 8, 16, c, device=dev, generator=g).bfloat16().permute(0, 3, 1, 2) for c in (ci, co))
    wq = torch.randn(co, ci, device=dev, generator=g).bfloat16()
    held = torch.full((co, ci), float("nan"), device=dev)
    del held      # the gradient takes its place
    _, dw, db = ext.conv_backward(dy, x, wq, ci, False, True, True)
    rows = lambda t: t.double().permute(1, 0, 2, 3).flatten(1)  # noqa: E731
    assert (dw.double() - rows(dy) @ rows(x).t()).norm() <= 1e-6 * (rows(dy) @ rows(x).t()).norm()
    assert (db.double() - rows(dy).sum(1)).norm() <= 1e-6 * rows(dy).abs().sum(1).norm()
    _ext.check_device_errors(dev)
