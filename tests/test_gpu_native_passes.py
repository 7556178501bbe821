"""The native layer passes (csrc/layers.cpp) against the stage functions of `makani_b200/ops` on the same CUDA tensors: the same
launches, so the same bits wherever a launch repeats itself."""

import pytest
import torch

from makani_b200.ops import _ext

pytestmark = pytest.mark.gpu


def _dev():
    if not torch.cuda.is_available():
        pytest.skip("needs a GPU")
    return torch.device("cuda", 0)


def _cl(g, *shape):
    b, c, h, w = shape
    return torch.randn(b, h, w, c, device="cuda", generator=g).bfloat16().permute(0, 3, 1, 2)


def _peak(fn):
    """Device memory that a call needs beyond what is held before it."""
    fn()
    torch.cuda.synchronize()
    before = torch.cuda.memory_allocated()
    torch.cuda.reset_peak_memory_stats()
    out = fn()
    del out
    return torch.cuda.max_memory_allocated() - before


@pytest.mark.parametrize("b,c,co,h,w,ho,wo,lmax,m_in,m_out,resid", [
    (2, 16, 24, 33, 64, 16, 32, 16, 17, 17, True),       # regridded residual
    (1, 40, 8, 48, 96, 45, 90, 40, 46, 46, True),        # 90 longitudes out: an odd half; ragged channels
    (2, 8, 16, 32, 64, 33, 65, 32, 33, 33, False),       # an odd number of longitudes out
    (1, 136, 72, 40, 80, 40, 80, 40, 41, 41, False),     # two column tiles
    (2, 16, 16, 24, 48, 24, 48, 24, 25, 25, False),      # nothing folded
    (1, 16, 32, 48, 96, 48, 96, 40, 12, 12, True),       # few orders: the analysis stays whole
    (1, 64, 72, 96, 192, 96, 192, 96, 97, 97, True),     # both transforms folded in both directions
])
def test_spectral_passes(b, c, co, h, w, ho, wo, lmax, m_in, m_out, resid):
    from makani_b200.ops.spectral import SHTPlan, backward_stages, forward_stages, weight_planes
    dev = _dev()
    g = torch.Generator(dev).manual_seed(c + w)
    pin, pout = SHTPlan(h, w, lmax, m_in, "equiangular", dev), SHTPlan(ho, wo, lmax, m_out, "legendre-gauss", dev)
    x, dy, dr = _cl(g, b, c, h, w), _cl(g, b, co, ho, wo), _cl(g, b, c, ho, wo) if resid else None
    wx = weight_planes(torch.randn(c, co, lmax, device=dev, generator=g, dtype=torch.complex64) * c ** -0.5)
    ext = _ext.require()

    def fwd():
        return ext.spectral_forward(x, wx, *pin.native, *pout.native, resid)

    y, r, t2 = fwd()
    want = forward_stages(x, wx, pin, pout, resid)
    for got, ref in zip((y, r, t2), want):
        assert (got is None and ref is None) or (torch.equal(got, ref) and got.stride() == ref.stride())
    for need_x, need_w in ((True, True), (True, False), (False, True)):
        got = ext.spectral_backward(dy, dr, t2, wx, *pin.native, *pout.native, need_x, need_w)
        ref = backward_stages(dy, dr, t2, wx, pin, pout, need_x, need_w)
        for a, e in zip(got, ref):
            assert (a is None and e is None) or torch.equal(a, e)
    _ext.check_device_errors(dev)


def test_spectral_forward_frees_its_intermediates():
    """Where the transform keeps all orders its intermediates are as large as the field: one is gone before the next but one is made."""
    from makani_b200.ops.spectral import SHTPlan, forward_stages, weight_planes
    dev = _dev()
    g = torch.Generator(dev).manual_seed(0)
    plan = SHTPlan(64, 128, 64, 65, "legendre-gauss", dev)
    x, wx = _cl(g, 4, 64, 64, 128), weight_planes(torch.randn(64, 64, 64, device=dev, generator=g, dtype=torch.complex64))
    native = _peak(lambda: _ext.require().spectral_forward(x, wx, *plan.native, *plan.native, False))
    assert native <= _peak(lambda: forward_stages(x, wx, plan, plan, False))


def test_fewer_orders_forward_than_inverse():
    """Through the module: the orders that the forward transform does not keep are zero, as in the whole transform of 48 longitudes."""
    from makani_b200.models.common.spectral_convolution import SpectralConv
    from makani_b200.sht import InverseRealSHT, RealSHT
    dev = _dev()
    for h, w, m_in, m_out in ((64, 128, 24, 33), (24, 48, 12, 17)):
        lmax = 24
        g = torch.Generator(dev).manual_seed(w)
        fwd, inv = (t(h, w, lmax=lmax, mmax=m, grid="legendre-gauss").to(dev) for t, m in ((RealSHT, m_in), (InverseRealSHT, m_out)))
        net = SpectralConv(fwd, inv, 16, 16, operator_type="dhconv").to(dev)
        x = _cl(g, 2, 16, h, w)
        with torch.no_grad():
            y = net(x)[0].double()
            c = torch.zeros(2, 16, lmax, m_out, dtype=torch.complex64, device=dev)
            c[..., :m_in] = fwd(x.float())
            ref = inv(torch.einsum("bilm,iol->bolm", c, net.weight)).double()
        assert (y - ref).norm() < 1e-2 * ref.norm()      # five bf16 stages


def _as(x, layout):
    return x.contiguous(memory_format=torch.channels_last) if layout == "cl" else x.contiguous()


def _close_sums(got, ref):
    """Gradients that several CTAs add into one output: the same partial sums in another order."""
    assert (got is None and ref is None) or (got.double() - ref.double()).norm() <= 1e-6 * ref.double().norm() + 1e-12


@pytest.mark.parametrize("b,ci,co,h,w,lay,out,act,bias,resid", [
    (2, 24, 40, 9, 16, "cl", None, "none", True, True),       # channels-last throughout, ragged channels
    (2, 73, 384, 8, 24, "nchw", None, "gelu", True, False),   # fields in, padded weight pitch
    (1, 136, 73, 13, 24, "cl", None, "none", False, False),   # fields out: sums by a pass of their own
    (1, 16, 16, 8, 8, "nchw", "nchw", "none", True, True),
    (3, 520, 8, 5, 8, "cl", "nchw", "gelu", True, False),
])
def test_convolution_passes(b, ci, co, h, w, lay, out, act, bias, resid):
    from makani_b200.ops.conv import (_LAYOUT_CODE, ACT_GELU, ACT_NONE, _chan_sum, _conv_dgrad, _conv_fwd, _conv_wgrad, default_out_layout,
                                      layout_of, prep_weight)
    dev = _dev()
    g = torch.Generator(dev).manual_seed(ci + co)
    ext, a = _ext.require(), ACT_GELU if act == "gelu" else ACT_NONE
    x, wt = _as(_cl(g, b, ci, h, w), lay), torch.randn(co, ci, 1, 1, device=dev, generator=g) * ci ** -0.5
    bi = torch.randn(co, device=dev, generator=g) if bias else None
    r = _as(_cl(g, b, co, h, w), out or default_out_layout(co)) if resid else None
    y, wq, pre = ext.conv_forward(x, wt, bi, r, a, _LAYOUT_CODE[out], a == ACT_GELU)
    ref, pre_ref = _conv_fwd(x, prep_weight(wt), ci, bi, a, r, a == ACT_GELU, out_layout=out)
    assert torch.equal(y, ref) and y.stride() == ref.stride() and torch.equal(wq, prep_weight(wt))
    assert pre is None if pre_ref is None else torch.equal(pre, pre_ref)
    for dy in (_as(_cl(g, b, co, h, w), lay) for lay in (("cl", "nchw") if co % 8 == 0 else ("nchw",))):
        dx, dw, db = ext.conv_backward(dy, x, wq, ci, True, True, True)
        want = _conv_dgrad(dy, wq, ci, x_layout=layout_of(x))
        assert torch.equal(dx, want) and dx.stride() == want.stride()
        dw_ref, db_ref = _conv_wgrad(dy, x, bias=True)
        _close_sums(dw, dw_ref)
        assert torch.equal(db, db_ref)
        # sums of their own, without the weight gradient
        alone = ext.conv_backward(dy, x, wq, ci, False, False, True)
        assert alone[0] is None and alone[1] is None and torch.equal(alone[2], _chan_sum(dy))


@pytest.mark.parametrize("b,ci,ch,co,h,w,lay,out,resid", [
    (2, 24, 48, 24, 9, 16, "cl", None, True), (1, 73, 136, 73, 8, 24, "nchw", "nchw", False), (1, 40, 384, 16, 5, 24, "cl", None, False),
])
def test_mlp_passes(b, ci, ch, co, h, w, lay, out, resid):
    from makani_b200.ops.conv import (_LAYOUT_CODE, ACT_GELU, ACT_MULAUX, ACT_NONE, CL, _conv_dgrad, _conv_fwd, _conv_wgrad,
                                      default_out_layout, layout_of, prep_weight)
    dev = _dev()
    g = torch.Generator(dev).manual_seed(ch)
    ext = _ext.require()
    x = _as(_cl(g, b, ci, h, w), lay)
    w1, w2 = torch.randn(ch, ci, 1, 1, device=dev, generator=g) * ci ** -0.5, torch.randn(co, ch, 1, 1, device=dev, generator=g) * ch ** -0.5
    b1, b2 = torch.randn(ch, device=dev, generator=g), torch.randn(co, device=dev, generator=g)
    r = _as(_cl(g, b, co, h, w), out or default_out_layout(co)) if resid else None
    for train in (True, False):
        y, w1q, w2q, dact, h1 = ext.mlp_forward(x, w1, b1, w2, b2, r, _LAYOUT_CODE[out], train)
        h_ref, d_ref = _conv_fwd(x, prep_weight(w1), ci, b1, ACT_GELU, None, train, out_layout=CL, deriv=train)
        y_ref, _ = _conv_fwd(h_ref, prep_weight(w2), ch, b2, ACT_NONE, r, False, out_layout=out)
        assert torch.equal(y, y_ref) and y.stride() == y_ref.stride() and torch.equal(h1, h_ref)
        assert dact is None if d_ref is None else torch.equal(dact, d_ref)
    *_, dact, h1 = ext.mlp_forward(x, w1, b1, w2, b2, r, _LAYOUT_CODE[out], True)
    dy = _as(_cl(g, b, co, h, w), layout_of(y))
    dx, dw1, db1, dw2, db2 = ext.mlp_backward(dy, x, w1q, w2q, dact, h1, ci, True, True, True)
    dpre = _conv_dgrad(dy, w2q, ch, act=ACT_MULAUX, aux=dact, x_layout=CL)
    want = _conv_dgrad(dpre, w1q, ci, x_layout=layout_of(x))
    assert torch.equal(dx, want) and dx.stride() == want.stride()
    for (dw, db), (dw_ref, db_ref) in (((dw2, db2), _conv_wgrad(dy, h1, bias=True)), ((dw1, db1), _conv_wgrad(dpre, x, bias=True))):
        _close_sums(dw, dw_ref)
        assert torch.equal(db, db_ref)


@pytest.mark.parametrize("t,c,o", [(9, 8, 16), (77, 24, 40), (300, 136, 520)])
def test_linear_passes_are_those_of_a_convolution(t, c, o):
    """Tokens [t, c] are the channels-last image [1, c, 1, t]."""
    dev = _dev()
    g = torch.Generator(dev).manual_seed(t)
    ext = _ext.require()
    image = lambda v: v.t()[None, :, None]  # noqa: E731
    x, dy = (torch.randn(t, n, device=dev, generator=g).bfloat16() for n in (c, o))
    w, bi = torch.randn(o, c, device=dev, generator=g), torch.randn(o, device=dev, generator=g)
    y, wq, _ = ext.conv_forward(x, w, bi, None, 0, -1, False)
    assert torch.equal(image(y), ext.conv_forward(image(x), w, bi, None, 0, 1, False)[0])
    dx, dw, db = ext.conv_backward(dy, x, wq, c, True, True, True)
    dxi, dwi, dbi = ext.conv_backward(image(dy), image(x), wq, c, True, True, True)
    _close_sums(dw, dwi)
    assert torch.equal(image(dx), dxi) and torch.equal(db, dbi)


@pytest.mark.parametrize("b,c,h,w,act,affine", [(2, 16, 9, 16, 1, True), (1, 200, 33, 64, 0, True), (3, 1024, 3, 5, 1, False)])
def test_norm_passes(b, c, h, w, act, affine):
    dev = _dev()
    g = torch.Generator(dev).manual_seed(c)
    ext, eps = _ext.require(), 1e-6
    x, dy = _cl(g, b, c, h, w), _cl(g, b, c, h, w)
    wt, bi = ((torch.randn(c, device=dev, generator=g) for _ in range(2)) if affine else (None, None))
    y, stats, wf, bf = ext.norm_forward(x, wt, bi, eps, act, float(h * w))
    sums, st = torch.zeros(b, c, 2, device=dev), torch.empty(b, c, 2, device=dev)
    ref = torch.empty_like(x)
    ext.inorm_cl_sums(x, None, None, None, None, sums, None, None, b, c, 0, 2)
    ext.inorm_cl_apply(x, None, ref, wf, bf, sums, st, b, c, float(h * w), eps, act, 2)
    # the sums are added up by atomics in any order: results may round to the other neighbour
    assert (stats - st).abs().max() <= 1e-5 * st.abs().max() and (y.double() - ref.double()).norm() <= 2.0 ** -8 * ref.double().norm()
    got = ext.norm_backward(x, dy, wf, bf, stats, affine, act, float(h * w))
    acc, dx = torch.zeros(2 * b + 2, c, device=dev), torch.empty_like(x)
    sums, dw, db = acc[:2 * b].view(b, c, 2), *((acc[2 * b], acc[2 * b + 1]) if affine else (None, None))
    ext.inorm_cl_sums(x, dy, wf, bf, stats, sums, dw, db, b, c, act, 1)
    ext.inorm_cl_apply(x, dy, dx, wf, bf, sums, stats, b, c, float(h * w), 0.0, act, 1)
    assert (got[0].double() - dx.double()).norm() <= 2.0 ** -8 * dx.double().norm()
    for a, e in zip(got[1:], (dw, db)):
        assert (a is None and e is None) or (a - e).norm() <= 1e-5 * e.norm()


@pytest.mark.parametrize("b,h,w,c,nb,f,frac,bias,skip", [
    (1, 16, 32, 128, 2, 1, 1.0, True, "x"),           # blocks of 64
    (2, 9, 14, 48, 3, 2, 0.7, True, None),            # narrow blocks, few rows each: one product over all rows
    (1, 40, 80, 256, 32, 1, 1.0, False, "other"),     # many narrow blocks: one product over all channels
    (1, 70, 12, 64, 1, 1, 1.0, True, "x"),            # rows that fill more than half a tile
    (2, 45, 90, 256, 8, 2, 1.0, True, "x"),
])
def test_afno_passes(b, h, w, c, nb, f, frac, bias, skip):
    from makani_b200.ops import afno
    dev = _dev()
    g = torch.Generator(dev).manual_seed(c + h)
    bs, hid, lam = c // nb, c // nb * f, 0.03
    kx, ncols = afno.mode_window_v2(h, w, frac)
    plan = afno.AFNOPlan(h, w, kx, ncols, dev, torch.bfloat16)
    x, dy, other = (torch.randn(b, h, w, c, device=dev, generator=g).bfloat16() for _ in range(3))
    w1, w2 = (torch.randn(2, nb, *s, device=dev, generator=g) * s[0] ** -0.5 for s in ((bs, hid), (hid, bs)))
    b1, b2 = (torch.randn(2, nb, n, device=dev, generator=g) * 0.1 if bias else None for n in (hid, bs))
    sk = {"x": x, "other": other, None: None}[skip]
    ext = _ext.require()
    got = ext.afno_forward(x, w1, b1, w2, b2, sk, plan.tables, plan.extents(nb), lam)
    for a, e in zip(got, afno.forward_stages(x, w1, b1, w2, b2, sk, plan, lam)):
        assert torch.equal(a, e)
    back = ext.afno_backward(dy, *got[1:], plan.tables, plan.extents(nb), bias, bias, skip == "x")
    want = afno.backward_stages(dy, *got[1:], plan, bias, bias, skip == "x")
    assert torch.equal(back[0], want[0])
    for a, e in zip(back[1:], want[1:]):
        _close_sums(a, e)
    _ext.check_device_errors(dev)


def test_launches_that_begin_early_see_their_operands():
    """Dependent launches of a microsecond each, all of which begin while the one before them ends: the bits of the same launches with the
    device idle in between, eager and from a graph, also where the allocator hands memory on from one to the next."""
    dev = _dev()
    g = torch.Generator(dev).manual_seed(11)
    ext = _ext.require()
    x = _cl(g, 1, 64, 24, 32)
    ws = [torch.randn(c, k, 1, 1, device=dev, generator=g) * k ** -0.5 for c, k in ((136, 64), (24, 136), (64, 24))]
    b = [torch.randn(w.shape[0], device=dev, generator=g) for w in ws]

    def chain(pause):
        y, sums = x, []
        for _ in range(4):
            for w, bi in zip(ws, b):
                y, wq, _ = ext.conv_forward(y, w, bi, None, 0, -1, False)
                pause()
                sums.append(ext.conv_backward(y, y, wq, w.shape[0], False, False, True)[2])      # column sums: two launches
                pause()
        return y, sums

    want, want_sums = chain(torch.cuda.synchronize)
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        chain(lambda: None)
        graph = torch.cuda.CUDAGraph()
    stream.synchronize()
    with torch.cuda.graph(graph, stream=stream):
        captured = chain(lambda: None)
    for k in range(20):
        if k % 2:
            graph.replay()
            y, sums = captured
        else:
            y, sums = chain(lambda: None)
        torch.cuda.synchronize()
        assert torch.equal(y, want) and all(torch.equal(a, e) for a, e in zip(sums, want_sums))
    _ext.check_device_errors(dev)


@pytest.mark.parametrize("co,ch", [(1, 8), (3, 8), (4, 24), (9, 40), (73, 384)])
def test_mlp_gradients_are_added_to_zero(co, ch):
    """Both weight gradients of an MLP start from zero, whatever the memory held, and both bias gradients are complete: numbers of values off
    and at whole vectors, sums from the slabs of the gradients and by passes of their own (fields out)."""
    dev = _dev()
    g = torch.Generator(dev).manual_seed(ch)
    ext, ci = _ext.require(), 8
    for out, layout in ((0, "nchw"), (1, "cl")) if co % 8 == 0 else ((0, "nchw"),):
        x = _cl(g, 2, ci, 8, 16)
        w1, w2 = torch.randn(ch, ci, 1, 1, device=dev, generator=g), torch.randn(co, ch, 1, 1, device=dev, generator=g)
        b1, b2 = torch.randn(ch, device=dev, generator=g), torch.randn(co, device=dev, generator=g)
        y, w1q, w2q, dact, h = ext.mlp_forward(x, w1, b1, w2, b2, None, out, True)
        dy = _as(_cl(g, 2, co, 8, 16), layout)
        held = [torch.full((k,), float("nan"), device=dev) for k in (ch * ci, co * ch, co, ch, 4096)]
        del held      # the gradients take their places
        _, dw1, db1, dw2, db2 = ext.mlp_backward(dy, x, w1q, w2q, dact, h, ci, True, True, True)
        rows = lambda t: t.double().permute(1, 0, 2, 3).flatten(1)  # noqa: E731
        dpre = (torch.einsum("oc,bohw->bchw", w2q[:, :ch].double(), dy.double()) * dact.double()).bfloat16()
        for got, ref, tol in ((dw2, rows(dy) @ rows(h).t(), 1e-6), (db2, dy.double().sum((0, 2, 3)), 1e-6),
                              (dw1, rows(dpre) @ rows(x).t(), 1e-2), (db1, dpre.double().sum((0, 2, 3)), 1e-2)):      # (dpre: other roundings)
            assert (got.double() - ref).norm() <= tol * ref.norm()
    _ext.check_device_errors(dev)
