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
    (2, 16, 24, 33, 64, 16, 32, 16, 17, 17, True),       # folded to whole, regridded residual
    (1, 40, 8, 48, 96, 45, 90, 40, 46, 46, True),        # 90 longitudes out: an odd half; ragged channels
    (2, 8, 16, 32, 64, 33, 65, 32, 33, 33, False),       # an odd number of longitudes out
    (1, 136, 72, 40, 80, 40, 80, 40, 41, 41, False),     # two column tiles, both transforms folded both ways
    (2, 16, 16, 24, 48, 24, 48, 24, 25, 25, False),      # nothing folded
    (1, 16, 32, 48, 96, 48, 96, 40, 12, 12, True),       # few orders: the analysis stays whole
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
