"""Performance cases of the framework: what a training or forecast program asks of it, through its public entry points.

Every case is one pass through a module, an optimiser step or a whole network, in the data type its users run it in
(bf16 activations with fp32 parameters; complex64 for the mode-wise operators; fp32 for the optimiser).  Sizes are those
of the recipes in `config/` (721 x 1440 grid, internal grid 240 x 480 or 360 x 720, 384 channels, 73 fields, 90 x 180
tokens of 768 channels) and of the small plumbing recipe (32 x 64, 16 channels).

`prepare` makes inputs and parameters from a seed on the GPU, `run` is one pass, `exact` the same pass in float64 with
plain torch (own quadrature, Legendre and Fourier formulas).
"""

import functools
import math

import numpy as np
import torch
import torch.nn.functional as F

DEV = "cuda"
BF = torch.bfloat16


# ---------------------------------------------------------------------------------------------------- cases

def listed():
    return [
        # the plumbing recipe: launches and host latency count; a whole training pass with all gradients
        dict(name="tiny_sfno_train", kind="sfno_train", B=2, H=32, W=64, scale=1, chans=4, embed=16, layers=2),
        # one 6 h step of an autoregressive forecast with the 73-field network, batch 1; four of its eight blocks, so that the
        # rounding of two correct implementations (which every block multiplies) stays comparable
        dict(name="sfno_forecast_step", kind="sfno_infer", B=1, H=721, W=1440, scale=3, chans=73, embed=384, layers=4),
        # block MLP on the internal grid: seven of the eight blocks of a training step
        dict(name="mlp_internal_train", kind="mlp", B=1, H=240, W=480, C=384, hidden=768),
        # block MLP of the last block, which works on the full grid
        dict(name="mlp_full_train", kind="mlp", B=1, H=721, W=1440, C=384, hidden=768),
        # decoder: 384 channels to 73 fields in NCHW (an odd channel count and a ragged number of tokens)
        dict(name="decoder_full_train", kind="decoder", B=1, H=721, W=1440, C=384, out=73),
        # spherical convolution on the internal grid, weights per degree
        dict(name="spectral_internal_train", kind="spectral", B=1, H=240, W=480, Ho=240, Wo=480, C=384, lmax=240, mmax=241),
        # spherical convolution of the first block: full grid to internal grid, with the regridded residual
        dict(name="spectral_down_train", kind="spectral", B=1, H=721, W=1440, Ho=240, Wo=480, C=384, lmax=240, mmax=241),
        # instance norm + GELU behind the filter of the last block
        dict(name="norm_gelu_full_train", kind="norm", B=1, H=721, W=1440, C=384, gelu=True),
        # AFNO token mixer: 720 x 1440 in 8 x 8 patches, 768 channels in 8 blocks
        dict(name="afno_filter_train", kind="afno", B=1, H=90, W=180, C=768, blocks=8),
        # token MLP of AFNO / ViT, ratio 4
        dict(name="token_mlp_train", kind="token_mlp", B=1, T=16200, C=768, hidden=3072),
        # mode-wise ("diagonal") operator of the planar FNO recipes: 360 x 720 internal grid, half of the modes, 64 channels
        dict(name="diagonal_modes_train", kind="diagonal", B=1, C=64, L=180, M=180),
        # AdamW over the parameters of two blocks
        dict(name="adamw_step", kind="adamw", C=384, hidden=768, lmax=240, layers=2),
    ]


def _log(rng, lo, hi, step=1):
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(lo, min(hi, int(round(v / step)) * step))


def draw(rng):
    """One more case of the same ranges: from the plumbing sizes to the full grid, odd numbers of rows and tokens among them."""
    kind = rng.choice(["mlp", "mlp", "decoder", "spectral", "spectral", "norm", "afno", "token_mlp", "diagonal", "sfno_train", "adamw"])
    H = _log(rng, 32, 721)
    W = max(64, (2 * H) // 16 * 16)
    C = _log(rng, 128 if H * W > 18000 else 16, 384, 8)      # the narrow networks of the recipes work on small grids
    B = 2 if H * W <= 360 * 720 and rng.random() < 0.4 else 1
    if kind == "mlp":
        return dict(kind=kind, B=B, H=H, W=W, C=C, hidden=2 * C)
    if kind == "decoder":
        return dict(kind=kind, B=B, H=H, W=W, C=C, out=rng.randint(4, 96))
    if kind == "norm":
        return dict(kind=kind, B=B, H=H, W=W, C=C, gelu=rng.random() < 0.6)
    if kind == "spectral":
        Ho = H if rng.random() < 0.5 else max(16, H // rng.choice([2, 3]))
        Wo = W if Ho == H else max(32, (2 * Ho) // 16 * 16)
        lmax = min(240, Ho)
        return dict(kind=kind, B=B, H=H, W=W, Ho=Ho, Wo=Wo, C=C, lmax=lmax, mmax=min(lmax + 1, Wo // 2 + 1))
    if kind == "afno":
        h = _log(rng, 8, 90)
        return dict(kind=kind, B=rng.choice([1, 2]), H=h, W=2 * h, C=rng.choice([256, 512, 768]), blocks=8)
    if kind == "token_mlp":
        c = _log(rng, 128, 768, 8)
        return dict(kind=kind, B=rng.choice([1, 2]), T=_log(rng, 256, 8100), C=c, hidden=4 * c)
    if kind == "diagonal":
        m = _log(rng, 24, 180)
        return dict(kind=kind, B=rng.choice([1, 2]), C=_log(rng, 16, 64), L=m, M=m + rng.randint(0, 1))
    if kind == "sfno_train":
        h = rng.randint(24, 72)
        return dict(kind=kind, B=rng.choice([1, 2]), H=h, W=2 * h // 16 * 16, scale=1, chans=rng.choice([4, 8, 20]),
                    embed=_log(rng, 16, 64, 8), layers=2)
    return dict(kind=kind, C=C, hidden=2 * C, lmax=_log(rng, 32, 240), layers=rng.choice([1, 2]))


# ---------------------------------------------------------------------------------------------------- inputs

def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _randn(g, *shape, scale=1.0, dtype=torch.float32):
    return (torch.randn(*shape, device=DEV, generator=g, dtype=dtype) * scale)


def _field(g, B, C, H, W):
    """A channels-last activation as the blocks hand it on."""
    return torch.randn(B, H, W, C, device=DEV, generator=g, dtype=BF).permute(0, 3, 1, 2)


def _sfno_shape(case):
    h, w = case["H"] // case["scale"], case["W"] // case["scale"]
    return h, w, h, w // 2 + 1        # internal grid, lmax, mmax


def _sfno_params(g, case):
    """Parameters by their names in the network's state dict."""
    E, L, cin, cout = case["embed"], case["layers"], case["chans"] + 1, case["chans"]
    _, _, lmax, _ = _sfno_shape(case)
    p = {}

    def w1x1(name, co, ci, gain, bias=False):
        p[name + ".weight"] = _randn(g, co, ci, 1, 1, scale=math.sqrt(gain / ci))
        if bias:
            p[name + ".bias"] = _randn(g, co, scale=0.05)

    w1x1("encoder.fwd.0", E, cin, 2.0, True)
    w1x1("encoder.fwd.2", E, E, 1.0)
    for i in range(L):
        b = "blocks.%d." % i
        p[b + "filter.filter.weight"] = _randn(g, E, E, lmax, scale=math.sqrt(2.0 / E), dtype=torch.complex64)
        for n in ("norm0", "norm1"):
            p[b + n + ".weight"] = 1.0 + _randn(g, E, scale=0.1)
            p[b + n + ".bias"] = _randn(g, E, scale=0.1)
        w1x1(b + "mlp.fwd.0", 2 * E, E, 2.0, True)
        w1x1(b + "mlp.fwd.3", E, 2 * E, 0.5, True)
        w1x1(b + "outer_skip", E, E, 0.5)
    w1x1("decoder.fwd.0", E, E, 2.0, True)
    w1x1("decoder.fwd.2", cout, E, 0.5)
    w1x1("residual_transform", cout, cin, 0.5)
    return p


def _has_grad(name):
    """The bias in front of an instance norm has no gradient but rounding noise: the norm takes the mean away again."""
    return not name.endswith("mlp.fwd.3.bias")


def _inputs(case, seed):
    """Tensors of one case, from the seed alone."""
    g, k = _gen(seed), case["kind"]
    if k in ("sfno_train", "sfno_infer"):
        t = dict(params=_sfno_params(g, case), x=_randn(g, case["B"], case["chans"] + 1, case["H"], case["W"]).to(BF))
        if k == "sfno_train":
            t["target"] = _randn(g, case["B"], case["chans"], case["H"], case["W"]).to(BF)
        return t
    if k == "mlp":
        C, Hd = case["C"], case["hidden"]
        return dict(x=_field(g, case["B"], C, case["H"], case["W"]), dy=_field(g, case["B"], C, case["H"], case["W"]),
                    w1=_randn(g, Hd, C, 1, 1, scale=math.sqrt(2.0 / C)), b1=_randn(g, Hd, scale=0.05),
                    w2=_randn(g, C, Hd, 1, 1, scale=math.sqrt(1.0 / Hd)), b2=_randn(g, C, scale=0.05))
    if k == "decoder":
        C, O = case["C"], case["out"]
        return dict(x=_field(g, case["B"], C, case["H"], case["W"]), dy=_randn(g, case["B"], O, case["H"], case["W"]).to(BF),
                    w1=_randn(g, C, C, 1, 1, scale=math.sqrt(2.0 / C)), b1=_randn(g, C, scale=0.05),
                    w2=_randn(g, O, C, 1, 1, scale=math.sqrt(0.5 / C)))
    if k == "spectral":
        C = case["C"]
        t = dict(x=_field(g, case["B"], C, case["H"], case["W"]), dy=_field(g, case["B"], C, case["Ho"], case["Wo"]),
                 w=_randn(g, C, C, case["lmax"], scale=math.sqrt(1.0 / C), dtype=torch.complex64))
        if _regrids(case):
            t["dr"] = _field(g, case["B"], C, case["Ho"], case["Wo"])
        return t
    if k == "norm":
        C = case["C"]
        # fields behind a filter: every channel has a mean and a spread of its own
        x = _field(g, case["B"], C, case["H"], case["W"]).float()
        x = x * (0.5 + torch.rand(1, C, 1, 1, device=DEV, generator=g)) + torch.randn(1, C, 1, 1, device=DEV, generator=g)
        return dict(x=x.to(BF), dy=_field(g, case["B"], C, case["H"], case["W"]), w=1.0 + _randn(g, C, scale=0.1),
                    b=_randn(g, C, scale=0.1))
    if k == "afno":
        C, nb = case["C"], case["blocks"]
        bs = C // nb
        sc = math.sqrt(1.0 / bs)
        return dict(x=_randn(g, case["B"], case["H"], case["W"], C, dtype=BF), dy=_randn(g, case["B"], case["H"], case["W"], C, dtype=BF),
                    w1=_randn(g, 2, nb, bs, bs, scale=sc), b1=_randn(g, 2, nb, bs, scale=0.1), w2=_randn(g, 2, nb, bs, bs, scale=sc),
                    b2=_randn(g, 2, nb, bs, scale=0.1))
    if k == "token_mlp":
        C, Hd = case["C"], case["hidden"]
        return dict(x=_randn(g, case["B"], case["T"], C, dtype=BF), dy=_randn(g, case["B"], case["T"], C, dtype=BF),
                    w1=_randn(g, Hd, C, scale=math.sqrt(2.0 / C)), b1=_randn(g, Hd, scale=0.05),
                    w2=_randn(g, C, Hd, scale=math.sqrt(1.0 / Hd)), b2=_randn(g, C, scale=0.05))
    if k == "diagonal":
        B, C, L, M = case["B"], case["C"], case["L"], case["M"]
        c64 = torch.complex64
        return dict(x=_randn(g, B, C, L, M, dtype=c64), w=_randn(g, C, C, L, M, scale=math.sqrt(1.0 / C), dtype=c64),
                    dy=_randn(g, B, C, L, M, dtype=c64))
    if k == "adamw":
        C, Hd = case["C"], case["hidden"]
        shapes = []
        for _ in range(case["layers"]):
            shapes += [((C, C, case["lmax"]), torch.complex64)]
            shapes += [(s, torch.float32) for s in ((Hd, C, 1, 1), (Hd,), (C, Hd, 1, 1), (C,), (C, C, 1, 1), (C,), (C,), (C,), (C,))]
        t = []
        for s, d in shapes:
            p, gr, m = _randn(g, *s, scale=0.05, dtype=d), _randn(g, *s, scale=1e-3, dtype=d), _randn(g, *s, scale=1e-3, dtype=d)
            r = torch.rand(*s, *((2,) if d.is_complex else ()), device=DEV, generator=g) * 1e-6
            t.append((p, gr, m, torch.view_as_complex(r) if d.is_complex else r))
        return dict(params=t)
    raise ValueError(k)


def _regrids(case):
    return (case["H"], case["W"]) != (case["Ho"], case["Wo"])


def _grids(case):
    """Grid types as the network lays them out: full-grid fields are equiangular, the internal grid is Gaussian."""
    return ("equiangular", "legendre-gauss") if _regrids(case) else ("legendre-gauss", "legendre-gauss")


# ---------------------------------------------------------------------------------------------------- prepare / run

@functools.lru_cache(maxsize=64)
def _transform(forward, nlat, nlon, lmax, mmax, grid):
    from makani_b200.sht import InverseRealSHT, RealSHT
    return (RealSHT if forward else InverseRealSHT)(nlat, nlon, lmax=lmax, mmax=mmax, grid=grid).to(DEV)


def _fill(module, tensors):
    with torch.no_grad():
        for name, p in module.named_parameters():
            p.copy_(tensors[name])
    _weights_set()
    return module


def _weights_set():
    """What an optimiser step or a restart announces: weights have new values, nothing derived from them may be kept."""
    from makani_b200.ops.spectral import note_weights_changed
    note_weights_changed()


def _sfno(case, params):
    from makani_b200.models.networks.sfnonet import SphericalFourierNeuralOperatorNet
    with torch.device(DEV):
        net = SphericalFourierNeuralOperatorNet(
            spectral_transform="sht", model_grid_type="equiangular", sht_grid_type="legendre-gauss", filter_type="linear",
            operator_type="dhconv", inp_shape=(case["H"], case["W"]), out_shape=(case["H"], case["W"]), scale_factor=case["scale"],
            inp_chans=case["chans"] + 1, out_chans=case["chans"], embed_dim=case["embed"], num_layers=case["layers"],
            use_mlp=True, mlp_ratio=2.0, activation_function="gelu", encoder_layers=1, pos_embed="none",
            normalization_layer="instance_norm", hard_thresholding_fraction=1.0, big_skip=True)
    net = _fill(net.to(DEV), params)
    net.set_compute_dtype(BF)
    return net


def _state(module, t):
    return dict(module=module, params=list(module.parameters()), x=t["x"].requires_grad_(True), dy=t["dy"])


def prepare(case, seed):
    t, k = _inputs(case, seed), case["kind"]
    if k in ("sfno_train", "sfno_infer"):
        s = dict(kind=k, net=_sfno(case, t["params"]), x=t["x"])
        if k == "sfno_infer":
            s["net"].eval()
            return s
        from makani_b200.utils.losses import GeometricLpLoss
        hw = (case["H"], case["W"])
        s["net"].train()
        s["loss"] = GeometricLpLoss(hw, hw, (0, 0), p=2, absolute=True, squared=True).to(DEV)
        s["target"], s["params"] = t["target"], [p for n, p in sorted(s["net"].named_parameters()) if _has_grad(n)]
        s["chw"] = torch.full((1, case["chans"]), 1.0 / case["chans"], device=DEV)
        return s
    if k == "mlp":
        from makani_b200.models.common.layers import MLP
        with torch.device(DEV):
            m = MLP(case["C"], hidden_features=case["hidden"])
        m = _fill(m, {"fwd.0.weight": t["w1"], "fwd.0.bias": t["b1"], "fwd.3.weight": t["w2"], "fwd.3.bias": t["b2"]})
        return dict(_state(m, t), kind="module")
    if k == "decoder":
        from makani_b200.models.common.layers import EncoderDecoder
        with torch.device(DEV):
            m = EncoderDecoder(1, case["C"], case["out"], case["C"], torch.nn.GELU, gain=0.5)
        m = _fill(m, {"fwd.0.weight": t["w1"], "fwd.0.bias": t["b1"], "fwd.2.weight": t["w2"]})
        return dict(_state(m, t), kind="module")
    if k == "spectral":
        from makani_b200.models.common.spectral_convolution import SpectralConv
        gi, go = _grids(case)
        fwd = _transform(True, case["H"], case["W"], case["lmax"], case["mmax"], gi)
        inv = _transform(False, case["Ho"], case["Wo"], case["lmax"], case["mmax"], go)
        with torch.device(DEV):
            m = SpectralConv(fwd, inv, case["C"], case["C"], operator_type="dhconv")
        m = _fill(m, {"weight": t["w"]})
        return dict(_state(m, t), kind="spectral", dr=t.get("dr"))
    if k == "norm":
        from makani_b200.models.networks.sfnonet import InstanceNorm2d
        with torch.device(DEV):
            m = InstanceNorm2d(case["C"], eps=1e-6, affine=True, track_running_stats=False)
        m = _fill(m, {"weight": t["w"], "bias": t["b"]})
        return dict(_state(m, t), kind="norm", act="gelu" if case["gelu"] else "none")
    if k == "afno":
        from makani_b200.models.networks.afnonet import AFNO2D
        with torch.device(DEV):
            m = AFNO2D(case["C"], num_blocks=case["blocks"], sparsity_threshold=0.01, hard_thresholding_fraction=1.0)
        return dict(_state(_fill(m, t), t), kind="module")
    if k == "token_mlp":
        from makani_b200.models.networks.afnonet import Mlp
        with torch.device(DEV):
            m = Mlp(case["C"], hidden_features=case["hidden"])
        m = _fill(m, {"fc1.weight": t["w1"], "fc1.bias": t["b1"], "fc2.weight": t["w2"], "fc2.bias": t["b2"]})
        return dict(_state(m, t), kind="module")
    if k == "diagonal":
        from makani_b200.models.common.contractions import get_contract_fun
        w = t["w"].requires_grad_(True)
        fn = get_contract_fun("diagonal", False)
        return dict(module=lambda x: fn(x, w), params=[w], x=t["x"].requires_grad_(True), dy=t["dy"], kind="module")
    from makani_b200.ops.optim import FusedAdamW
    params = [torch.nn.Parameter(p) for p, _, _, _ in t["params"]]
    opt = FusedAdamW(params, lr=1e-3, betas=(0.9, 0.95), weight_decay=0.01)
    sd = opt.state_dict()
    sd["state"] = {i: {"step": torch.tensor(10.0), "exp_avg": m, "exp_avg_sq": v} for i, (_, _, m, v) in enumerate(t["params"])}
    opt.load_state_dict(sd)
    for p, (_, gr, _, _) in zip(params, t["params"]):
        p.grad = gr
    return dict(kind="adamw", opt=opt, params=params)


def run(s):
    k = s["kind"]
    if k in ("sfno_train", "spectral"):
        _weights_set()      # in training every pass meets weights that the optimiser has just changed
    if k == "sfno_infer":
        with torch.no_grad():
            return s["net"](s["x"])
    if k == "sfno_train":
        y = s["net"](s["x"])
        loss = s["loss"](y, s["target"], s["chw"])
        return [y.detach(), loss.detach()] + list(torch.autograd.grad(loss, s["params"]))
    if k == "adamw":
        s["opt"].step()
        st = s["opt"].state
        return [[p.detach(), st[p]["exp_avg"], st[p]["exp_avg_sq"]] for p in s["params"]]
    if k == "spectral":
        y, r = s["module"](s["x"])
        if s["dr"] is not None:
            return [y.detach(), r.detach()] + list(torch.autograd.grad([y, r], [s["x"]] + s["params"], [s["dy"], s["dr"]]))
        return [y.detach()] + list(torch.autograd.grad(y, [s["x"]] + s["params"], s["dy"]))
    y = s["module"](s["x"], act=s["act"]) if k == "norm" else s["module"](s["x"])
    return [y.detach()] + list(torch.autograd.grad(y, [s["x"]] + s["params"], s["dy"]))


# ---------------------------------------------------------------------------------------------------- work

def _sht_flops(B, C, H, W, lmax, mmax):
    """Longitude DFT as a dense product plus the Legendre stage over l >= m, one direction, real operations."""
    pairs = sum(max(0, lmax - m) for m in range(mmax))
    return B * C * (2.0 * H * W * 2 * mmax + 2.0 * H * pairs * 2)


def _spectral_work(B, C, H, W, Ho, Wo, lmax, mmax, resid, train):
    T, To = B * H * W, B * Ho * Wo
    pairs = sum(max(0, lmax - m) for m in range(mmax))
    f_in, f_out = _sht_flops(B, C, H, W, lmax, mmax), _sht_flops(B, C, Ho, Wo, lmax, mmax)
    mix = 8.0 * B * pairs * C * C
    n = 2 if resid else 1
    wbytes = 8.0 * C * C * lmax
    if not train:
        return 2.0 * C * (T + n * To) + wbytes, f_in + mix + n * f_out
    # x and the output gradients in, outputs and the input gradient out, weight in and its gradient out
    return 2.0 * C * (2 * T + 2 * n * To) + 2 * wbytes, 2 * (f_in + n * f_out) + 3 * mix


def work(case):
    k = case["kind"]
    if k == "mlp" or k == "token_mlp":
        T = case["B"] * (case["T"] if k == "token_mlp" else case["H"] * case["W"])
        C, Hd = case["C"], case["hidden"]
        return {"bytes": 2.0 * T * C * 4 + 4.0 * 2 * (2 * C * Hd + C + Hd), "flops": 3 * 2 * 2.0 * T * C * Hd}
    if k == "decoder":
        T, C, O = case["B"] * case["H"] * case["W"], case["C"], case["out"]
        return {"bytes": 2.0 * T * (2 * C + 2 * O) + 8.0 * (C * C + C + C * O), "flops": 3 * 2.0 * T * (C * C + C * O)}
    if k == "spectral":
        b, f = _spectral_work(case["B"], case["C"], case["H"], case["W"], case["Ho"], case["Wo"], case["lmax"], case["mmax"],
                              _regrids(case), True)
        return {"bytes": b, "flops": f}
    if k == "norm":
        n = float(case["B"] * case["H"] * case["W"] * case["C"])
        return {"bytes": 2 * n * 4 + 16.0 * case["C"], "flops": 40 * n}
    if k == "afno":
        B, H, W, C, nb = case["B"], case["H"], case["W"], case["C"], case["blocks"]
        bs, modes = C // nb, B * H * (W // 2 + 1)
        dft = 2.0 * B * H * W * 2 * (W // 2 + 1) * C + 2.0 * modes * 2 * 2 * H * C
        return {"bytes": 2.0 * B * H * W * C * 4 + 2 * 4.0 * 4 * (nb * bs * bs + nb * bs), "flops": 4 * dft + 3 * 2 * 8.0 * modes * C * bs}
    if k == "diagonal":
        n = case["L"] * case["M"]
        B, C = case["B"], case["C"]
        return {"bytes": 8.0 * n * (2 * C * C + 4 * B * C), "flops": 3 * 8.0 * B * C * C * n}
    if k == "adamw":
        C, Hd = case["C"], case["hidden"]
        n = case["layers"] * (2.0 * C * C * case["lmax"] + 2 * C * Hd + Hd + C * C + 6 * C)
        return {"bytes": 4 * 7 * n, "flops": 12 * n}
    E, L, cin, cout, B, H, W = case["embed"], case["layers"], case["chans"] + 1, case["chans"], case["B"], case["H"], case["W"]
    h, w, lmax, mmax = _sfno_shape(case)
    T, t = B * H * W, B * h * w
    conv = 2.0 * T * (cin * E + E * E + E * E + E * cout + cin * cout) + 2.0 * (T + (L - 1) * t) * (4 * E * E + E * E)
    pairs = sum(max(0, lmax - m) for m in range(mmax))
    resid = (H, W) != (h, w)
    sht = 0.0
    for i in range(L):
        hi, ho = (H, W) if i == 0 else (h, w), (H, W) if i == L - 1 else (h, w)
        sht += _sht_flops(B, E, hi[0], hi[1], lmax, mmax) + (2 if hi != ho and resid else 1) * _sht_flops(B, E, ho[0], ho[1], lmax, mmax)
    mix = 8.0 * B * pairs * E * E * L
    nparams = 2.0 * E * E * lmax * L + L * (5 * E * E + 7 * E) + cin * E + 2 * E * E + 2 * E + E * cout + cin * cout
    if k == "sfno_infer":
        return {"bytes": 2.0 * T * (cin + cout) + 4 * nparams, "flops": conv + sht + mix}
    return {"bytes": 2.0 * T * (cin + 2 * cout) + 8 * nparams, "flops": 3 * (conv + mix) + 2 * sht}


# ---------------------------------------------------------------------------------------------------- tolerances

def tolerance(case):
    """bf16 activations (8 bits of mantissa) between the stages of a layer; about four times the distance from float64
    measured for each kind, within what one layer or a whole network may show."""
    k = case["kind"]
    if k == "adamw" or k == "diagonal":
        return {"rel": 1e-5, "max": 1e-3}
    if k == "sfno_infer" or k == "sfno_train":
        return {"rel": 3e-2, "max": 0.5}
    return {"rel": 1.5e-2, "max": 0.2}


# ---------------------------------------------------------------------------------------------------- float64

@functools.lru_cache(maxsize=16)
def _latitudes(n, grid):
    """(cos of colatitude from north to south, quadrature weights summing to 2)."""
    if grid == "legendre-gauss":
        x, w = np.polynomial.legendre.leggauss(n)
        return x[::-1].copy(), w[::-1].copy()
    # equiangular with both poles: weights that integrate the cosine series of the samples (Clenshaw and Curtis)
    th = np.pi * np.arange(n) / (n - 1)
    w = np.ones(n)
    for j in range(1, (n - 1) // 2 + 1):
        w -= (1.0 if 2 * j == n - 1 else 2.0) / (4.0 * j * j - 1.0) * np.cos(2 * j * th)
    w *= 2.0 / (n - 1)
    w[[0, -1]] *= 0.5
    return np.cos(th), w


@functools.lru_cache(maxsize=6)
def _legendre64(n, grid, lmax, mmax):
    """P[m, l, k] (orthonormal on the sphere, zero for l < m) and quadrature weights, float64 on the GPU."""
    x, w = _latitudes(n, grid)
    x, w = torch.from_numpy(x).to(DEV), torch.from_numpy(w).to(DEV)
    s = torch.sqrt(torch.clamp(1.0 - x * x, min=0.0))
    P = torch.zeros(mmax, lmax, n, dtype=torch.float64, device=DEV)
    diag = torch.full((n,), math.sqrt(0.25 / math.pi), dtype=torch.float64, device=DEV)
    for m in range(min(mmax, lmax)):
        if m:
            diag = diag * s * math.sqrt((2 * m + 1) / (2.0 * m))
        P[m, m] = diag
    # degree by degree: P_l = a (x P_{l-1} - c P_{l-2}), all orders at once
    for l in range(1, lmax):
        m = torch.arange(min(l, mmax), dtype=torch.float64, device=DEV)[:, None]
        a = torch.sqrt((4.0 * l * l - 1.0) / (l * l - m * m))
        v = x[None] * P[: m.shape[0], l - 1]
        if l > 1:
            c = torch.sqrt(((l - 1.0) ** 2 - m * m).clamp(min=0.0) / (4.0 * (l - 1.0) ** 2 - 1.0))
            v = v - c * P[: m.shape[0], l - 2]
        P[: m.shape[0], l] = a * v
    return P, w


def _sht64(x, grid, lmax, mmax):
    """Real field [B, C, H, W] -> coefficients [B, C, l, m]."""
    P, w = _legendre64(x.shape[2], grid, lmax, mmax)
    f = torch.fft.rfft(x, dim=-1)[..., :mmax] * (2.0 * math.pi / x.shape[3])
    f = torch.view_as_real(f).permute(3, 2, 0, 1, 4).reshape(mmax, x.shape[2], -1)          # [m, k, (b c ri)]
    c = torch.bmm(P * w, f).reshape(mmax, lmax, x.shape[0], x.shape[1], 2)
    return torch.view_as_complex(c.permute(2, 3, 1, 0, 4).contiguous())


def _isht64(c, H, W, grid):
    """Coefficients [B, C, l, m] -> real field [B, C, H, W]."""
    B, C, lmax, mmax = c.shape
    P, _ = _legendre64(H, grid, lmax, mmax)
    v = torch.view_as_real(c).permute(3, 2, 0, 1, 4).reshape(mmax, lmax, -1)
    f = torch.bmm(P.transpose(1, 2), v).reshape(mmax, H, B, C, 2).permute(2, 3, 1, 0, 4).contiguous()
    return torch.fft.irfft(torch.view_as_complex(f), n=W, dim=-1, norm="forward")


def _filter64(x, w, Ho, Wo, gi, go, lmax, mmax, resid):
    c = _sht64(x, gi, lmax, mmax)
    y = torch.einsum("bilm,iol->bolm", c, w)
    return _isht64(y, Ho, Wo, go), (_isht64(c, Ho, Wo, go) if resid else None)


def _lin64(x, w, b=None):
    y = torch.einsum("oc,bchw->bohw", w.reshape(w.shape[0], -1), x)
    return y if b is None else y + b[None, :, None, None]


def _norm64(x, w, b):
    m = x.mean(dim=(2, 3), keepdim=True)
    v = (x - m).square().mean(dim=(2, 3), keepdim=True)
    return (x - m) / torch.sqrt(v + 1e-6) * w[None, :, None, None] + b[None, :, None, None]


def _afno64(x, w1, b1, w2, b2, lam=0.01):
    """Every kept mode of the real FFT through the block MLP (fraction 1 keeps `H // 2 + 1` columns and all rows but none twice)."""
    B, H, W, C = x.shape
    nb, bs = w1.shape[1], w1.shape[2]
    total = H // 2 + 1
    rows, cols = slice(0, min(2 * total, H)), slice(0, min(total, W // 2 + 1))
    X = torch.fft.rfft2(x, dim=(1, 2), norm="ortho").reshape(B, H, W // 2 + 1, nb, bs)[:, rows, cols]
    mul = lambda re, im, w: (torch.einsum("...ni,nio->...no", re, w[0]) - torch.einsum("...ni,nio->...no", im, w[1]),  # noqa: E731
                             torch.einsum("...ni,nio->...no", im, w[0]) + torch.einsum("...ni,nio->...no", re, w[1]))
    r, i = mul(X.real, X.imag, w1)
    r, i = mul(F.relu(r + b1[0]), F.relu(i + b1[1]), w2)
    r, i = F.softshrink(r + b2[0], lam), F.softshrink(i + b2[1], lam)
    Y = torch.zeros(B, H, W // 2 + 1, nb, bs, dtype=torch.complex128, device=x.device)
    Y[:, rows, cols] = torch.complex(r, i)
    return torch.fft.irfft2(Y.reshape(B, H, W // 2 + 1, C), s=(H, W), dim=(1, 2), norm="ortho") + x


def _sfno64(case, p, x):
    H, W, L = case["H"], case["W"], case["layers"]
    h, w, lmax, mmax = _sfno_shape(case)
    y = _lin64(F.gelu(_lin64(x, p["encoder.fwd.0.weight"], p["encoder.fwd.0.bias"])), p["encoder.fwd.2.weight"])
    for i in range(L):
        b = "blocks.%d." % i
        first, last = i == 0, i == L - 1
        gi, go = "equiangular" if first else "legendre-gauss", "equiangular" if last else "legendre-gauss"
        Ho, Wo = (H, W) if last else (h, w)
        differ = (y.shape[2], y.shape[3], gi) != (Ho, Wo, go)
        y, r = _filter64(y, p[b + "filter.filter.weight"], Ho, Wo, gi, go, lmax, mmax, differ) if differ else (
            _filter64(y, p[b + "filter.filter.weight"], Ho, Wo, gi, go, lmax, mmax, False)[0], y)
        y = F.gelu(_norm64(y, p[b + "norm0.weight"], p[b + "norm0.bias"]))
        y = _lin64(F.gelu(_lin64(y, p[b + "mlp.fwd.0.weight"], p[b + "mlp.fwd.0.bias"])), p[b + "mlp.fwd.3.weight"], p[b + "mlp.fwd.3.bias"])
        y = _norm64(y, p[b + "norm1.weight"], p[b + "norm1.bias"]) + _lin64(r, p[b + "outer_skip.weight"])
        del r
    y = _lin64(F.gelu(_lin64(y, p["decoder.fwd.0.weight"], p["decoder.fwd.0.bias"])), p["decoder.fwd.2.weight"])
    return y + _lin64(x, p["residual_transform.weight"])


def _d(t):
    return t.detach().to(torch.complex128 if t.is_complex() else torch.float64)


def _grads(y, leaves, dy):
    return list(torch.autograd.grad(y, leaves, dy))


def exact(case, seed):
    t, k = _inputs(case, seed), case["kind"]
    if k == "sfno_infer":
        with torch.no_grad():
            return _sfno64(case, {n: _d(v) for n, v in t["params"].items()}, _d(t["x"]))
    if k == "sfno_train":
        p = {n: _d(v).requires_grad_(True) for n, v in t["params"].items()}
        y = _sfno64(case, p, _d(t["x"]))
        # area weights of the rows of the equiangular grid, normalised to a mean over the sphere
        n, m = case["H"], case["W"]
        q = torch.from_numpy(np.sin(np.linspace(0.0, np.pi, n))).to(DEV)
        q = q * (np.pi / n) * (2.0 * np.pi / m)
        q = q / (q.sum() * m)
        e = ((y - _d(t["target"])).square() * q[None, None, :, None]).sum(dim=(2, 3))
        loss = (e / case["chans"]).sum()
        return [y.detach(), loss.detach()] + _grads(loss, [p[n] for n in sorted(p) if _has_grad(n)], None)
    if k in ("mlp", "decoder"):
        x, w1, b1, w2 = (_d(t[n]).requires_grad_(True) for n in ("x", "w1", "b1", "w2"))
        b2 = _d(t["b2"]).requires_grad_(True) if k == "mlp" else None
        y = _lin64(F.gelu(_lin64(x, w1, b1)), w2, b2)
        return [y.detach()] + _grads(y, [x, w1, b1, w2] + ([b2] if b2 is not None else []), _d(t["dy"]))
    if k == "token_mlp":
        x, w1, b1, w2, b2 = (_d(t[n]).requires_grad_(True) for n in ("x", "w1", "b1", "w2", "b2"))
        y = F.linear(F.gelu(F.linear(x, w1, b1)), w2, b2)
        return [y.detach()] + _grads(y, [x, w1, b1, w2, b2], _d(t["dy"]))
    if k == "spectral":
        x, w = _d(t["x"]).requires_grad_(True), _d(t["w"]).requires_grad_(True)
        gi, go = _grids(case)
        y, r = _filter64(x, w, case["Ho"], case["Wo"], gi, go, case["lmax"], case["mmax"], _regrids(case))
        if r is None:
            return [y.detach()] + _grads(y, [x, w], _d(t["dy"]))
        return [y.detach(), r.detach()] + list(torch.autograd.grad([y, r], [x, w], [_d(t["dy"]), _d(t["dr"])]))
    if k == "norm":
        x, w, b = (_d(t[n]).requires_grad_(True) for n in ("x", "w", "b"))
        y = _norm64(x, w, b)
        y = F.gelu(y) if case["gelu"] else y
        return [y.detach()] + _grads(y, [x, w, b], _d(t["dy"]))
    if k == "afno":
        x, w1, b1, w2, b2 = (_d(t[n]).requires_grad_(True) for n in ("x", "w1", "b1", "w2", "b2"))
        y = _afno64(x, w1, b1, w2, b2)
        return [y.detach()] + _grads(y, [x, w1, b1, w2, b2], _d(t["dy"]))
    if k == "diagonal":
        # written out so that one input channel at a time is in float64 with its weights
        x, w, dy = _d(t["x"]), t["w"], _d(t["dy"])
        y, dx, dw = torch.zeros_like(dy), torch.empty_like(x), torch.empty(w.shape, dtype=torch.complex128, device=DEV)
        for i in range(w.shape[0]):
            wi = _d(w[i])
            y += x[:, i, None] * wi[None]
            dx[:, i] = (dy * wi.conj()[None]).sum(1)
            dw[i] = (x[:, i, None].conj() * dy).sum(0)
        return [y, dx, dw]
    out = []
    for p, gr, m, v in t["params"]:
        ri = lambda z: torch.view_as_real(_d(z)) if z.is_complex() else _d(z)  # noqa: E731
        P, G, M, V = ri(p), ri(gr), ri(m), ri(v)
        lr, b1, b2, eps, wd, step = 1e-3, 0.9, 0.95, 1e-8, 0.01, 11
        M, V = b1 * M + (1 - b1) * G, b2 * V + (1 - b2) * G * G
        P = P * (1 - lr * wd) - lr / (1 - b1 ** step) * M / (torch.sqrt(V) / math.sqrt(1 - b2 ** step) + eps)
        back = (lambda z: torch.view_as_complex(z.contiguous())) if p.is_complex() else (lambda z: z)
        out.append([back(P), back(M), back(V)])
    return out
