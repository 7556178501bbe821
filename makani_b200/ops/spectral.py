"""Spherical-harmonic spectral convolution as a chain of tensor-core GEMMs.

The reference computes `x -> SHT -> per-degree complex contraction -> inverse SHT` with cuFFT plus cuBLAS
einsums in fp32 (makani/models/common/spectral_convolution.py:124-148, contractions.py:130-136, and the
torch-harmonics RealSHT/InverseRealSHT it imports).  Here every stage is one launch of the batched GEMM
engine, and each stage writes its result directly in the layout the next one reads, so no transpose or
truncation pass ever touches HBM:

    x  [B, H, W, C]                  real grid data, channels-last (bf16)
    S1 longitude DFT      -> T1 [B, H, (m,ri), C]       A = DFT matrix [(m,ri), W], batched over latitude rows
                                                        (or folded: orders m and W / 2 - m share their products)
    S2 Legendre analysis  -> T2 [B, l, m, (ri, C)]      A = P_l^m(theta_k) w_k, batched over m, rows l < m skipped
    S3 complex contraction-> T3 [B, m, l, (ri, Co)]     B = real and imaginary planes of W_l, batched over l, rows m > l skipped
    S4 Legendre synthesis -> T4 [B, H', (m,ri), Co]     k-loop restricted to l >= m
    S5 inverse DFT        -> y  [B, H', W', Co]         (or folded: longitudes i and W' - i share their products)

(ri = real/imaginary part; the rows of all tables start on 128-byte boundaries.)
The adjoints used by the backward pass are the same five launches with the constant operands read in the
other major (no transposed copies of the tables are stored).
"""

from __future__ import annotations

import math
from typing import Dict, Optional, Tuple

import numpy as np
import torch
from torch.utils.weak import TensorWeakRef, WeakTensorKeyDictionary

from ..sht.legendre import legendre_table
from ..sht.quadrature import precompute_latitudes
from . import _ext
from .conv import records_grad
from .gemm import Operand, Output, Tri, gemm, gemm_complex, gemm_fold, pad_to, plain_columns


class SHTPlan:
    """Constant operands (DFT matrices, Legendre tables) for one (nlat, nlon, lmax, mmax, grid) transform pair."""

    _cache: Dict[Tuple, "SHTPlan"] = {}

    def __init__(self, nlat: int, nlon: int, lmax: int, mmax: int, grid: str, device, dtype=torch.bfloat16):
        self.nlat, self.nlon, self.lmax, self.mmax, self.grid = nlat, nlon, lmax, mmax, grid
        self.device, self.dtype = torch.device(device), dtype
        # rows of the tables start on 128-byte boundaries: a 128-byte row of a TMA box is then one line, not two
        self.hp = pad_to(nlat, 64)         # padded latitude extent of the Legendre tables
        self.k2 = 2 * mmax                 # DFT K extent (m, ri)
        self.k2p = pad_to(self.k2, 64)
        theta, wq = precompute_latitudes(nlat, grid)
        self.theta, self.wq = theta, wq
        p = legendre_table(mmax, lmax, theta)                     # [m, l, k] float64
        tab = np.zeros((2, mmax, lmax, self.hp), dtype=np.float32)
        np.multiply(p, wq, out=tab[0, :, :, :nlat], casting="same_kind")
        tab[1, :, :, :nlat] = p
        self.pw = torch.from_numpy(tab[0]).to(self.device, dtype).contiguous()   # analysis table (weighted)
        self.p = torch.from_numpy(tab[1]).to(self.device, dtype).contiguous()    # synthesis table
        # forward DFT rows (m, ri) ordered as ri-major: row = ri*mmax... no: row index j = 2*m + ri
        phi = 2.0 * np.pi * np.arange(nlon) / nlon
        m = np.arange(mmax)[:, None]
        ang = m * phi[None, :]
        cos, sin = np.cos(ang), np.sin(ang)
        f = np.empty((self.k2, nlon), dtype=np.float32)
        f[0::2] = cos * (2.0 * np.pi / nlon)
        f[1::2] = -sin * (2.0 * np.pi / nlon)
        self.f = torch.from_numpy(f).to(self.device, dtype).contiguous()      # [(m,ri), W]
        # inverse DFT: x_i = sum_m c_m (Xr cos - Xi sin); c_0 = 1, c_m = 2, Nyquist (if kept) = 1
        cm = np.full((mmax, 1), 2.0)
        cm[0] = 1.0
        if nlon % 2 == 0 and mmax > nlon // 2:
            cm[nlon // 2] = 1.0
        g = np.zeros((nlon, self.k2p), dtype=np.float32)
        g[:, 0:self.k2:2] = (cm * cos).T
        g[:, 1:self.k2:2] = (-cm * sin).T
        self.gt = torch.from_numpy(g).to(self.device, dtype).contiguous()     # [W, (m,ri) padded]

        # The same matrices with their columns in two halves, for `gemm_fold`.  The synthesis (rows are longitudes) may fold from the 64
        # rows on that `gemm_fold` asks for.  The analysis (rows (m, ri)) only saves work where most orders up to half the points are
        # kept, order m sharing its products with order W / 2 - m; orders past half the points, which alias, have no mirror and
        # stay whole.  `folding_pays` decides for a number of channels.
        self.folds_synthesis = nlon >= 64
        self.folds_analysis = (nlon >= 64 and nlon % 2 == 0 and 8 * mmax > 3 * nlon and
                               nlon // 2 + 32 <= 2 * mmax <= nlon + 2)
        self._folded = self._fold_tables()

        # what the native passes take: matrices (empty where one is not folded) and extents
        none = torch.empty(0, device=self.device, dtype=dtype)
        self.native = ([self.f, self.gt, self.pw, self.p] + [self._folded.get((syn, fwd), none) for syn in (True, False) for fwd in (True, False)],
                       [nlat, nlon, lmax, mmax])

    def _fold_tables(self) -> Dict[Tuple[bool, bool], torch.Tensor]:
        """(synthesis, forward) -> the inverse transform's matrix (`synthesis`; rows are longitudes, halves the cosine and sine terms)
        or the forward one's (rows (m, ri), halves the even and odd points), from the coefficients of the forward transform
        (`forward`) or of the inverse one.  Symmetric to the bit: a row and its mirror hold the same numbers, and those that cancel
        are zero.  The halves start on 128-byte boundaries, so that a TMA row is one line (721 x 1440: 364 -> 336 us)."""
        W, mmax = self.nlon, self.mmax
        if not (self.folds_synthesis or self.folds_analysis):
            return {}
        h, angle = W // 2, 2.0 * np.pi * np.arange(W) / W
        at = np.arange(mmax)[:, None] * np.arange(W)[None, :] % W
        cos, sin = np.cos(angle)[at], np.sin(angle)[at]              # [m, i]
        tables = {}
        for forward in (True, False):
            scale = np.full((mmax, 1), 2.0 * np.pi / W if forward else 2.0)
            if not forward:
                scale[0] = 1.0
                if W % 2 == 0 and mmax > W // 2:
                    scale[W // 2] = 1.0
            c, s = scale * cos, -scale * sin
            if self.folds_synthesis:
                t = np.zeros((W, 2, pad_to(mmax, 64)), dtype=np.float32)
                t[:, 0, :mmax], t[:, 1, :mmax] = c.T, s.T
                t[h + 1:, 0], t[h + 1:, 1] = t[W - h - 1:0:-1, 0], -t[W - h - 1:0:-1, 1]
                t[0, 1] = 0.0
                if W % 2 == 0:
                    t[h, 1] = 0.0
                tables[True, forward] = t
            if self.folds_analysis:
                t = np.zeros((mmax, 2, 2, pad_to(h, 64)), dtype=np.float32)                  # [m, ri, half, point]
                for ri, x in enumerate((c, s)):
                    t[:, ri, 0, :h], t[:, ri, 1, :h] = x[:, 0::2], x[:, 1::2]
                if h % 2 == 0 and h // 2 < mmax:
                    t[h // 2, 0, 1] = t[h // 2, 1, 0] = 0.0
                m = np.arange(h // 2 + 1, mmax)
                t[m] = t[h - m] * np.array([[1.0, -1.0], [-1.0, 1.0]], dtype=np.float32)[:, :, None]
                tables[False, forward] = t.reshape(2 * mmax, 2, -1)
        return {k: torch.from_numpy(t.reshape(t.shape[0], -1)).to(self.device, self.dtype).contiguous() for k, t in tables.items()}

    @classmethod
    def get(cls, nlat, nlon, lmax, mmax, grid, device, dtype=torch.bfloat16) -> "SHTPlan":
        key = (nlat, nlon, lmax, mmax, grid, str(torch.device(device)), dtype)
        plan = cls._cache.get(key)
        if plan is None:
            plan = cls(nlat, nlon, lmax, mmax, grid, device, dtype)
            cls._cache[key] = plan
        return plan


# ------------------------------------------------------------------------------------------------ stages
# Activations are channels-last: x is logically [B, C, H, W] and physically [B][k][i][c] (k latitude, i longitude).
# Row index of the DFT side is j = 2*m + ri.  T1 / T4 are [B, H, 2*mmax, C]; T2 is [B, l, m, (ri, C)];
# T3 is [B, m, l, (ri, Co)].


def _to_cl(x: torch.Tensor) -> torch.Tensor:
    if x.is_contiguous(memory_format=torch.channels_last) and not (x.is_contiguous() and x.shape[1] != 1):
        return x
    return x.contiguous(memory_format=torch.channels_last)


def dft_analysis(x: torch.Tensor, mat: torch.Tensor, mat_mn: bool, mat_ld: int, k2: int) -> torch.Tensor:
    """T1[b, k, j, c] = sum_i M[j, i] x[b, c, k, i];  M given K-major ([j, i]) or MN-major ([i, j])."""
    B, C, H, W = x.shape
    t1 = torch.empty(B, H, k2, C, dtype=x.dtype, device=x.device)
    gemm(k2, C, W,
         Operand(mat, ld=mat_ld, mn_major=mat_mn),
         Operand(x, ld=C, mn_major=True, zs_lo=W * C, zs_hi=H * W * C),
         Output(t1, rs_lo=C, d_zlo=k2 * C, d_zhi=H * k2 * C),
         zlo_n=H, zhi_n=B)
    return t1


def dft_synthesis(t4: torch.Tensor, mat: torch.Tensor, mat_mn: bool, mat_ld: int, W: int) -> torch.Tensor:
    """y[b, c, k, i] = sum_j T4[b, k, j, c] M[i, j];  M given K-major ([i, j]) or MN-major ([j, i]).  y is channels-last."""
    B, H, k2, C = t4.shape
    y = torch.empty(B, C, H, W, dtype=t4.dtype, device=t4.device, memory_format=torch.channels_last)
    gemm(W, C, k2,
         Operand(mat, ld=mat_ld, mn_major=mat_mn),
         Operand(t4, ld=C, mn_major=True, zs_lo=k2 * C, zs_hi=H * k2 * C),
         Output(y, rs_lo=C, d_zlo=W * C, d_zhi=H * W * C),
         zlo_n=H, zhi_n=B)
    return y


def folding_pays(rows: int, folded_rows: int, k: int, folded_k: int, C: int) -> bool:
    """Whether a folded product of two halves of `folded_k` columns beats the whole one: fewer columns of 128-row tiles, each counted
    with its slabs of 64 products and one more for its epilogue.  The folded product halves rows or products, but rounds them up
    to whole tiles and slabs once more (129 of 256 rows are two tiles, as all 256 are; 32 orders are one slab, and two halves of them
    two) and has tiles of 128 columns only.  Some 1700 transforms of 64 to 1440 points, 8 to 361 orders and 16 to 768 channels: always
    folding takes 3.9 % more than the better of the two, never 9.9 %, this rule 0.6 %.  Synthesis, us, whole / folded: 1440 points, 64
    orders, 136 channels 102 / 88, 264 channels 281 / 144; 256 points, 129 orders, 384 channels 24 / 30; 128 points, 32 orders,
    768 channels 27 % slower folded.  The native passes (csrc/layers.cpp) have the same rule."""
    tiles = lambda r, w: -(-r // 128) * -(-C // w) * w      # noqa: E731
    return tiles(folded_rows, 128) * (2 * -(-folded_k // 64) + 1) < tiles(rows, plain_columns(C)) * (-(-k // 64) + 1)


def folded_analysis(x: torch.Tensor, plan: SHTPlan, forward: bool = True) -> torch.Tensor:
    B, C, H, W = x.shape
    k2, table = plan.k2, plan._folded[False, forward]
    t1 = torch.empty(B, H, k2, C, dtype=x.dtype, device=x.device)
    gemm_fold(k2, 2 * (W // 4 + 1), C, W // 2, W, True, table, table.shape[1] // 2,
              Operand(x, ld=2 * C, mn_major=True, zs_hi=W * C), C, Output(t1, rs_lo=C, d_zhi=k2 * C), zhi_n=B * H)
    return t1


def folded_synthesis(t4: torch.Tensor, plan: SHTPlan, forward: bool = False) -> torch.Tensor:
    B, H, k2, C = t4.shape
    W, table = plan.nlon, plan._folded[True, forward]
    y = torch.empty(B, C, H, W, dtype=t4.dtype, device=t4.device, memory_format=torch.channels_last)
    gemm_fold(W, W // 2 + 1, C, k2 // 2, W, False, table, table.shape[1] // 2,
              Operand(t4, ld=2 * C, mn_major=True, zs_hi=k2 * C), C, Output(y, rs_lo=C, d_zhi=W * C), zhi_n=B * H)
    return y


def analyse(x: torch.Tensor, plan: SHTPlan, forward: bool = True) -> torch.Tensor:
    """Longitude DFT of x (`forward`), or the adjoint of the inverse one: [B, H, (m, ri), C].  (The whole matrix of the forward transform
    has rows of W columns: only the folded ones are aligned for any W.)"""
    W = plan.nlon
    if plan.folds_analysis and (folding_pays(plan.k2, 2 * (W // 4 + 1), W, W // 2, x.shape[1]) or (forward and W % 8)):
        return folded_analysis(x, plan, forward)
    return dft_analysis(x, plan.f, False, W, plan.k2) if forward else dft_analysis(x, plan.gt, True, plan.k2p, plan.k2)


def synthesise(t4: torch.Tensor, plan: SHTPlan, forward: bool = False) -> torch.Tensor:
    """Inverse longitude DFT of t4 [B, H, (m, ri), C], or the adjoint of the forward one (`forward`); channels-last.  t4 may hold
    fewer orders than the plan: those of a forward transform that keeps fewer than the inverse one."""
    W, k2 = plan.nlon, t4.shape[2]
    if plan.folds_synthesis and (folding_pays(W, W // 2 + 1, k2, k2 // 2, t4.shape[3]) or (forward and W % 8)):
        return folded_synthesis(t4, plan, forward)
    return dft_synthesis(t4, plan.f, True, W, W) if forward else dft_synthesis(t4, plan.gt, False, plan.k2p, W)


def legendre_analysis(t1: torch.Tensor, table: torch.Tensor, by_order: bool = False) -> torch.Tensor:
    """T2[b, l, m, n] = sum_k table[m, l, k] T1[b, k, m, n], n = (ri, c);  zero for l < m.  `by_order`: as [b, m, l, n]."""
    B, H, k2, C = t1.shape
    mmax, lmax, hpt = table.shape
    n2 = 2 * C
    t2 = torch.empty(*((B, mmax, lmax) if by_order else (B, lmax, mmax)), n2, dtype=t1.dtype, device=t1.device)
    gemm(lmax, n2, H,
         Operand(table, ld=hpt, zs_hi=lmax * hpt),
         Operand(t1, ld=k2 * C, mn_major=True, zs_hi=n2, zs_lo=H * k2 * C),
         Output(t2, rs_lo=n2 if by_order else mmax * n2, d_zhi=lmax * n2 if by_order else n2, d_zlo=lmax * mmax * n2),
         zhi_n=mmax, zlo_n=B, tri=Tri(rmin_a=1))
    return t2


def legendre_synthesis(t: torch.Tensor, lm_order: bool, table: torch.Tensor, H: int) -> torch.Tensor:
    """T4[b, k, m, n] = sum_l table[m, l, k] T[b, ., ., n]  with T given as [b, m, l, n] (lm_order False)
    or [b, l, m, n] (lm_order True); only l >= m contributes."""
    if lm_order:
        B, lmax, mmax, n2 = t.shape
        ld, zs_m = mmax * n2, n2
    else:
        B, mmax, lmax, n2 = t.shape
        ld, zs_m = n2, lmax * n2
    hpt = table.shape[2]
    t4 = torch.empty(B, H, 2 * mmax, n2 // 2, dtype=t.dtype, device=t.device)
    gemm(H, n2, lmax,
         Operand(table, ld=hpt, mn_major=True, zs_hi=lmax * hpt),
         Operand(t, ld=ld, mn_major=True, zs_hi=zs_m, zs_lo=lmax * mmax * n2),
         Output(t4, rs_lo=mmax * n2, d_zhi=n2, d_zlo=H * mmax * n2),
         zhi_n=mmax, zlo_n=B, tri=Tri(kmin_a=1))
    return t4


def contract(t2: torch.Tensor, wx: torch.Tensor, transpose_w: bool, resid=None) -> torch.Tensor:
    """T3[b, m, l, q] = sum_p T2[b, l, m, p] Wx[l, q, p]   (transpose_w False; Wx [l, 2Co, 2Ci])
       T3[b, m, l, p] = sum_q T2[b, l, m, q] Wx[l, q, p]   (transpose_w True: adjoint w.r.t. the input)
    plus `resid`, which has the layout of the result.  Wx is the real block form or the planes of `weight_planes`."""
    B, lmax, mmax, kin = t2.shape
    if wx.dim() == 4:
        # planes [l, 2, Co, Ci]: half the bytes of the real block matrix, in memory and through L2
        co, ci = wx.shape[2], wx.shape[3]
        n, k = (ci, co) if transpose_w else (co, ci)
        t3 = torch.empty(B, mmax, lmax, 2 * n, dtype=t2.dtype, device=t2.device)
        gemm_complex(2 if transpose_w else 1, mmax, n, k,
                     Operand(t2, ld=kin, zs_hi=mmax * kin, zs_lo=lmax * mmax * kin),
                     Operand(wx, ld=ci, mn_major=transpose_w, zs_hi=2 * co * ci),
                     Output(t3, rs_lo=lmax * 2 * n, d_zhi=2 * n, d_zlo=mmax * lmax * 2 * n), n, zhi_n=lmax, zlo_n=B,
                     b_plane=co * ci, resid=resid, rmax=(1, 1))
        return t3
    nq, npp = wx.shape[1], wx.shape[2]
    nout = npp if transpose_w else nq
    t3 = torch.empty(B, mmax, lmax, nout, dtype=t2.dtype, device=t2.device)
    gemm(mmax, nout, kin,
         Operand(t2, ld=kin, zs_hi=mmax * kin, zs_lo=lmax * mmax * kin),
         Operand(wx, ld=npp, mn_major=transpose_w, zs_hi=nq * npp),
         Output(t3, rs_lo=lmax * nout, d_zhi=nout, d_zlo=mmax * lmax * nout),
         zhi_n=lmax, zlo_n=B, tri=Tri(rmax_a=1, rmax_b=1), resid=resid)
    return t3


def contract_wgrad2(dt: torch.Tensor, t2: torch.Tensor, l0: int = 0, m0: int = 0) -> torch.Tensor:
    """(dWr, dWi)[l, o, c] as fp32 [2, L, Co, Ci] without forming the full real 2x2-block gradient:

        dWr[l, o, c] = sum_{b, m <= l} dTr T2r + dTi T2i        dWi[l, o, c] = sum_{b, m <= l} dTi T2r - dTr T2i

    One complex product over the planes of both operands per sample.  `l0`, `m0`: global offsets of the local (l, m) block."""
    B, L, M, nq = dt.shape
    co, ci = nq // 2, t2.shape[3] // 2
    dt, t2 = dt.contiguous(), t2.contiguous()
    out = (torch.empty if B == 1 else torch.zeros)(2, L, co, ci, dtype=torch.float32, device=dt.device)
    for b in range(B):
        gemm_complex(3, co, ci, M,
                     Operand(dt, ld=nq, mn_major=True, zs_hi=M * nq, offset=b * L * M * nq),
                     Operand(t2, ld=2 * ci, mn_major=True, zs_hi=M * 2 * ci, offset=b * L * M * 2 * ci),
                     Output(out, rs_lo=ci, d_zhi=co * ci), L * co * ci, zhi_n=L, a_plane=co, b_plane=ci, accumulate=(B > 1),
                     kmax=(1, 1 + l0 - m0))
    return out


def fold_weight_grad2(dw2: torch.Tensor) -> torch.Tensor:
    """fp32 [2, L, Co, Ci] = (dWr, dWi) -> complex64 [Ci, Co, L]."""
    _, L, co, ci = dw2.shape
    if dw2.is_cuda and _ext.native():
        dw = torch.empty(ci, co, L, dtype=torch.complex64, device=dw2.device)
        _ext.require().spectral_fold(dw2, dw, True, True)
        return dw
    return torch.complex(dw2[0], dw2[1]).permute(2, 1, 0).contiguous()


def weight_gradient(dt: torch.Tensor, t2: torch.Tensor) -> torch.Tensor:
    """Both at once for a whole transform: on the GPU one launch per sample that writes complex64 [Ci, Co, L] (csrc/spectral_wgrad.cu)."""
    if dt.is_cuda and _ext.native():
        return _ext.require().spectral_weight_gradient(dt, t2)
    return fold_weight_grad2(contract_wgrad2(dt, t2))


# ------------------------------------------------------------------------------------------------ weights


# Inference re-uses the expanded weights: they are kept as long as the parameter lives (a weak key, so that a new
# parameter in recycled memory never meets them), and dropped when the parameter is modified in place (`_version`) or by
# a writer that `_version` does not see and that says so through `note_weights_changed` (the fused optimiser, which writes
# through raw pointers, and every write to `.data`).  They serve the stream that made them only, and never a capture: a
# captured pass expands the weights itself, so that its replays read the values of the day from memory of their own.
#
# Training shares an expansion among the forward passes that are recorded before the first of their graphs is gone (the steps of
# a roll-out): only a weak reference is kept, so the last graph takes the expansion with it and nothing outlives the
# backward pass, also where weights are written through `.data` without a word (averaged weights swapped in and out).
# Inside a capture the passes of that capture share one.  Two roll-out steps: one cast of 69 us and one copy of 142 MB per
# block of 384 channels and 240 degrees instead of two.
_WEIGHT_EPOCH = 0
_EXPANDED = WeakTensorKeyDictionary()      # parameter -> (state, expansion), inference
_RECORDED = WeakTensorKeyDictionary()      # parameter -> (state, weak reference to the expansion), training


def note_weights_changed() -> None:
    global _WEIGHT_EPOCH
    _WEIGHT_EPOCH += 1
    for table in (_EXPANDED, _RECORDED):
        if len(table):
            table.clear()


def expand_weight(w: torch.Tensor, dtype=torch.bfloat16, keep: bool = False, share: bool = False) -> torch.Tensor:
    """complex [Ci, Co, L] -> real [L, 2Co, 2Ci] with rows (ri', o), columns (ri, c):  [[Wr, -Wi], [Wi, Wr]].

    `keep`: the caller does not record gradients, the result is kept with the parameter for its next call.
    `share`: the caller records them, the result is shared with other calls as long as a recorded graph holds it."""
    return _kept(w, dtype, _expand_weight, keep, share)


def weight_planes(w: torch.Tensor, dtype=torch.bfloat16, keep: bool = False, share: bool = False) -> torch.Tensor:
    """complex [Ci, Co, L] -> its real and imaginary planes [L, 2, Co, Ci]."""
    return _kept(w, dtype, _planes, keep, share)


def _planes(w: torch.Tensor, dtype) -> torch.Tensor:
    if not w.is_cuda or dtype != torch.bfloat16:
        return torch.stack([w.real, w.imag]).permute(3, 0, 2, 1).to(dtype).contiguous()
    ci, co, L = w.shape
    wp = torch.empty(L, 2, co, ci, dtype=dtype, device=w.device)
    _ext.require().spectral_planes(w.detach().contiguous(), wp)
    return wp


def _kept(w: torch.Tensor, dtype, make, keep: bool, share: bool) -> torch.Tensor:
    if not (keep or share) or not w.is_cuda or w.is_inference():
        return make(w, dtype)
    stream, capture = _ext.require().stream_state(w.device.index)
    if capture < 0 or (capture and keep):
        return make(w, dtype)
    state = (w._version, _WEIGHT_EPOCH, w.data_ptr(), dtype, make, stream, capture)
    table = _EXPANDED if keep else _RECORDED
    hit = table.get(w)
    if hit is not None and hit[0] == state:
        wx = hit[1] if keep else hit[1]()
        if wx is not None:
            return wx
    wx = make(w, dtype)
    table[w] = (state, wx if keep else TensorWeakRef(wx))
    return wx


def _expand_weight(w: torch.Tensor, dtype=torch.bfloat16) -> torch.Tensor:
    ci, co, L = w.shape
    if w.is_cuda and dtype == torch.bfloat16:
        wx = torch.empty(L, 2 * co, 2 * ci, dtype=dtype, device=w.device)
        _ext.require().spectral_expand(w.detach().contiguous(), wx)
        return wx
    wr = w.real.permute(2, 1, 0)
    wi = w.imag.permute(2, 1, 0)
    top = torch.cat([wr, -wi], dim=2)
    bot = torch.cat([wi, wr], dim=2)
    return torch.cat([top, bot], dim=1).to(dtype).contiguous()


def fold_weight_grad(dwx: torch.Tensor) -> torch.Tensor:
    """fp32 [L, 2Co, 2Ci] -> complex64 [Ci, Co, L] gradient (dWr = d00 + d11, dWi = d10 - d01)."""
    L, co2, ci2 = dwx.shape
    co, ci = co2 // 2, ci2 // 2
    if dwx.is_cuda:
        dw = torch.zeros(ci, co, L, dtype=torch.complex64, device=dwx.device)
        _ext.require().spectral_fold(dwx.contiguous(), dw)
        return dw
    d00, d01 = dwx[:, :co, :ci], dwx[:, :co, ci:]
    d10, d11 = dwx[:, co:, :ci], dwx[:, co:, ci:]
    return torch.complex(d00 + d11, d10 - d01).permute(2, 1, 0).contiguous()


# ------------------------------------------------------------------------------------------------ autograd


def forward_stages(x, wx, plan_in: SHTPlan, plan_out: SHTPlan, want_resid: bool):
    """(y, r or None, T2), launch by launch: the pass on the CPU, and what `spectral_forward` of csrc/layers.cpp does on the GPU."""
    t1 = analyse(x, plan_in)
    t2 = legendre_analysis(t1, plan_in.pw)
    del t1
    t3 = contract(t2, wx, False)
    t4 = legendre_synthesis(t3, False, plan_out.p, plan_out.nlat)
    del t3
    y = synthesise(t4, plan_out)
    del t4
    r = None
    if want_resid:
        t4r = legendre_synthesis(t2, True, plan_out.p, plan_out.nlat)
        r = synthesise(t4r, plan_out)
    return y, r, t2


def backward_stages(dy, dr, t2, wx, plan_in: SHTPlan, plan_out: SHTPlan, need_x: bool, need_w: bool):
    """(dx, dw) as `spectral_backward` of csrc/layers.cpp has them on the GPU; dr: the gradient of the residual, or None."""
    # adjoint of the inverse DFT / synthesis on the output grid
    dt4 = analyse(dy, plan_out, forward=False)
    dt3 = legendre_analysis(dt4, plan_out.p)                       # [B, l, m, (ri, o)]
    del dt4
    dw = weight_gradient(dt3, t2) if need_w else None
    dx = None
    if need_x:
        dr2 = None
        if dr is not None:
            # laid out by order, as the contraction writes: its epilogue adds the residual's share
            dr4 = analyse(dr, plan_out, forward=False)
            dr2 = legendre_analysis(dr4, plan_out.p, by_order=True)
            del dr4
        dt2 = contract(dt3, wx, True, resid=dr2)                   # [B, m, l, (ri, c)]
        del dr2
        dt1 = legendre_synthesis(dt2, False, plan_in.pw, plan_in.nlat)
        dx = synthesise(dt1, plan_in, forward=True)
    return dx, dw


class _SpectralConv(torch.autograd.Function):
    """y = iSHT_out(W . SHT_in(x)) and, when `want_resid`, r = iSHT_out(SHT_in(x)) (regridded residual).
    Input and outputs are channels-last."""

    @staticmethod
    def forward(ctx, x, w, plan_in: SHTPlan, plan_out: SHTPlan, want_resid: bool, train: bool):
        x = _to_cl(x)
        wx = weight_planes(w, x.dtype, keep=not train, share=train)
        ctx.plans = (plan_in, plan_out)
        ctx.want_resid = want_resid
        ctx.wshape = w.shape
        if x.is_cuda:
            y, r, t2 = _ext.require().spectral_forward(x, wx, *plan_in.native, *plan_out.native, want_resid)
        else:
            y, r, t2 = forward_stages(x, wx, plan_in, plan_out, want_resid)
        ctx.save_for_backward(t2, wx)
        return (y, r) if want_resid else y

    @staticmethod
    def backward(ctx, dy, dr=None):
        t2, wx = ctx.saved_tensors
        plan_in, plan_out = ctx.plans
        dy = _to_cl(dy)
        dr = _to_cl(dr) if ctx.want_resid and dr is not None else None
        if dy.is_cuda:
            dx, dw = _ext.require().spectral_backward(dy, dr, t2, wx, *plan_in.native, *plan_out.native, ctx.needs_input_grad[0],
                                                      ctx.needs_input_grad[1])
        else:
            dx, dw = backward_stages(dy, dr, t2, wx, plan_in, plan_out, ctx.needs_input_grad[0], ctx.needs_input_grad[1])
        return dx, (None if dw is None else dw.reshape(ctx.wshape)), None, None, None, None


def spectral_conv_supported(x: torch.Tensor, w: torch.Tensor) -> bool:
    return (_ext.native() and x.dim() == 4 and x.dtype == torch.bfloat16 and x.shape[1] % 8 == 0 and w.dim() == 3 and w.shape[1] % 8 == 0
            and x.shape[3] % 8 == 0)


def spectral_conv_dhconv(x, w, plan_in: SHTPlan, plan_out: SHTPlan, want_resid: bool):
    """Fused spherical convolution with per-degree ("dhconv") complex weights on the GEMM engine."""
    return _SpectralConv.apply(x, w, plan_in, plan_out, want_resid, records_grad(x, w))
