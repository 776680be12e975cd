"""llsa_rms_rope_bwd (inverse rotation and RMSNorm backward of q and k in one launch) against the oracle's rotation and the
normalisation's gradient in fp64."""
import ctypes as C

import pytest
import torch

from llsa_b200 import _lib
from oracle import llsa_oracle as O

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
EPS = 1e-5


def _reference(dy, x, w, table, eps=EPS):
    """(dx in fp64, dw in fp64): g is the rotation's backward rounded to the data's type, as the stand-alone kernel leaves it."""
    # evaluated in the wider of the two types, as the kernel does (the oracle itself narrows the table to its tensor's type)
    g = (O.rope_bwd(dy.to(torch.promote_types(dy.dtype, table.dtype)), table).to(dy.dtype) if table is not None else dy).double()
    if w is None:
        return g, None
    xd = x.double()
    rstd = torch.rsqrt(xd.square().mean(-1, keepdim=True) + eps)
    xh, gw = xd * rstd, g * w.double()
    return rstd * (gw - xh * (gw * xh).mean(-1, keepdim=True)), (g * xh).sum((0, 1, 2))


# S: fewer rows than one pass of a CTA, one row past a chunk's end, whole chunks, several chunks per CTA
@pytest.mark.parametrize("S", [3, 129, 256, 4111])
@pytest.mark.parametrize("dtype,table,norm,view", [
    (torch.bfloat16, torch.bfloat16, True, True), (torch.bfloat16, torch.float32, False, False), (torch.bfloat16, torch.bfloat16, False, True),
    (torch.bfloat16, None, True, False), (torch.float32, torch.float32, True, True), (torch.float32, torch.float32, False, False)])
def test_rms_rope_bwd(S, dtype, table, norm, view):
    B, H, D = 2, 3, 64
    gen = torch.Generator().manual_seed(S)
    dy, x = [[torch.randn(B, H, S, D, generator=gen).to(dtype) for _ in range(2)] for _ in range(2)]
    w = [1 + 0.2 * torch.randn(D, generator=gen), None]                        # the second tensor's norm has no weight
    ang = torch.rand(S, 32, generator=gen, dtype=torch.float64) * 6.3
    tab = torch.stack([ang.sin(), ang.cos()], -1).reshape(S, D).to(table) if table is not None else None
    want = [_reference(dy[i], x[i], (w[i] if w[i] is not None else torch.ones(D)) if norm else None, tab) for i in range(2)]
    place = (lambda t: t.to(DEV).transpose(1, 2).contiguous().transpose(1, 2)) if view else (lambda t: t.to(DEV))
    dyd, xd = [place(t) for t in dy], [place(t) for t in x]
    lib, TP = _lib.lib(), C.POINTER(_lib.LlsaTensor)
    tabd, wd = (tab.to(DEV) if tab is not None else None), w[0].to(DEV)
    dw = [torch.full((D,), float("nan"), device=DEV) for _ in range(2)]
    part = torch.empty(lib.llsa_rms_rope_bwd_partial_elems(2), device=DEV)
    arr = lambda ts: (_lib.LlsaTensor * 2)(*[_lib.desc(t) for t in ts])
    wdesc, dwdesc, tdesc, pdesc = _lib.desc(wd), [_lib.desc(t) for t in dw], _lib.desc(tabd), _lib.desc(part)
    wp, dwp = (TP * 2)(C.pointer(wdesc), TP()), (TP * 2)(*[C.pointer(d) for d in dwdesc])
    dya = arr(dyd)                                                             # in place: dx is dy's memory
    _lib.check(lib.llsa_rms_rope_bwd(2, dya, arr(xd), wp, 3 if norm else 0, EPS, _lib.ref(tdesc), dya, _lib.ref(pdesc), dwp,
                                     _lib.stream_ptr(torch.device(DEV))), "rms_rope_bwd")
    for i in range(2):
        got, (dx, dwr) = dyd[i].cpu().double(), want[i]
        # one rounding to the data's type, on top of fp32 arithmetic whose terms are a few units in size (|rstd g w| < 16)
        ulp, noise = (2.0 ** -8, 2e-5) if dtype == torch.bfloat16 else (2.0 ** -23, 2e-5)
        if not norm:
            ulp, noise = 0.0, 0.0                                              # the rotation alone: the same roundings, the same bits
        assert ((got - dx).abs() <= ulp * dx.abs() + noise).all(), float((got - dx).abs().max())
        if norm:      # a sum of B H S terms in fp32: sqrt(n) 2^-24 per unit of size, with an order of magnitude to spare
            assert float((dw[i].cpu().double() - dwr).norm() / dwr.norm()) < 1e-5


# Without an eps: rows whose reciprocal root mean square, squared and times dy, is beyond a float's largest value, or below its smallest, while
# dx is well inside.  Bounds as above, in units of |rstd g|.
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("size_x,size_dy", [(1e-18, 1e4), (1e18, 1e-8)])
def test_norm_of_very_small_and_very_large_rows_without_eps(size_x, size_dy, dtype):
    gen = torch.Generator().manual_seed(5)
    dy, x = [(size * torch.randn(1, 2, 300, 64, generator=gen)).to(dtype) for size in (size_dy, size_x)]
    w = 1 + 0.2 * torch.randn(64, generator=gen)
    lib, TP = _lib.lib(), C.POINTER(_lib.LlsaTensor)
    got, dw, part = dy.to(DEV), torch.empty(64, device=DEV), torch.empty(lib.llsa_rms_rope_bwd_partial_elems(1), device=DEV)
    xd, wd = x.to(DEV), w.to(DEV)
    one = lambda t: (TP * 1)(C.pointer(t))
    dyt, xt, wt, dwt, pt = [_lib.desc(t) for t in (got, xd, wd, dw, part)]
    _lib.check(lib.llsa_rms_rope_bwd(1, _lib.ref(dyt), _lib.ref(xt), one(wt), 1, 0.0, None, _lib.ref(dyt), _lib.ref(pt), one(dwt),
                                     _lib.stream_ptr(torch.device(DEV))), "rms_rope_bwd")
    dx, dwr = _reference(dy, x, w, None, 0.0)
    ulp = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -23
    assert ((got.cpu().double() - dx).abs() <= ulp * dx.abs() + 2e-5 * size_dy / size_x).all()
    assert float((dw.cpu().double() - dwr).norm() / dwr.norm()) < 1e-5
