"""Row kernels at the edges of their forms: evo_sum_norm (rows in registers up to 4096 columns, shared memory beyond, single elements), evo_conv_act (batches of rows,
chunks of 32, carried inputs) and evo_rmsnorm (a CTA per row, or a warp)."""
import ctypes as C
import os
import sys

import pytest
import torch

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
from evo_b200 import _lib  # noqa: E402
from evo_b200._lib import ConvActParams, SumNormParams, check, ptr  # noqa: E402

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _stream():
    return C.c_void_p(torch.cuda.current_stream().cuda_stream)


def _near(got, want, dtype):
    # fp32: rounding of a few operations; bf16: one rounding of the result (half a step of 2^-8) and the fp32 ones
    rel = 2e-6 if dtype == torch.float32 else 2.0 ** -8
    assert ((got.double() - want).abs() <= rel * want.abs() + 1e-6 * want.abs().max()).all()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("D,ldo,branches,normed,scaled,outs,gather", [
    (4, 64, 1, False, False, 1, False), (1020, 1024, 2, True, False, 2, False), (1024, 1024, 0, False, False, 1, True), (1028, 1088, 3, True, True, 2, False), (2048, 2048, 2, False, True, 2, False),
    (2052, 2112, 1, True, False, 1, True), (4096, 4096, 3, False, False, 2, False), (4096, 4160, 2, True, True, 0, False), (4100, 4160, 2, True, False, 2, False), (1023, 1024, 2, False, True, 1, False)])
def test_sum_norm(dtype, D, ldo, branches, normed, scaled, outs, gather):
    g = torch.Generator(device=DEV).manual_seed(D)
    n = lambda *s: torch.randn(*s, generator=g, device=DEV)  # noqa: E731
    R = 37
    x, ys = n(R, D), [n(R, D + 4 * b).to(dtype) for b in range(branches)]
    nw, ws = [(1 + 0.2 * n(D)).bfloat16() for _ in range(branches)], [(1 + 0.2 * n(D)).bfloat16() for _ in range(outs)]
    cs = n(D).bfloat16() if scaled else None
    idx = torch.tensor([5, 0, 36, 5], device=DEV) if gather else None
    rows = 4 if gather else R
    rms = lambda v: v / torch.sqrt((v * v).mean(-1, keepdim=True) + 1e-6)  # noqa: E731
    add = torch.zeros(R, D, dtype=torch.float64, device=DEV)
    for b in range(branches):
        y = ys[b][:, :D].double()
        add += (0.5 + b) * (rms(y) * nw[b].double() if normed else y)
    want = x.double() + (add * cs.double() if scaled else add)
    p = SumNormParams(x=x.data_ptr(), n_branches=branches, eps=1e-6, dtype=int(dtype == torch.float32), rows=rows, D=D, ldo=ldo, gather=idx.data_ptr() if gather else None,
                      col_scale=cs.data_ptr() if scaled else None)
    for b in range(branches):
        p.y[b], p.ldy[b], p.norm_w[b], p.scale[b] = ys[b].data_ptr(), ys[b].shape[1], nw[b].data_ptr() if normed else None, 0.5 + b
    got = [torch.full((rows, ldo), 3.0, dtype=dtype, device=DEV) for _ in range(outs)]
    for i in range(outs):
        p.out[i], p.w[i] = got[i].data_ptr(), ws[i].data_ptr()
    before = x.clone()
    check(_lib.lib().evo_sum_norm(C.byref(p), _stream()), "evo_sum_norm")
    if gather:
        assert torch.equal(x, before)
    else:
        _near(x, want, torch.float32)
    for i in range(outs):
        _near(got[i][:, :D], (rms(want) * ws[i].double())[idx if gather else slice(None)], dtype)
        assert not got[i][:, D:].any()


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("B,L,C_,taps,carried", [(2, 1, 64, 4, True), (1, 2, 64, 4, True), (2, 3, 68, 3, False), (1, 31, 64, 4, True), (2, 32, 64, 2, False), (2, 33, 64, 4, True), (1, 34, 128, 4, False),
                                                 (3, 37, 68, 4, False), (2, 64, 64, 1, False), (1, 67, 66, 4, True), (1, 100, 64, 6, False)])
def test_conv_act(dtype, B, L, C_, taps, carried):
    g = torch.Generator(device=DEV).manual_seed(L * 10 + taps)
    x, w = (2 * torch.randn(B * L, C_ + 12, generator=g, device=DEV)).to(dtype), (0.5 * torch.randn(C_, taps, generator=g, device=DEV)).bfloat16()
    bias, carry = torch.randn(C_, generator=g, device=DEV).bfloat16(), torch.randn(B, max(taps - 1, 1), C_, generator=g, device=DEV)
    pre = carry[:, :taps - 1].double() if carried else torch.zeros(B, taps - 1, C_, dtype=torch.float64, device=DEV)
    z = torch.cat([pre, x.view(B, L, -1)[:, :, :C_].double()], 1)
    want = torch.nn.functional.silu(sum(z[:, j:j + L] * w[:, j].double() for j in range(taps)) + bias.double()).reshape(B * L, C_)
    out = torch.empty(B * L, C_, dtype=dtype, device=DEV)
    p = ConvActParams(inp=x.data_ptr(), ld=x.shape[1], weight=w.data_ptr(), bias=bias.data_ptr(), carry=carry.data_ptr(), zero_start=int(not carried), out=out.data_ptr(), ldo=C_,
                      B=B, L=L, C=C_, taps=taps, act=1, dtype=int(dtype == torch.float32))
    check(_lib.lib().evo_conv_act(C.byref(p), _stream()), "evo_conv_act")
    _near(out, want, dtype)
    if taps > 1:
        assert torch.equal(carry, z[:, L:].float())


# CTAs of more than 32 rows that end in 1 to 7 rows, sequences that are more than a wave of CTAs, taps that start on two bytes, no activation, no bias
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("B,L,C_,taps,act,off,carried", [(40, 257, 2048, 4, 1, 0, True), (40, 262, 2048, 4, 0, 1, True), (37, 263, 2044, 3, 1, 1, False), (700, 43, 512, 2, 1, 0, True),
                                                          (1, 39, 64, 4, 1, 3, True), (3, 46, 64, 1, 1, 1, False), (2, 8, 64, 4, 1, 0, True), (2, 5, 64, 3, 0, 0, True)])
def test_conv_act_splits(dtype, B, L, C_, taps, act, off, carried):
    g = torch.Generator(device=DEV).manual_seed(L)
    x, buf = torch.randn(B * L, C_ + 4, generator=g, device=DEV).to(dtype), (0.5 * torch.randn(C_ * taps + 8, generator=g, device=DEV)).bfloat16()
    w, carry = buf[off:off + C_ * taps].view(C_, taps), torch.randn(B, max(taps - 1, 1), C_, generator=g, device=DEV)
    z = torch.cat([carry[:, :taps - 1].double() if carried else torch.zeros(B, taps - 1, C_, dtype=torch.float64, device=DEV), x.view(B, L, -1)[:, :, :C_].double()], 1)
    want = sum(z[:, j:j + L] * w[:, j].double() for j in range(taps)).reshape(B * L, C_)
    out = torch.empty(B * L, C_, dtype=dtype, device=DEV)
    p = ConvActParams(inp=x.data_ptr(), ld=x.shape[1], weight=w.data_ptr(), carry=carry.data_ptr(), zero_start=int(not carried), out=out.data_ptr(), ldo=C_, B=B, L=L, C=C_, taps=taps,
                      act=act, dtype=int(dtype == torch.float32))
    check(_lib.lib().evo_conv_act(C.byref(p), _stream()), "evo_conv_act")
    _near(out, torch.nn.functional.silu(want) if act else want, dtype)
    if taps > 1:
        assert torch.equal(carry, z[:, L:].float())


def test_conv_act_limits():
    """SiLU far from zero and beyond: large negative inputs end at (minus) zero, infinities and NaN as in v / (1 + e^-v)."""
    v = torch.tensor([-1e38, -200.0, -89.0, -30.0, 0.0, 30.0, 200.0, 1e38, float("inf"), float("-inf"), float("nan"), -1.0], device=DEV).bfloat16().view(1, 12)
    w, out = torch.ones(12, 1, device=DEV).bfloat16(), torch.empty(1, 12, device=DEV, dtype=torch.bfloat16)
    p = ConvActParams(inp=v.data_ptr(), ld=12, weight=w.data_ptr(), out=out.data_ptr(), ldo=12, zero_start=1, B=1, L=1, C=12, taps=1, act=1, dtype=0)
    check(_lib.lib().evo_conv_act(C.byref(p), _stream()), "evo_conv_act")
    f = v.float()
    want = f / (1 + torch.exp(-f))
    assert torch.equal(torch.isnan(out), torch.isnan(want))
    ok = ~torch.isnan(want)
    assert ((out.float() - want)[ok & torch.isfinite(want)].abs() <= 2.0 ** -8 * want[ok & torch.isfinite(want)].abs() + 1e-30).all()
    assert torch.equal(out.float()[torch.isinf(want)], want[torch.isinf(want)])


def test_conv_act_silu_of_every_bf16_number():
    """The activation of every finite bf16 argument within half a step of bf16 plus 2^-20 of the result in 64 bits, also where e^-v is beyond fp32's 1 / x (from -87.3 down)."""
    bits = torch.arange(1 << 16, dtype=torch.int32, device=DEV).to(torch.int16)
    v = bits.view(torch.bfloat16)
    v = torch.where(torch.isfinite(v.float()), v, torch.zeros_like(v)).view(1024, 64)
    for lo in range(0, 1024, 32):
        x = v[lo:lo + 32].contiguous()
        w, out = torch.ones(64, 1, device=DEV).bfloat16(), torch.empty(32, 64, device=DEV, dtype=torch.bfloat16)
        p = ConvActParams(inp=x.data_ptr(), ld=64, weight=w.data_ptr(), out=out.data_ptr(), ldo=64, zero_start=1, B=1, L=32, C=64, taps=1, act=1, dtype=0)
        check(_lib.lib().evo_conv_act(C.byref(p), _stream()), "evo_conv_act")
        d = x.double()
        want = d * torch.exp(torch.minimum(d, torch.zeros_like(d))) / (1 + torch.exp(-d.abs()))
        # the step of bf16 at `want`: 2^-7 of its power of two; 2^-133 below its smallest normal number.  silu_f ends at zero from -88.73 (e^-v overflows) on
        step = torch.exp2(torch.floor(torch.log2(want.abs().clamp(min=2.0 ** -126))) - 7)
        err = (out.double() - want).abs()
        ok = (err <= 0.5 * step + 2.0 ** -20 * want.abs() + 2.0 ** -134) | ((d < -88.7) & (out == 0))
        assert ok.all(), (x[~ok][:4], out[~ok][:4], want[~ok][:4])


@pytest.mark.parametrize("rows,D", [(65, 256), (2048, 2048), (2049, 2048), (8192, 4096), (8193, 4096), (1024, 1024), (1025, 1024), (12288, 4096), (12289, 4096), (300, 8192), (12300, 8192), (70, 4352)])
def test_rmsnorm_forms(rows, D):
    g = torch.Generator(device=DEV).manual_seed(rows)
    x, s = torch.randn(rows, D, generator=g, device=DEV).bfloat16(), (1 + 0.1 * torch.randn(D, generator=g, device=DEV)).bfloat16()
    out = torch.empty_like(x)
    check(_lib.lib().evo_rmsnorm(ptr(x), ptr(s), ptr(out), rows, D, 1e-6, _stream()), "evo_rmsnorm")
    d = x.double()
    want = d / (d.norm(dim=-1, keepdim=True) * D ** -0.5 + 1e-6) * s.double()
    # five roundings to bf16 (norm, times D^-1/2, plus eps, quotient, product), each at most half a step of 2^-7
    assert ((out.double() - want).abs() <= 5 * 2.0 ** -8 * want.abs()).all()


@pytest.mark.parametrize("ids_dtype", [torch.int32, torch.int64])
@pytest.mark.parametrize("rows,D", [(1, 256), (3, 4096), (16, 2304), (2, 8192), (300, 512)])
def test_embed_norm_is_embed_and_rmsnorm(rows, D, ids_dtype):
    """The beginning of a decode step in one launch: the bits of the two it stands for, ids out of range included, and the position."""
    g = torch.Generator(device=DEV).manual_seed(D + rows)
    table, scale = torch.randn(512, D, generator=g, device=DEV).bfloat16(), (1 + 0.1 * torch.randn(D, generator=g, device=DEV)).bfloat16()
    ids = torch.randint(-3, 520, (rows,), generator=g, device=DEV).to(ids_dtype)
    lib, new = _lib.lib(), lambda: torch.full((rows, D), 9.0, dtype=torch.bfloat16, device=DEV)  # noqa: E731
    u, xn, u2, xn2 = new(), new(), new(), new()
    wide, pos = int(ids_dtype == torch.int64), torch.tensor([-1, 77], device=DEV)
    check(lib.evo_embed(C.c_void_p(ids.data_ptr()), wide, C.c_void_p(table.data_ptr()), C.c_void_p(u.data_ptr()), rows, D, 512, _stream()), "evo_embed")
    check(lib.evo_rmsnorm(C.c_void_p(u.data_ptr()), C.c_void_p(scale.data_ptr()), C.c_void_p(xn.data_ptr()), rows, D, 1e-6, _stream()), "evo_rmsnorm")
    check(lib.evo_embed_norm(C.c_void_p(ids.data_ptr()), wide, C.c_void_p(table.data_ptr()), C.c_void_p(scale.data_ptr()), C.c_void_p(u2.data_ptr()), C.c_void_p(xn2.data_ptr()), rows, D, 512,
                             1e-6, C.c_void_p(pos.data_ptr()), 1234567, _stream()), "evo_embed_norm")
    assert torch.equal(u, u2) and pos.tolist() == [1234567, 77]
    if rows <= 64:                                   # (beyond, evo_rmsnorm may sum a row's squares in another order)
        assert torch.equal(xn, xn2)
    else:
        assert ((xn.float() - xn2.float()).abs() <= 2.0 ** -6 * xn.float().abs()).all()
    with pytest.raises(_lib.EvoError):
        check(lib.evo_embed_norm(C.c_void_p(ids.data_ptr()), wide, C.c_void_p(table.data_ptr()), C.c_void_p(scale.data_ptr()), C.c_void_p(u2.data_ptr()), C.c_void_p(xn2.data_ptr()), rows, 8448,
                                 512, 1e-6, None, 0, _stream()), "evo_embed_norm")
