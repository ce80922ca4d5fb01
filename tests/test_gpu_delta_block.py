"""The gated delta rule by blocks of 64 tokens (tensor cores) at the edges of its blocks, tiles and channel groups, with decays and inputs that random weights do not give."""
import ctypes as C
import math
import os
import sys

import pytest
import torch

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
from evo_b200 import _lib  # noqa: E402
from evo_b200._lib import GatedDeltaParams, check, ptr  # noqa: E402

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _inputs(B, L, H, G, dk, dv, seed=0, alike=False):
    g = torch.Generator(device=DEV).manual_seed(seed)
    n = lambda *s: torch.randn(*s, generator=g, device=DEV)  # noqa: E731
    pad = 8
    x = torch.nn.functional.silu(n(B * L, 2 * G * dk + H * dv + pad))
    if alike:                                     # keys that hardly differ: the block's triangular system is as far from the identity as it gets
        x[:, G * dk:2 * G * dk] = n(1, G * dk) + 0.05 * n(B * L, G * dk)
    z = n(B * L, H * dv + 2 * H)
    a_log, dt = torch.log(1 + 15 * torch.rand(H, generator=g, device=DEV)), torch.full((H,), -3.0, device=DEV)
    return dict(x=x.bfloat16(), z=z.bfloat16(), A=a_log.bfloat16(), dt=dt.bfloat16(), w=(1 + 0.2 * n(dv)).bfloat16(), S=0.3 * n(B, H, dk, dv))


def _run(t, B, L, H, G, dk, dv, zero=0, state=True, ldo=None):
    x, z = t["x"], t["z"]
    ldo = ldo or H * dv
    out = torch.full((B * L, ldo), 7.0, dtype=x.dtype, device=DEV)
    S = t["S"].clone()
    e = x.element_size()
    p = GatedDeltaParams(q=x.data_ptr(), k=x.data_ptr() + G * dk * e, v=x.data_ptr() + 2 * G * dk * e, ld=x.shape[1], b=z.data_ptr() + H * dv * e, a=z.data_ptr() + (H * dv + H) * e,
                         gate=z.data_ptr(), ldz=z.shape[1], A_log=t["A"].data_ptr(), dt_bias=t["dt"].data_ptr(), norm_w=t["w"].data_ptr(), eps=1e-6, unit_eps=1e-6, q_scale=dk ** -0.5,
                         state=S.data_ptr() if state else None, zero_start=zero, out=out.data_ptr(), ldo=ldo, dtype=0 if e == 2 else 1, B=B, L=L, H=H, G=G, dk=dk, dv=dv)
    nb = _lib.lib().evo_gated_delta_workspace(C.byref(p))
    ws = torch.empty(max(nb, 1), dtype=torch.uint8, device=DEV)
    check(_lib.lib().evo_gated_delta_fwd(C.byref(p), ptr(ws) if nb else None, nb, C.c_void_p(torch.cuda.current_stream().cuda_stream)), "evo_gated_delta_fwd")
    torch.cuda.synchronize()
    return out, S, nb


def _oracle(t, B, L, H, G, dk, dv, zero):
    x, z = t["x"].double(), t["z"].double()
    q, k = (x[:, i * G * dk:(i + 1) * G * dk].view(B, L, G, dk).repeat_interleave(H // G, 2) for i in (0, 1))
    v = x[:, 2 * G * dk:2 * G * dk + H * dv].view(B, L, H, dv)
    gate, b, a = z[:, :H * dv].view(B, L, H, dv), z[:, H * dv:H * dv + H].view(B, L, H), z[:, H * dv + H:].view(B, L, H)
    k = k / torch.sqrt((k * k).sum(-1, keepdim=True) + 1e-6)
    q = q / torch.sqrt((q * q).sum(-1, keepdim=True) + 1e-6) * dk ** -0.5
    g = torch.exp(-torch.exp(t["A"].double()) * torch.nn.functional.softplus(a + t["dt"].double()))
    beta = torch.sigmoid(b)
    S = torch.zeros_like(t["S"], dtype=torch.float64) if zero else t["S"].double()
    o = torch.empty(B, L, H, dv, dtype=torch.float64, device=DEV)
    for i in range(L):
        S = S * g[:, i, :, None, None]
        u = beta[:, i, :, None] * (v[:, i] - torch.einsum("bhk,bhkv->bhv", k[:, i], S))
        S = S + k[:, i, :, :, None] * u[:, :, None, :]
        o[:, i] = torch.einsum("bhk,bhkv->bhv", q[:, i], S)
    o = o / torch.sqrt((o * o).mean(-1, keepdim=True) + 1e-6) * t["w"].double() * torch.nn.functional.silu(gate)
    return o.reshape(B * L, H * dv), S


@pytest.mark.parametrize("B,L,H,G,dk,dv,zero,alike", [
    (1, 32, 1, 1, 128, 16, 0, False), (2, 63, 2, 1, 64, 32, 0, True), (1, 64, 3, 3, 128, 128, 1, False), (2, 65, 4, 2, 128, 64, 0, True), (1, 127, 2, 2, 64, 128, 0, False),
    (1, 129, 2, 2, 128, 48, 0, True), (3, 200, 2, 1, 64, 64, 1, False), (1, 321, 40, 40, 128, 128, 0, False), (5, 70, 32, 32, 64, 128, 0, False)])
def test_blocks_against_the_recurrence_in_64_bits(B, L, H, G, dk, dv, zero, alike):
    t = _inputs(B, L, H, G, dk, dv, seed=L, alike=alike)
    out, S, nb = _run(t, B, L, H, G, dk, dv, zero, ldo=H * dv + 24)
    assert nb > 4 * B * L * H * dv                                              # the block form was taken
    want, state = _oracle(t, B, L, H, G, dk, dv, zero)
    got = out[:, :H * dv].double()
    assert (got - want).norm() <= 2.2e-3 * want.norm()                          # one rounding to bf16: 2^-9 / sqrt(3) of an element, on average
    assert (S.double() - state).norm() <= (4e-6 if alike else 1e-6) * state.norm()      # fp32 throughout
    assert not out[:, H * dv:].any()
    none, _, _ = _run(t, B, L, H, G, dk, dv, 1, state=False)                    # no state given: from zero, none kept
    assert torch.equal(none, _run(t, B, L, H, G, dk, dv, 1)[0])


def test_agrees_with_the_token_by_token_kernel_in_fp32():
    B, L, H, dk, dv = 1, 150, 2, 128, 128
    t = _inputs(B, L, H, H, dk, dv, seed=4)
    out, S, _ = _run(t, B, L, H, H, dk, dv)
    f = dict(t, x=t["x"].float(), z=t["z"].float())
    out32, S32, _ = _run(f, B, L, H, H, dk, dv)
    assert (S - S32).norm() <= 1e-6 * S32.norm()
    assert (out.float() - out32).norm() <= 2.2e-3 * out32.norm()


@pytest.mark.parametrize("what", ["v", "k", "q", "a", "b"])
@pytest.mark.parametrize("value", [math.nan, math.inf])
def test_what_is_not_finite_stays_behind_its_token(what, value):
    B, L, H, dk, dv, at = 1, 200, 2, 128, 64, 75
    t = _inputs(B, L, H, H, dk, dv, seed=9)
    clean, _, _ = _run(t, B, L, H, H, dk, dv)
    bad = {k: v.clone() for k, v in t.items()}
    if what in "qkv":
        bad["x"][at, {"q": 0, "k": H * dk, "v": 2 * H * dk}[what] + 3] = value
    else:
        bad["z"][at, H * dv + (H if what == "a" else 0)] = value
    out, _, _ = _run(bad, B, L, H, H, dk, dv)
    assert (out[:at].float() - clean[:at].float()).norm() <= 1e-4 * clean[:at].float().norm()
    assert torch.equal(out[:, dv:], clean[:, dv:])                              # the other head
    f = dict(bad, x=bad["x"].float(), z=bad["z"].float())
    step = _run(f, B, L, H, H, dk, dv)[0]
    assert torch.equal(torch.isfinite(out.float()), torch.isfinite(step))


def test_decays_that_reach_zero_and_come_back():
    """A token whose decay underflows forgets everything before it; the tokens behind it still see each other exactly."""
    B, L, H, dk, dv = 1, 128, 1, 128, 64
    t = _inputs(B, L, H, H, dk, dv, seed=2)
    t["z"][20, H * dv + H] = 300.0
    t["z"][90, H * dv + H] = 3e38
    out, S, _ = _run(t, B, L, H, H, dk, dv)
    want, state = _oracle(t, B, L, H, H, dk, dv, 0)
    assert (out.double() - want).norm() <= 2.2e-3 * want.norm() and (S.double() - state).norm() <= 1e-6 * state.norm()


@pytest.mark.parametrize("B,H,L", [(64, 32, 589), (300, 32, 130)])
def test_slabs_hand_the_state_on(B, H, L):
    """A call whose blocks' matrices pass 256 MB runs slab after slab: 4 + 4 + 2 blocks (the last one ragged), and one block at a time where a single one of every
    (head, sequence) pair is more than that.  Bit for bit the sequences one by one (a single slab each), with a state carried, from zero, and with none given."""
    G, dk, dv = 2, 64, 16
    t = _inputs(B, L, H, G, dk, dv, seed=B)
    one = lambda b: {k: (v[b * L:(b + 1) * L] if k in "xz" else v[b:b + 1] if k == "S" else v) for k, v in t.items()}  # noqa: E731
    out, S, nb = _run(t, B, L, H, G, dk, dv)
    block = 32768 * B * H                                                       # T, P and vectors of one block of every pair
    assert nb - 4 * B * L * H * dv < max(256 << 20, block) + 1024 < (L + 63) // 64 * block
    zero, S0, _ = _run(t, B, L, H, G, dk, dv, 1)
    none, _, nb_none = _run(t, B, L, H, G, dk, dv, 1, state=False)
    assert torch.equal(none, zero) and nb_none >= nb + 4 * B * H * dk * dv      # the state between the slabs is the workspace's
    for b in (0, B // 2, B - 1):
        o, s, _ = _run(one(b), 1, L, H, G, dk, dv)
        assert torch.equal(out[b * L:(b + 1) * L], o) and torch.equal(S[b], s[0])
        o, s, _ = _run(one(b), 1, L, H, G, dk, dv, 1)
        assert torch.equal(zero[b * L:(b + 1) * L], o) and torch.equal(S0[b], s[0])
    b = B // 3
    want, state = _oracle(one(b), 1, L, H, G, dk, dv, 0)
    assert (out[b * L:(b + 1) * L].double() - want).norm() <= 2.2e-3 * want.norm()
    assert (S[b].double() - state[0]).norm() <= 1e-6 * state.norm()
