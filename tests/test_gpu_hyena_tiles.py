"""The tensor-core form of the Hyena operator at the edges of its blocks (16 tokens), rows (16 R), stages (128) and tiles (256 R), and with values
that its products must not carry backwards."""
import math
import os
import sys

import pytest
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)
sys.path.insert(0, os.path.join(ROOT, "tests", "harness"))

from oracle import stripedhyena_oracle as O  # noqa: E402
import gpu_bringup as G  # noqa: E402

G._imports()

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
D, H = 256, 2


def _filter(seed=5):
    sd = O.random_state_dict(O.tiny_config(num_layers=1, attn_layer_idxs=(), hidden_size=D, num_heads=H), seed=seed)
    p = "blocks.0.filter."
    return {k: sd[p + n].to(DEV) for k, n in (("w", "short_filter_weight"), ("b", "short_filter_bias"), ("D", "D"), ("p", "poles"), ("r", "residues"))}


def _oracle(z, f, halo, state_in):
    """The reference's rounding points (bf16 tensor operations), the convolution and the state in 64 bits."""
    c = {k: v.cpu() for k, v in f.items()}
    B, L, C3 = z.shape
    zp = torch.cat([halo if halo is not None else torch.zeros(B, 2, C3, dtype=z.dtype), z], 1).float()
    w = c["w"].float()[:, 0]
    f1 = (zp[:, :L] * w[:, 0]).double() + zp[:, 1:L + 1].double() * w[:, 1].double()
    zf = (f1.float().double() + zp[:, 2:].double() * w[:, 2].double()).float().bfloat16() + c["b"]          # two fused multiply-adds
    x2, x1, v = (zf.view(B, L, H, 3, 128)[:, :, :, i].reshape(B, L, D) for i in range(3))
    x = x1 * v
    p, r = torch.view_as_complex(c["p"].double())[..., 0], torch.view_as_complex(c["r"].double())[..., 0]
    S = torch.view_as_complex(state_in.double()) if state_in is not None else torch.zeros(B, D, 8, dtype=torch.complex128)
    conv = torch.empty(B, L, D, dtype=torch.float64)
    for t in range(L):
        S = p[None] * S + x[:, t, :, None].double()
        conv[:, t] = (r[None] * S).sum(-1).real
    return (conv.float().bfloat16() + x * c["D"]) * x2, torch.view_as_real(S)


@pytest.mark.parametrize("B,L,R,nseg,carried", [
    (2, 1, 1, 1, True), (1, 15, 1, 1, False), (1, 16, 2, 1, True), (2, 17, 4, 1, True), (1, 64, 4, 1, False), (1, 65, 4, 1, True), (1, 128, 1, 1, False),
    (1, 129, 2, 1, True), (1, 255, 1, 1, False), (2, 256, 1, 1, True), (1, 257, 1, 1, True), (1, 272, 1, 1, False), (1, 273, 1, 1, False), (1, 512, 2, 1, True), (1, 530, 2, 3, True),
    (3, 700, 1, 2, True), (1, 1024, 4, 1, True), (1, 1040, 4, 1, False), (2, 1100, 4, 4, True), (1, 3, 4, 3, True)])
def test_blocks_rows_tiles_and_segments(monkeypatch, B, L, R, nseg, carried):
    monkeypatch.setenv("EVO_B200_HYENA_VARIANT", "2")
    monkeypatch.setenv("EVO_B200_HYENA_R", str(R))
    f = _filter()
    g = torch.Generator().manual_seed(L)
    z = torch.randn(B, L, 3 * D, generator=g).bfloat16()
    halo = torch.randn(B, 2, 3 * D, generator=g).bfloat16() if carried else None
    s0 = torch.randn(B, D, 8, 2, generator=g) if carried else None
    want, state = _oracle(z, f, halo, s0)
    on = lambda t: t.to(DEV) if t is not None else None  # noqa: E731
    y, st, fs = G._hyena_call(on(z), f, B, L, D, H, force=nseg, halo=on(halo), state_in=on(s0))
    # fp32 sums before the rounding to bf16: an element differs only where the exact sum lies within about 2^-20 of a rounding edge, 2^-9 apart
    assert (y.cpu() != want).float().mean() < 1e-3
    assert (y.cpu().double() - want.double()).norm() <= 2e-4 * want.double().norm()
    assert (st.cpu().double() - state).norm() <= 1e-6 * state.norm()           # fp32 throughout; segments fold with p^length from 64 bits
    _, only, _ = G._hyena_call(on(z), f, B, L, D, H, force=nseg, halo=on(halo), state_in=on(s0), state_only=True)
    assert (only.cpu().double() - state).norm() <= 5e-6 * state.norm()         # (the fold of a carry pass takes its powers in fp32)


@pytest.mark.parametrize("where,value", [(37, math.inf), (300, math.nan), (511, -math.inf), (128, 3e38)])
def test_values_that_are_not_finite_stay_behind_their_token(monkeypatch, where, value):
    monkeypatch.setenv("EVO_B200_HYENA_VARIANT", "2")
    monkeypatch.setenv("EVO_B200_HYENA_R", "2")
    f = _filter()
    L = 700
    z = torch.randn(1, L, 3 * D, generator=torch.Generator().manual_seed(1)).bfloat16().to(DEV)
    clean, _, _ = G._hyena_call(z, f, 1, L, D, H)
    bad = z.clone()
    ch = 41
    bad[0, where, 256 + ch] = value                         # v of channel 41
    bad[0, where, 128 + ch] = value if abs(value) == 3e38 else 1.0
    y, _, _ = G._hyena_call(bad, f, 1, L, D, H)
    monkeypatch.setenv("EVO_B200_HYENA_VARIANT", "1")
    scan, _, _ = G._hyena_call(bad, f, 1, L, D, H)
    assert (y[0, :where] == clean[0, :where]).float().mean() > 0.999
    assert torch.isfinite(y[0, :where].float()).all()
    rest = [c for c in range(D) if c != ch]
    assert torch.equal(y[..., rest], clean[..., rest])
    assert torch.equal(torch.isfinite(y.float()), torch.isfinite(scan.float()))


@pytest.mark.parametrize("B,L", [(1, 60), (1, 200), (2, 520), (1, 1500)])
def test_the_rule_picks_a_path_that_agrees_with_the_scan(monkeypatch, B, L):
    monkeypatch.delenv("EVO_B200_HYENA_VARIANT", raising=False)
    monkeypatch.delenv("EVO_B200_HYENA_R", raising=False)
    f = _filter()
    z = torch.randn(B, L, 3 * D, generator=torch.Generator().manual_seed(2)).bfloat16().to(DEV)
    y, st, fs = G._hyena_call(z, f, B, L, D, H)
    monkeypatch.setenv("EVO_B200_HYENA_VARIANT", "1")
    y1, st1, fs1 = G._hyena_call(z, f, B, L, D, H)
    assert (y != y1).float().mean() < 1e-3 and torch.equal(fs, fs1)
    assert (st - st1).norm() <= 2e-6 * st1.norm()
