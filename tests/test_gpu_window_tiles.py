"""The tcgen05 form of the windowed attention (one map, heads of 64 or 128, position known to the host) against a float64 oracle over the same bf16 inputs:
the edges of its 128-query and 128-key tiles, windows around a tile, carried positions, shared key heads, row strides, gates and sinks, and values that are not finite.

Tolerance: a probability enters the products with relative error 2^-17 (bf16 high and low part), its exponential with 2^-21, the sums of at most 2^10 keys in fp32 with
2^-14 of the sum of magnitudes, and the result is rounded to bf16 (2^-9 of itself; 2^-8 leaves room for the fast exponential of the gate).  Magnitudes are at most the
row's largest value, so |out - oracle| <= 2^-8 |oracle| + 2^-12 max|v|.
"""
import ctypes as C
import math

import pytest
import torch

pytestmark = pytest.mark.gpu

BF = torch.bfloat16


def _oracle(q, k, v, pos, window, scale, sink, gate, per_head):
    B, L, H, d = q.shape
    G = k.shape[2]
    out = torch.empty(B, L, H, d, dtype=torch.float64, device=q.device)
    i = torch.arange(L, device=q.device)[:, None] + pos
    j = torch.arange(pos + L, device=q.device)[None]
    seen = (j <= i) & ((i - j < window) if window > 0 else True)
    for b in range(B):
        for h in range(H):
            kk, vv = k[b, :pos + L, h * G // H].double(), v[b, :pos + L, h * G // H].double()
            s = (q[b, :, h].double() @ kk.T * scale).masked_fill(~seen, -math.inf)
            if sink is not None:
                s = torch.cat([s, sink[h].double().expand(L, 1)], 1)
            p = torch.softmax(s, 1)[:, :pos + L]
            fin = torch.isfinite(vv)
            o = p @ torch.where(fin, vv, 0.0)
            for c in torch.nonzero(~fin.all(0)).flatten().tolist():                # a value that is not finite reaches the rows that see it, no other
                for t in torch.nonzero(~fin[:, c]).flatten().tolist():
                    o[:, c] += torch.where(seen[:, t], p[:, t] * vv[t, c], 0.0)
            if gate is not None:
                o = o * torch.sigmoid(gate[b, :, h].double()).reshape(L, -1)
            out[b, :, h] = o
    return out


def _run(B, L, H, G, d, pos, window, *, gate=None, sink=False, pad=0, seed=0, spoil=(), cap=0, on_device=False):
    from evo_b200 import _lib
    from evo_b200._lib import WindowAttnParams, check
    lib = _lib.lib()
    g = torch.Generator(device="cuda").manual_seed(seed)
    rn = lambda *s: torch.randn(*s, generator=g, device="cuda").to(BF)
    q = rn(B * L, H * d + pad)
    kv = rn(B, pos + L + cap, 2 * G * d + pad)
    for b, t, c, x in spoil:
        kv[b, t, G * d + c] = x
    gt = rn(B * L, H * d + pad) if gate == "channel" else rn(B * L, H) if gate == "head" else None
    sk = rn(H) if sink else None
    out = torch.full((B * L, H * d + pad), 7.0, dtype=BF, device="cuda")
    p = WindowAttnParams(q=q.data_ptr(), q_tok_stride=q.shape[1], k=kv.data_ptr(), v=kv.data_ptr() + 2 * G * d, k_tok_stride=kv.shape[2], v_tok_stride=kv.shape[2],
                         k_batch_stride=kv.stride(0), v_batch_stride=kv.stride(0), out=out.data_ptr(), ldo=out.shape[1], dtype=0, B=B, Lq=L, H=H, G=G, dk=d, dv=d, n_maps=1,
                         q_pos0=pos, window=window, keep_first=0, scale=d ** -0.5)
    if gt is not None:
        p.gate, p.gate_tok_stride, p.gate_per_head = gt.data_ptr(), gt.shape[1], int(gate == "head")
    if sk is not None:
        p.sink = sk.data_ptr()
    at = torch.tensor([pos], dtype=torch.int64, device="cuda")
    if on_device:
        p.pos_dev = at.data_ptr()
    check(lib.evo_window_attn_fwd(C.byref(p), torch.cuda.current_stream().cuda_stream), "evo_window_attn_fwd")
    kk, vv = kv[:, :, :G * d].reshape(B, -1, G, d), kv[:, :, G * d:2 * G * d].reshape(B, -1, G, d)
    gg = None if gt is None else gt[:, :H * d].reshape(B, L, H, d) if gate == "channel" else gt.reshape(B, L, H, 1)
    ref = _oracle(q[:, :H * d].reshape(B, L, H, d), kk, vv, pos, window, d ** -0.5, sk, gg, gate == "head")
    if pad:
        assert (out[:, H * d:] == 0).all()
    return out[:, :H * d].reshape(B, L, H, d).double(), ref, vv[torch.isfinite(vv)].abs().max().item()


def _close(out, ref, vmax):
    bad = ~((out - ref).abs() <= 2.0 ** -8 * ref.abs() + 2.0 ** -12 * vmax)
    assert not bad.any(), (int(bad.sum()), (out - ref).abs().max().item())


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("L", [16, 127, 128, 129, 256, 257, 400])
@pytest.mark.parametrize("window", [0, 1, 100, 128, 129, 300])
def test_edges_of_the_tiles(d, L, window):
    _close(*_run(1, L, 2, 1, d, 0, window, gate="channel", sink=True, seed=L + window))


@pytest.mark.parametrize("B,L,H,G,d,pos,window,gate,sink,pad,cap", [
    (2, 200, 4, 2, 128, 0, 64, "head", False, 0, 0),
    (2, 300, 4, 4, 64, 5, 0, None, True, 8, 0),
    (3, 130, 2, 2, 128, 777, 256, "channel", True, 24, 50),
    (1, 1111, 2, 1, 128, 513, 1024, None, False, 0, 3),
    (2, 640, 8, 2, 64, 1, 127, "channel", False, 0, 0),
    (40, 150, 16, 4, 128, 0, 0, "channel", True, 0, 0),        # the last heads taken together
])
def test_options(B, L, H, G, d, pos, window, gate, sink, pad, cap):
    _close(*_run(B, L, H, G, d, pos, window, gate=gate, sink=sink, pad=pad, cap=cap, seed=1))


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("window", [0, 100])
def test_values_that_are_not_finite_reach_only_the_rows_that_see_them(d, window):
    out, ref, vmax = _run(1, 300, 1, 1, d, 0, window, sink=True, gate="channel", spoil=[(0, 200, 3, math.inf), (0, 140, 7, math.nan), (0, 250, d - 1, -math.inf)])
    assert torch.equal(torch.isnan(out), torch.isnan(ref))
    assert torch.equal(torch.isposinf(out), torch.isposinf(ref)) and torch.equal(torch.isneginf(out), torch.isneginf(ref))
    fin = torch.isfinite(ref)
    assert fin[0, :140].all() and not fin.all()
    _close(out[fin], ref[fin], vmax)


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("L", [1, 2, 4, 5, 9, 15])
@pytest.mark.parametrize("pos,window", [(0, 100), (37, 100), (900, 0), (1000, 256)])
def test_a_few_queries_run_as_in_a_captured_step(d, L, pos, window):
    """Up to 15 queries belong to the CUDA-core kernels wherever the position is known: a step called directly gives the bits of its captured twin, whose position
    is in device memory, with fp32 weights and the exact gate."""
    opt = dict(gate="channel", sink=True, seed=L, cap=4)
    out, ref, vmax = _run(2, L, 4, 2, d, pos, window, **opt)
    twin, _, _ = _run(2, L, 4, 2, d, pos, window, on_device=True, **opt)
    assert torch.equal(out, twin)
    _close(out, ref, vmax)


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("L,pos,window", [(16, 0, 0), (200, 5, 0), (300, 77, 100)])
def test_rows_that_do_not_start_on_16_bytes(d, L, pos, window):
    """What the tensor maps cannot read goes to the mma.sync form, whose heads of 64 and 128 nothing else reaches."""
    _close(*_run(2, L, 4, 2, d, pos, window, gate="channel", sink=True, pad=4, seed=L))
