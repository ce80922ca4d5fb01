"""Chains of small kernels that are resident at once, their buffers written again by the next turn: in a stream and in a captured graph they give the bits of calls that are waited for."""
import ctypes as C

import pytest
import torch

import evo_b200._lib as _lib
from evo_b200._lib import AttnParams, ConvActParams, GatedDeltaParams, HyenaParams, SumNormParams, WindowAttnParams, check, ptr
from evo_b200.engine import KernelOps

pytestmark = pytest.mark.gpu
DEV, BF = "cuda:0", torch.bfloat16


class _Ops(KernelOps):
    _prof, gemm_variant, gemm_variant_gate = None, 0, 0


def _stream():
    return C.c_void_p(torch.cuda.current_stream().cuda_stream)


def _runs(make, turns, level):
    """What `turns` turns of make() leave: waited for after every call, in a stream, and in a captured graph."""
    lib, out = _lib.lib(), []
    for form in ("waited", "stream", "graph"):
        calls, results = make()
        prev = lib.evo_set_pdl(level)
        try:
            if form == "graph":
                warm, _ = make()                                  # first launches outside of the capture
                for call in warm:
                    call()
                torch.cuda.synchronize()
                graph = torch.cuda.CUDAGraph()
                with torch.cuda.graph(graph):
                    for _ in range(4):
                        for call in calls:
                            call()
                for _ in range(turns // 4):
                    graph.replay()
            else:
                for _ in range(turns):
                    for call in calls:
                        call()
                        if form == "waited":
                            torch.cuda.synchronize()
            torch.cuda.synchronize()
        finally:
            lib.evo_set_pdl(prev)
        out.append([t.clone() for t in results])
    return out


# up to 64 rows and more (the norm's two launches); one tile and several per layer
@pytest.mark.parametrize("level", [-1, 0, 1, 2, 3, 4])
@pytest.mark.parametrize("rows,D", [(2, 256), (65, 256), (96, 512), (16, 1024)])
def test_steps_of_one_layer_in_order(rows, D, level):
    """evo_gemm, evo_hyena_step, evo_gemm, evo_rmsnorm over and over: a step's states are there when the next one fetches them, ahead of its wait or not."""
    def make():
        g = torch.Generator(device=DEV).manual_seed(rows + D)
        n = lambda *s: torch.randn(*s, generator=g, device=DEV)  # noqa: E731
        x, u, y, t = n(rows, D).to(BF), torch.zeros(rows, 3 * D, dtype=BF, device=DEV), torch.zeros(rows, D, dtype=BF, device=DEV), torch.zeros(rows, D, dtype=BF, device=DEV)
        w_in, w_out, scale = (n(3 * D, D) / D ** 0.5).to(BF), (n(D, D) / D ** 0.5).to(BF), (1 + 0.1 * n(D)).to(BF)
        fir, state = n(rows, 3 * D, 2).to(BF), n(rows, D, 8, 2)
        fw, fb, skip = (0.5 * n(3 * D, 1, 3)).to(BF), (0.1 * n(3 * D)).to(BF), (0.5 * n(D)).to(BF)
        poles, residues = (0.6 * n(D, 8, 1, 2)).clamp(-0.6, 0.6).contiguous(), 0.35 * n(D, 8, 1, 2)
        ops, lib = _Ops(), _lib.lib()
        calls = [lambda: ops._gemm(x, w_in, u, rows, 3 * D, D, _lib.EPI_NONE),
                 lambda: check(lib.evo_hyena_step(ptr(u), ptr(y), ptr(fir), ptr(state), ptr(fw), ptr(fb), ptr(skip), ptr(poles), ptr(residues), rows, D, 8, D // 128, _stream()), "evo_hyena_step"),
                 lambda: ops._gemm(y, w_out, t, rows, D, D, _lib.EPI_NONE),
                 lambda: check(lib.evo_rmsnorm(ptr(t), ptr(scale), ptr(x), rows, D, 1e-6, _stream()), "evo_rmsnorm")]
        keep = (w_in, w_out, scale, fw, fb, skip, poles, residues)
        calls[0].keep = keep
        return calls, [x, u, y, t, fir, state]

    waited, stream, graph = _runs(make, 200, level)
    assert all(torch.isfinite(t.float()).all() for t in waited)
    for a, b, c in zip(waited, stream, graph):
        assert torch.equal(a, b) and torch.equal(a, c)


def _prompt_chain(B, L, D):
    """One layer of everything: sums and norm, projection, convolution, delta rule, Hyena operator, both attentions, projection, norm; each buffer is written again by the next turn."""
    g = torch.Generator(device=DEV).manual_seed(B * L + D)
    n = lambda *s: torch.randn(*s, generator=g, device=DEV)  # noqa: E731
    R, H, lib, ops = B * L, D // 128, _lib.lib(), _Ops()
    new = lambda *s: torch.zeros(*s, dtype=BF, device=DEV)  # noqa: E731
    x, h, qkv, c, z = n(R, D), n(R, D).to(BF), new(R, 3 * D), new(R, 3 * D), new(R, D + 256)
    y = [new(R, D) for _ in range(4)]
    w_qkv, w_z, w_o = (n(3 * D, D) / D ** 0.5).to(BF), (n(D + 256, D) / D ** 0.5).to(BF), (n(D, D) / D ** 0.5).to(BF)
    scale, taps, carry, state = (1 + 0.1 * n(D)).to(BF), (0.5 * n(3 * D, 4)).to(BF), n(B, 3, 3 * D), 0.3 * n(B, H, 128, 128)
    A, dt, nw, sink = torch.log(1 + 15 * torch.rand(H, generator=g, device=DEV)).to(BF), torch.full((H,), -3.0, device=DEV).to(BF), (1 + 0.2 * n(128)).to(BF), n(H).to(BF)
    fw, fb, skip = (0.5 * n(3 * D, 1, 3)).to(BF), (0.1 * n(3 * D)).to(BF), (0.5 * n(D)).to(BF)
    poles, residues = (0.6 * n(D, 8, 1, 2)).clamp(-0.6, 0.6).contiguous(), 0.35 * n(D, 8, 1, 2)
    hs, fs = torch.zeros(B, D, 8, 2, device=DEV), new(B, 3 * D, 2)

    sums = SumNormParams(x=x.data_ptr(), n_branches=3, eps=1e-6, dtype=0, rows=R, D=D, ldo=D)
    for i in range(3):
        sums.y[i], sums.ldy[i], sums.scale[i] = y[i].data_ptr(), D, 0.1
    sums.out[0], sums.w[0] = h.data_ptr(), scale.data_ptr()
    conv = ConvActParams(inp=qkv.data_ptr(), ld=3 * D, weight=taps.data_ptr(), carry=carry.data_ptr(), zero_start=0, out=c.data_ptr(), ldo=3 * D, B=B, L=L, C=3 * D, taps=4, act=1, dtype=0)
    delta = GatedDeltaParams(q=c.data_ptr(), k=c.data_ptr() + 2 * D, v=c.data_ptr() + 4 * D, ld=3 * D, b=z.data_ptr() + 2 * D, a=z.data_ptr() + 2 * (D + H), gate=z.data_ptr(), ldz=D + 256,
                             A_log=A.data_ptr(), dt_bias=dt.data_ptr(), norm_w=nw.data_ptr(), eps=1e-6, unit_eps=1e-6, q_scale=128 ** -0.5, state=state.data_ptr(), zero_start=0,
                             out=y[0].data_ptr(), ldo=D, dtype=0, B=B, L=L, H=H, G=H, dk=128, dv=128)
    hyena = HyenaParams(z=qkv.data_ptr(), y=y[1].data_ptr(), fir_w=fw.data_ptr(), fir_b=fb.data_ptr(), Dskip=skip.data_ptr(), poles=poles.data_ptr(), residues=residues.data_ptr(),
                        B=B, L=L, D=D, S=8, nheads=H, state_out=hs.data_ptr(), fir_state_out=fs.data_ptr())
    attn = AttnParams(q=qkv.data_ptr(), k=qkv.data_ptr() + 2 * D, v=qkv.data_ptr() + 4 * D, out=y[2].data_ptr(), q_tok_stride=3 * D, kv_tok_stride=3 * D, q_batch_stride=L * 3 * D,
                      kv_batch_stride=L * 3 * D, B=B, Lq=L, Lk=L, H=H, hd=128, q_pos0=0, softmax_scale=128 ** -0.5)
    win = WindowAttnParams(q=c.data_ptr(), q_tok_stride=3 * D, k=c.data_ptr() + 2 * D, v=c.data_ptr() + 4 * D, k_tok_stride=3 * D, v_tok_stride=3 * D, k_batch_stride=L * 3 * D,
                           v_batch_stride=L * 3 * D, gate=z.data_ptr(), gate_tok_stride=D + 256, out=y[3].data_ptr(), ldo=D, dtype=0, B=B, Lq=L, H=H, G=H, dk=128, dv=128, n_maps=1,
                           q_pos0=0, window=100, keep_first=0, scale=128 ** -0.5, sink=sink.data_ptr())
    nd, nh, na = lib.evo_gated_delta_workspace(C.byref(delta)), lib.evo_hyena_fwd_workspace(C.byref(hyena)), lib.evo_attn_fwd_workspace(C.byref(attn), 2)
    wd, wh, wa = (torch.zeros(max(k, 1), dtype=torch.uint8, device=DEV) for k in (nd, nh, na))
    calls = [lambda: check(lib.evo_sum_norm(C.byref(sums), _stream()), "evo_sum_norm"),
             lambda: ops._gemm(h, w_qkv, qkv, R, 3 * D, D, _lib.EPI_NONE),
             lambda: ops._gemm(h, w_z, z, R, D + 256, D, _lib.EPI_NONE),
             lambda: check(lib.evo_conv_act(C.byref(conv), _stream()), "evo_conv_act"),
             lambda: check(lib.evo_gated_delta_fwd(C.byref(delta), ptr(wd), nd, _stream()), "evo_gated_delta_fwd"),
             lambda: check(lib.evo_hyena_fwd(C.byref(hyena), ptr(wh), nh, _stream()), "evo_hyena_fwd"),
             lambda: check(lib.evo_window_attn_fwd(C.byref(win), _stream()), "evo_window_attn_fwd"),
             lambda: check(lib.evo_attn_fwd_ws(C.byref(attn), 2, ptr(wa), na, _stream()), "evo_attn_fwd_ws"),
             lambda: ops._gemm(y[3], w_o, h, R, D, D, _lib.EPI_NONE),
             lambda: check(lib.evo_rmsnorm(ptr(h), ptr(scale), ptr(y[2]), R, D, 1e-6, _stream()), "evo_rmsnorm")]
    calls[0].keep = (w_qkv, w_z, w_o, scale, taps, A, dt, nw, sink, fw, fb, skip, poles, residues, wd, wh, wa)
    return calls, [x, h, qkv, c, z, *y, carry, state, hs, fs]


@pytest.mark.parametrize("level", [-1, 0, 1, 4])
@pytest.mark.parametrize("B,L,D", [(1, 70, 256), (2, 63, 512), (3, 301, 512), (1, 777, 1024)])
def test_prompt_kernels_in_order(B, L, D, level):
    waited, stream, graph = _runs(lambda: _prompt_chain(B, L, D), 40, level)
    assert all(torch.isfinite(t.float()).all() for t in waited)
    for a, b, c in zip(waited, stream, graph):
        assert torch.equal(a, b) and torch.equal(a, c)


def _programmatic_edges(calls):
    """Edges of the captured calls over which a kernel may start before the one in front of it has ended."""
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        for call in calls:
            call()
    get, count, handle = C.CDLL("libcuda.so.1").cuGraphGetEdges_v2, C.c_size_t(0), C.c_void_p(graph.raw_cuda_graph())
    assert get(handle, None, None, None, C.byref(count)) == 0
    n = count.value
    nodes, data = (C.c_void_p * n)(), (C.c_uint8 * 8 * n)()               # from_port, to_port, type, reserved
    assert get(handle, nodes, (C.c_void_p * n)(), data, C.byref(count)) == 0
    return sum(d[2] == 1 for d in data), n


def test_level_zero_launches_nothing_dependent():
    """0 is off: each launch of a prompt's and of a step's kernels waits for the one in front.  The library starts with the prompt's kernels dependent."""
    lib = _lib.lib()
    calls, _ = _prompt_chain(2, 203, 512)
    for call in calls:
        call()
    torch.cuda.synchronize()
    start = lib.evo_set_pdl(0)
    try:
        assert start == -1
        off, edges = _programmatic_edges(calls)
        assert off == 0 and edges >= len(calls) - 1
        for level in (-1, 4):
            lib.evo_set_pdl(level)
            on, _ = _programmatic_edges(calls)
            assert on >= len(calls) - 1, (level, on)
    finally:
        lib.evo_set_pdl(start)
