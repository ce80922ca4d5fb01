"""Waits with a limit inside the tensor-core kernels: one that runs out (a limit of no tries at all) ends the kernel, keeps the caller's state and is reported."""
import ctypes as C
import os
import sys

import pytest
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)
sys.path.insert(0, os.path.join(ROOT, "tests"))
from evo_b200 import _lib  # noqa: E402
from evo_b200._lib import EvoError, HyenaParams, WindowAttnParams, check, check_lost_waits, ptr  # noqa: E402
import test_gpu_delta_block as D  # noqa: E402

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
BF = torch.bfloat16


class _no_tries:
    def __enter__(self):
        assert _lib.lib().evo_lost_waits(1) == 0                     # nothing was lost before
        self.before = _lib.lib().evo_set_wait_polls(0)

    def __exit__(self, *exc):
        _lib.lib().evo_set_wait_polls(self.before)


def _reported():
    torch.cuda.synchronize()
    assert _lib.lib().evo_lost_waits(0) == 1
    with pytest.raises(EvoError, match="ran out"):
        check_lost_waits()
    check_lost_waits()                                               # reported once


@pytest.mark.parametrize("B,H,dv,L", [(2, 2, 64, 64), (2, 2, 64, 200), (2, 2, 80, 200), (2, 2, 128, 64), (2, 2, 128, 200), (2, 2, 192, 200), (76, 2, 32, 64)])
def test_gated_delta(B, H, dv, L):
    """A CTA for a head, two that are a cluster, several that leave read-outs to a norm, and the kernel for calls of one block."""
    dk = 128
    t = D._inputs(B, L, H, H, dk, dv)
    out, S, _ = D._run(t, B, L, H, H, dk, dv)
    with _no_tries():
        _, kept, _ = D._run(t, B, L, H, H, dk, dv)
    _reported()
    assert torch.equal(kept, t["S"])
    again, S2, _ = D._run(t, B, L, H, H, dk, dv)
    assert torch.equal(again, out) and torch.equal(S2, S) and _lib.lib().evo_lost_waits(0) == 0


@pytest.mark.parametrize("L,segments,state_only", [(100, 1, 0), (1500, 1, 0), (1500, 2, 0), (1500, 2, 1)])
def test_hyena(monkeypatch, L, segments, state_only):
    monkeypatch.setenv("EVO_B200_HYENA_VARIANT", "2")
    B, dim = 2, 256
    g = torch.Generator(device=DEV).manual_seed(L)
    n = lambda *s: torch.randn(*s, generator=g, device=DEV)  # noqa: E731
    z, fw, fb, sk = n(B, L, 3 * dim).to(BF), n(3 * dim, 1, 3).to(BF), n(3 * dim).to(BF), n(dim).to(BF)
    poles, res = (0.6 * n(dim, 8, 1, 2)).clamp(-0.6, 0.6).contiguous(), n(dim, 8, 1, 2)

    def run():
        y, state = torch.full((B, L, dim), 7.0, dtype=BF, device=DEV), torch.full((B, dim, 8, 2), 7.0, device=DEV)
        p = HyenaParams(z=z.data_ptr(), y=y.data_ptr(), fir_w=fw.data_ptr(), fir_b=fb.data_ptr(), Dskip=sk.data_ptr(), poles=poles.data_ptr(), residues=res.data_ptr(), B=B, L=L,
                        D=dim, S=8, nheads=dim // 128, state_out=state.data_ptr(), force_segments=segments, state_only=state_only)
        nb = _lib.lib().evo_hyena_fwd_workspace(C.byref(p))
        ws = torch.zeros(max(nb, 1), dtype=torch.uint8, device=DEV)
        check(_lib.lib().evo_hyena_fwd(C.byref(p), ptr(ws), nb, C.c_void_p(torch.cuda.current_stream().cuda_stream)), "evo_hyena_fwd")
        torch.cuda.synchronize()
        return y, state

    y, state = run()
    with _no_tries():
        _, kept = run()
    _reported()
    if not state_only:
        assert (kept == 7.0).all()
    y2, state2 = run()
    assert torch.equal(y2, y) and torch.equal(state2, state) and _lib.lib().evo_lost_waits(0) == 0


@pytest.mark.parametrize("d,L,window", [(64, 100, 0), (128, 700, 200)])
def test_window_attention(d, L, window):
    H, G = 4, 2
    g = torch.Generator(device=DEV).manual_seed(L)
    q, kv = torch.randn(L, H * d, generator=g, device=DEV).to(BF), torch.randn(L, 2 * G * d, generator=g, device=DEV).to(BF)

    def run():
        out = torch.full((L, H * d), 7.0, dtype=BF, device=DEV)
        p = WindowAttnParams(q=q.data_ptr(), q_tok_stride=H * d, k=kv.data_ptr(), v=kv.data_ptr() + 2 * G * d, k_tok_stride=2 * G * d, v_tok_stride=2 * G * d, k_batch_stride=L * 2 * G * d,
                             v_batch_stride=L * 2 * G * d, out=out.data_ptr(), ldo=H * d, dtype=0, B=1, Lq=L, H=H, G=G, dk=d, dv=d, n_maps=1, window=window, scale=d ** -0.5)
        check(_lib.lib().evo_window_attn_fwd(C.byref(p), torch.cuda.current_stream().cuda_stream), "evo_window_attn_fwd")
        torch.cuda.synchronize()
        return out

    out = run()
    with _no_tries():
        run()
    _reported()
    assert torch.equal(run(), out) and _lib.lib().evo_lost_waits(0) == 0


def test_a_model_call_that_reads_its_results_raises(monkeypatch):
    from evo_b200 import CharLevelTokenizer, score_sequences
    from evo_b200.stripedhyena import StripedHyena, dotdict
    from oracle import stripedhyena_oracle as O
    monkeypatch.setenv("EVO_B200_HYENA_VARIANT", "2")
    cfg = O.tiny_config(num_layers=2, attn_layer_idxs=(1,), hidden_size=256, num_heads=2)
    model = StripedHyena(dotdict(cfg))
    model.load_state_dict(O.random_state_dict(cfg, seed=1), strict=True)
    model = model.to_bfloat16_except_poles_residues().to(DEV)
    seqs = ["ACGT" * 40, "ACG"]
    want = score_sequences(seqs, model, CharLevelTokenizer(512), device=DEV)
    with _no_tries(), pytest.raises(EvoError, match="ran out"):
        score_sequences(seqs, model, CharLevelTokenizer(512), device=DEV)
    assert score_sequences(seqs, model, CharLevelTokenizer(512), device=DEV) == want
