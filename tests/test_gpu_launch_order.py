"""Chains of small kernels that are resident at once, their buffers written again by the next turn: in a stream and in a captured graph they give the bits of calls that are waited for."""
import ctypes as C

import pytest
import torch

import evo_b200._lib as _lib
from evo_b200._lib import check, ptr
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
@pytest.mark.parametrize("level", [0, 1, 2, 3, 4])
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
