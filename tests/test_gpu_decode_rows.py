"""The decode step's linear layer for few rows: the sums that are passed on, added up and stored are those of the rows that there are."""
import ctypes as C
import math
import os
import sys

import pytest
import torch

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
from evo_b200 import _lib  # noqa: E402
from evo_b200._lib import check, ptr  # noqa: E402

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
BF = torch.bfloat16


def _stream():
    return C.c_void_p(torch.cuda.current_stream().cuda_stream)


def _linear(a, w, M, epi, bias, resid):
    N, K = w.shape
    lib = _lib.lib()
    n_out = N // 2 if epi in (_lib.EPI_GELU_GATE, _lib.EPI_GELU_TANH_GATE) else N
    out = torch.full((M + 1, n_out), 7.0, dtype=BF, device=DEV)
    ws = torch.zeros(lib.evo_gemm_smallm_workspace(M, N, K, epi), dtype=torch.uint8, device=DEV)
    p = _lib.GemmSmallMParams(A=a.data_ptr(), lda=K, W=w.data_ptr(), C=out.data_ptr(), ldc=n_out, bias=bias.data_ptr(), residual=resid.data_ptr(), ldr=n_out, M=M, N=N, K=K,
                              epilogue=epi, workspace=ws.data_ptr(), workspace_bytes=ws.numel(), act_cols=N // 2)
    check(lib.evo_gemm_smallm(C.byref(p), _stream()), "evo_gemm_smallm")
    assert (out[M] == 7.0).all() and not ws[:16384].any()                     # the row behind stays, the tiles' counters are zero again
    return out[:M]


@pytest.mark.parametrize("epi", ["EPI_NONE", "EPI_BIAS", "EPI_BIAS_RESID", "EPI_RESID", "EPI_GELU_GATE", "EPI_GELU_TANH_GATE", "EPI_SILU_COLS"])
@pytest.mark.parametrize("N,K", [(768, 256), (4096, 4096), (1024, 64)])
def test_few_rows_are_the_first_rows_of_more(N, K, epi):
    """A row's sums do not depend on how many rows a call has (up to 16, and 17 to 32, share a tile width): bit for bit."""
    g = torch.Generator(device=DEV).manual_seed(N + K)
    n = lambda *s: torch.randn(*s, generator=g, device=DEV)  # noqa: E731
    a, w, bias, resid = n(32, K).to(BF), (n(N, K) / math.sqrt(K)).to(BF), n(N).to(BF), n(33, N).to(BF)
    for widest, rows in ((16, (1, 2, 3, 4, 5, 7, 8, 9, 12, 13, 15)), (32, (17, 21, 31))):
        full = _linear(a, w, widest, getattr(_lib, epi), bias, resid)
        for M in rows:
            assert torch.equal(_linear(a, w, M, getattr(_lib, epi), bias, resid), full[:M]), M


@pytest.mark.parametrize("epi", ["EPI_NONE", "EPI_BIAS_RESID", "EPI_GELU_GATE", "EPI_GELU_TANH_GATE"])
@pytest.mark.parametrize("N,K", [(768, 256), (8192, 2048), (2048, 5632)])
def test_many_rows_are_the_first_rows_of_more(N, K, epi):
    """The same around the number of rows from which on their sums are added up four rows at a time (or, gated, by column), and for each wider tile."""
    g = torch.Generator(device=DEV).manual_seed(N + K)
    n = lambda *s: torch.randn(*s, generator=g, device=DEV)  # noqa: E731
    a, w, bias, resid = n(64, K).to(BF), (n(N, K) / math.sqrt(K)).to(BF), n(N).to(BF), n(65, N).to(BF)
    for widest, rows in ((32, (17, 24, 25, 26, 29)), (48, (33, 40, 47)), (64, (49, 50, 63))):
        full = _linear(a, w, widest, getattr(_lib, epi), bias, resid)
        for M in rows:
            assert torch.equal(_linear(a, w, M, getattr(_lib, epi), bias, resid), full[:M]), M


@pytest.mark.parametrize("epi", ["EPI_BIAS_RESID", "EPI_NONE", "EPI_GELU_GATE", "EPI_SILU_COLS"])
@pytest.mark.parametrize("N,K", [(37632, 256), (37888, 256), (40960, 256), (77824, 128), (9728, 1088)])
def test_tiles_of_a_cta_in_turn(N, K, epi):
    """CTAs whose range is part of a tile, whole tiles and part of a third or fifth, on both sides of the line between one and two groups of epilogue warps (eight k-blocks per SM)."""
    g = torch.Generator(device=DEV).manual_seed(N + K)
    n = lambda *s: torch.randn(*s, generator=g, device=DEV)  # noqa: E731
    a, w, bias, resid = n(16, K).to(BF), (n(N, K) / math.sqrt(K)).to(BF), n(N).to(BF), n(17, N).to(BF)
    for M in (1, 16):
        got = _linear(a, w, M, getattr(_lib, epi), bias, resid).double()
        acc, r = a[:M].double() @ w.double().T, lambda x: x.to(BF).double()  # noqa: E731
        slack = torch.zeros_like(got)
        if epi == "EPI_NONE":
            want = acc
        elif epi == "EPI_BIAS_RESID":
            want, slack = r(acc + bias.double()) + resid[:M].double(), 2.0 ** -7 * (acc + bias.double()).abs()        # the rounded product may be a step away
        elif epi == "EPI_SILU_COLS":
            want = torch.where(torch.arange(N, device=DEV) < N // 2, torch.nn.functional.silu(acc), acc)
        else:
            t = acc.view(M, -1, 2, 128)
            want = (r(torch.nn.functional.gelu(r(t[:, :, 0]))) * r(t[:, :, 1])).reshape(M, -1)
            slack = (2.0 ** -6 * (t[:, :, 0].abs() * t[:, :, 1].abs())).reshape(M, -1)                                # three rounded factors, each a step of 2^-7 away at most
        # half a step of bf16 of the result, and 2^-16 of the sums' scale for K products in fp32
        assert ((got - want).abs() <= 1.01 * 2.0 ** -8 * want.abs() + slack + 2.0 ** -16 * want.abs().max()).all(), (M, epi)
