"""The tiles that evo_gemm picks for a shape leave the bits of a result as they are: around the lines of the rule, and its three forms against one another."""
import math

import pytest
import torch

import evo_b200._lib as _lib
from evo_b200.engine import KernelOps

pytestmark = pytest.mark.gpu
DEV, BF = "cuda:0", torch.bfloat16


class _Ops(KernelOps):
    _prof, gemm_variant, gemm_variant_gate = None, 0, 0


# one row block and several; 296 small tiles and more; a wave less in narrow tiles; one row behind and in front of a block's end; K past the small tile's line
@pytest.mark.parametrize("M,N,K", [(65, 512, 64), (127, 4096, 256), (129, 256, 4096), (384, 6144, 128), (385, 6144, 128), (300, 12288, 256), (513, 4096, 320), (141, 2048, 6208), (640, 11008, 128),
                                   (1, 256, 64), (2368, 1024, 64), (2369, 1024, 64)])
def test_picked_tiles_are_the_same_bits(M, N, K, monkeypatch):
    g = torch.Generator(device=DEV).manual_seed(M + N)
    a, w = torch.randn(M, K, generator=g, device=DEV).to(BF), (torch.randn(N, K, generator=g, device=DEV) / math.sqrt(K)).to(BF)
    bias, resid = torch.randn(N, generator=g, device=DEV).to(BF), torch.randn(M, N, generator=g, device=DEV).to(BF)
    for epi in (_lib.EPI_NONE, _lib.EPI_BIAS, _lib.EPI_BIAS_RESID, _lib.EPI_RESID, _lib.EPI_SILU_COLS, _lib.EPI_GELU_GATE, _lib.EPI_GELU_TANH_GATE):
        gate = epi in (_lib.EPI_GELU_GATE, _lib.EPI_GELU_TANH_GATE)
        outs = []
        for tile in (None, "0", "1", "2"):
            monkeypatch.delenv("EVO_B200_GEMM_TILE", raising=False)
            if tile is not None:
                monkeypatch.setenv("EVO_B200_GEMM_TILE", tile)
            out = torch.full((M + 1, N // 2 if gate else N), 7.0, dtype=BF, device=DEV)
            _Ops()._gemm(a, w, out, M, N, K, epi, bias=bias, resid=resid, ldc=out.shape[1], act_cols=N // 2)
            assert (out[M] == 7.0).all()
            outs.append(out)
        assert all(torch.equal(outs[0], o) for o in outs[1:]), epi
        if epi == _lib.EPI_NONE:
            want = a.double() @ w.double().T
            # half a step of bf16, and K products in fp32
            assert ((outs[0][:M].double() - want).abs() <= 1.01 * 2.0 ** -8 * want.abs() + 2.0 ** -16 * want.abs().max()).all()


@pytest.mark.parametrize("setting", ["3", "-1", "12", "two", ""])
def test_an_unknown_tile_is_no_tile(setting, monkeypatch):
    """EVO_B200_GEMM_TILE names a tile with 0, 1 or 2; anything else leaves the choice to the rule, for the epilogues that the 128 x 64 tile does not have as well."""
    g = torch.Generator(device=DEV).manual_seed(1)
    M, N, K = 100, 512, 192
    a, w = torch.randn(M, K, generator=g, device=DEV).to(BF), (torch.randn(N, K, generator=g, device=DEV) / math.sqrt(K)).to(BF)
    for epi in (_lib.EPI_NONE, _lib.EPI_GELU_GATE, _lib.EPI_GELU_TANH_GATE):
        outs = []
        for value in (None, setting):
            monkeypatch.delenv("EVO_B200_GEMM_TILE", raising=False)
            if value is not None:
                monkeypatch.setenv("EVO_B200_GEMM_TILE", value)
            outs.append(torch.zeros(M, N if epi == _lib.EPI_NONE else N // 2, dtype=BF, device=DEV))
            _Ops()._gemm(a, w, outs[-1], M, N, K, epi, ldc=outs[-1].shape[1])
        assert torch.equal(*outs) and outs[0].abs().max() > 0


@pytest.mark.parametrize("tile", ["0", "1"])
@pytest.mark.parametrize("M,N,K", [(1, 256, 64), (16, 12288, 4096), (65, 768, 256), (129, 512, 4096), (257, 256, 64), (300, 1024, 256)])
def test_big_tiles_on_few_rows(M, N, K, tile, monkeypatch):
    """Pairs and 128 x 256 tiles where the rule takes smaller ones: every epilogue against products in 64 bits."""
    monkeypatch.setenv("EVO_B200_GEMM_TILE", tile)
    g = torch.Generator(device=DEV).manual_seed(M + N + K)
    n = lambda *s: torch.randn(*s, generator=g, device=DEV)  # noqa: E731
    a, w, bias, resid = n(M, K).to(BF), (n(N, K) / math.sqrt(K)).to(BF), n(N).to(BF), n(M, N).to(BF)
    F, r = torch.nn.functional, lambda x: x.to(BF).double()  # noqa: E731
    acc = a.double() @ w.double().T
    t = acc.view(M, -1, 2, 128)
    l1, l2 = t[:, :, 0].reshape(M, -1), t[:, :, 1].reshape(M, -1)
    cols = torch.arange(N, device=DEV) < N // 2
    # what is expected, and by how much a sum that rounds to the other neighbour moves it (steps of 2^-8 of each rounded factor)
    want = {_lib.EPI_NONE: (acc, 0 * acc), _lib.EPI_BIAS: (acc + bias.double(), 0 * acc),
            _lib.EPI_BIAS_RESID: (r(acc + bias.double()) + resid.double(), 2.0 ** -7 * (acc + bias.double()).abs()), _lib.EPI_RESID: (r(acc) + resid.double(), 2.0 ** -7 * acc.abs()),
            _lib.EPI_SILU_COLS: (torch.where(cols, F.silu(acc), acc), 0 * acc), _lib.EPI_GELU_GATE: (r(F.gelu(r(l1))) * r(l2), 2.0 ** -6 * (l1 * l2).abs()),
            _lib.EPI_GELU_TANH_GATE: (F.gelu(l1, approximate="tanh") * l2, 0 * l1)}
    for epi, (ref, slack) in want.items():
        out = torch.full((M + 1, ref.shape[1]), 7.0, dtype=BF, device=DEV)
        _Ops()._gemm(a, w, out, M, N, K, epi, bias=bias, resid=resid, ldc=out.shape[1], act_cols=N // 2)
        assert (out[M] == 7.0).all()
        # half a step of bf16 of the result, and 2^-16 of the sums' scale for K products in fp32
        assert ((out[:M].double() - ref).abs() <= 1.01 * 2.0 ** -8 * ref.abs() + slack + 2.0 ** -16 * max(1.0, ref.abs().max().item())).all(), epi
