"""Attention of a decode step over caches that are not whole tiles, against 64 bits."""
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


@pytest.mark.parametrize("S", [1, 63, 64, 65, 127, 1063])
@pytest.mark.parametrize("B,H,nsplit", [(1, 2, 16), (3, 4, 3)])
def test_attention_of_a_step_over_caches_of_any_length(S, B, H, nsplit):
    """Against 64 bits.  The result is rounded to bf16 (2^-9 of an element at most); where the cache is whole tiles, the weights are rounded before they meet the values, too, which is
    below another 2^-9 of the result's norm.  What lies behind the last key, in the same sequence, the next or past the cache, holds NaN."""
    hd = 128
    g = torch.Generator(device=DEV).manual_seed(S)
    cache = torch.randn(B, S, 2, H, hd, generator=g, device=DEV).to(BF)
    qkv = torch.randn(B, 3, H, hd, generator=g, device=DEV).to(BF)
    lib = _lib.lib()
    for pos in sorted({0, min(S, 62) - 1, S // 2, S - 1} - {-1}):
        dirty = cache.clone()
        dirty[:, pos + 1:] = math.nan
        out = torch.empty(B, H, hd, dtype=BF, device=DEV)
        at = torch.tensor([pos], dtype=torch.int64, device=DEV)
        nws = lib.evo_decode_attn_workspace(B, H, nsplit)
        ws = torch.empty(nws, dtype=torch.uint8, device=DEV)
        check(lib.evo_decode_attn(ptr(qkv), ptr(dirty), ptr(out), ptr(at), B, H, hd, S, nsplit, hd ** -0.5, ptr(ws), nws, _stream()), "evo_decode_attn")
        q, k, v = qkv[:, 0].double(), cache[:, :pos + 1, 0].double(), cache[:, :pos + 1, 1].double()
        w = torch.softmax(torch.einsum("bhd,bkhd->bhk", q, k) * hd ** -0.5, -1)
        want = torch.einsum("bhk,bkhd->bhd", w, v)
        assert (out.double() - want).norm() <= 2.0 ** (-8 if S % 64 == 0 else -9) * want.norm(), pos
