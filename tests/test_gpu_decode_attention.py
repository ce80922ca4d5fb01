"""Attention of a decode step over caches that are not whole tiles, against 64 bits."""
import ctypes as C
import math
import os
import subprocess
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
    """Against 64 bits.  The result is rounded to bf16 (2^-9 of an element at most, 0.58 of that on average); where the cache is whole tiles, the weights are rounded before they meet the
    values, too, which is below another 2^-9 of the result's norm.  Other caches have a thread per 128th key of a split: all but the largest of its weights are rounded, by 0.58 * 2^-9
    on average, so with the result's rounding 0.82 * 2^-9 at most.  What lies behind the last key, in the same sequence, the next or past the cache, holds NaN."""
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


def _few_calls(path):
    """The attention of a step over caches that are not whole tiles, written to `path`."""
    hd, lib, got = 128, _lib.lib(), []
    for S, B, H, nsplit in ((1, 1, 2, 16), (63, 3, 4, 3), (65, 2, 4, 1), (1063, 1, 32, 16), (1063, 3, 4, 3), (2977, 2, 8, 7)):
        g = torch.Generator(device=DEV).manual_seed(S + B)
        cache, qkv = torch.randn(B, S, 2, H, hd, generator=g, device=DEV).to(BF), torch.randn(B, 3, H, hd, generator=g, device=DEV).to(BF)
        for pos in sorted({0, S // 2, S - 1}):
            out, at = torch.empty(B, H, hd, dtype=BF, device=DEV), torch.tensor([pos], dtype=torch.int64, device=DEV)
            nws = lib.evo_decode_attn_workspace(B, H, nsplit)
            ws = torch.empty(nws, dtype=torch.uint8, device=DEV)
            check(lib.evo_decode_attn(ptr(qkv), ptr(cache), ptr(out), ptr(at), B, H, hd, S, nsplit, hd ** -0.5, ptr(ws), nws, _stream()), "evo_decode_attn")
            got.append(out.cpu())
    torch.save(got, path)


def test_caches_that_are_not_whole_tiles_keep_their_bits(tmp_path):
    """The results over such caches are those of the kernel with a key per thread, bit for bit (the library reads the variable that picks it once per process)."""
    here, child = str(tmp_path / "here.pt"), str(tmp_path / "child.pt")
    _few_calls(here)
    root, tests = (os.path.dirname(os.path.dirname(os.path.abspath(__file__))), os.path.dirname(os.path.abspath(__file__)))
    code = f"import sys; sys.path[:0] = [{root!r}, {tests!r}]; import test_gpu_decode_attention as t; t._few_calls({child!r})"
    subprocess.run([sys.executable, "-c", code], check=True, timeout=300, env=dict(os.environ, EVO_B200_DECODE_ATTN_V1="1"))
    for a, b in zip(torch.load(here), torch.load(child), strict=True):
        assert torch.equal(a, b)
