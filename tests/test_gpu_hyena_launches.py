"""The inputs that a call of the Hyena operator leaves for the next one: copied beside the operator, and behind it where they take the place of those it begins with."""
import ctypes as C
import os
import sys

import pytest
import torch

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
from evo_b200 import _lib  # noqa: E402
from evo_b200._lib import HyenaParams, check, ptr  # noqa: E402

pytestmark = pytest.mark.gpu
DEV = "cuda:0"
BF = torch.bfloat16


@pytest.mark.parametrize("variant", ["0", "1", "2"])
@pytest.mark.parametrize("B,L", [(1, 1), (3, 2), (2, 70), (1, 1500)])
def test_kept_inputs(monkeypatch, variant, B, L):
    monkeypatch.setenv("EVO_B200_HYENA_VARIANT", variant)
    D = 256
    g = torch.Generator(device=DEV).manual_seed(L)
    n = lambda *s: torch.randn(*s, generator=g, device=DEV)  # noqa: E731
    z, halo, fw, fb, sk = n(B, L, 3 * D).to(BF), n(B, 2, 3 * D).to(BF), n(3 * D, 1, 3).to(BF), n(3 * D).to(BF), n(D).to(BF)
    poles, res, state = (0.6 * n(D, 8, 1, 2)).clamp(-0.6, 0.6).contiguous(), n(D, 8, 1, 2), n(B, D, 8, 2)

    def run(carried, over):
        y, end = torch.empty(B, L, D, dtype=BF, device=DEV), torch.empty(B, D, 8, 2, device=DEV)
        first = halo.clone()
        kept = first.view(B, 3 * D, 2) if over else torch.empty(B, 3 * D, 2, dtype=BF, device=DEV)
        p = HyenaParams(z=z.data_ptr(), y=y.data_ptr(), fir_w=fw.data_ptr(), fir_b=fb.data_ptr(), Dskip=sk.data_ptr(), poles=poles.data_ptr(), residues=res.data_ptr(), B=B, L=L,
                        D=D, S=8, nheads=D // 128, state_out=end.data_ptr(), fir_state_out=kept.data_ptr())
        if carried:
            p.halo, p.state_in = first.data_ptr(), state.data_ptr()
        nb = _lib.lib().evo_hyena_fwd_workspace(C.byref(p))
        ws = torch.empty(max(nb, 1), dtype=torch.uint8, device=DEV)
        check(_lib.lib().evo_hyena_fwd(C.byref(p), ptr(ws), nb, C.c_void_p(torch.cuda.current_stream().cuda_stream)), "evo_hyena_fwd")
        torch.cuda.synchronize()
        return y, end, kept

    for carried in (False, True):
        y, end, kept = run(carried, False)
        want = torch.cat([halo if carried else torch.zeros_like(halo), z], 1)[:, -2:].permute(0, 2, 1)
        assert torch.equal(kept, want)
        if L >= 2:                                    # (of a single token the place is read and written: its second input is the halo's)
            y2, end2, kept2 = run(carried, True)
            assert torch.equal(kept2, want) and torch.equal(y2, y) and torch.equal(end2, end)
