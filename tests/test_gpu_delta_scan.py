"""The gated delta rule's scan where its CTAs, lanes and rows are used differently: heads over one, two or three CTAs, channels that leave lanes empty, rows that start anywhere."""
import math
import os
import sys

import pytest
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, ROOT)
sys.path.insert(0, os.path.join(ROOT, "tests"))
import test_gpu_delta_block as D  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dk", [64, 128])
@pytest.mark.parametrize("dv", [16, 48, 64, 80, 96, 128, 144, 192])
def test_value_channels_over_ctas(dk, dv):
    """One CTA up to 64 channels, a cluster of two up to 128, and beyond that CTAs that leave fp32 read-outs to a norm of their own.  Bounds: one rounding to bf16, fp32 throughout."""
    B, L, H, G = 2, 150, 4, 2
    t = D._inputs(B, L, H, G, dk, dv, seed=dv)
    out, S, _ = D._run(t, B, L, H, G, dk, dv, ldo=H * dv + 8)
    want, state = D._oracle(t, B, L, H, G, dk, dv, 0)
    assert (out[:, :H * dv].double() - want).norm() <= 2.2e-3 * want.norm()
    assert (S.double() - state).norm() <= 1e-6 * state.norm()
    assert not out[:, H * dv:].any()


@pytest.mark.parametrize("dv", [32, 128])
@pytest.mark.parametrize("pad,extra", [(1, 0), (0, 3), (3, 5)])
def test_gates_and_outputs_that_start_anywhere(dv, pad, extra):
    """Gate rows and output rows that are not on four elements: the same bits as aligned ones."""
    B, L, H, dk = 1, 130, 3, 128
    t = D._inputs(B, L, H, H, dk, dv, seed=7)
    want, S, _ = D._run(t, B, L, H, H, dk, dv)
    odd = dict(t, z=torch.nn.functional.pad(t["z"], (0, pad)).contiguous())
    out, S2, _ = D._run(odd, B, L, H, H, dk, dv, ldo=H * dv + extra)
    assert torch.equal(out[:, :H * dv], want) and torch.equal(S2, S) and not out[:, H * dv:].any()


@pytest.mark.parametrize("dk,dv", [(128, 128), (64, 128), (64, 32)])
@pytest.mark.parametrize("what", ["v", "k", "q", "state"])
def test_what_is_not_finite_in_a_channel(dk, dv, what):
    """A block goes token by token where a read-out, an update or the state is not finite: what is behind the token, and only that, and only in the channels that it reaches."""
    B, L, H, at = 1, 200, 2, 70
    t = D._inputs(B, L, H, H, dk, dv, seed=5)
    clean, _, _ = D._run(t, B, L, H, H, dk, dv)
    bad = {k: v.clone() for k, v in t.items()}
    if what == "state":
        bad["S"][0, 0, 3, dv - 1] = math.inf
        at = 0
    else:
        bad["x"][at, {"q": 0, "k": H * dk, "v": 2 * H * dk + dv - 2}[what] + 1] = math.nan
    out, _, _ = D._run(bad, B, L, H, H, dk, dv)
    assert (out[:at].float() - clean[:at].float()).norm() <= 1e-4 * clean[:at].float().norm()
    assert torch.equal(out[:, dv:], clean[:, dv:])                              # the other head
    step = D._run(dict(bad, x=bad["x"].float(), z=bad["z"].float()), B, L, H, H, dk, dv)[0]
    assert torch.equal(torch.isfinite(out.float()), torch.isfinite(step))


@pytest.mark.parametrize("H,B", [(36, 2), (38, 2), (75, 2)])
def test_pairs_around_the_number_of_sms(H, B):
    """Dependent and ordinary launches, and a second wave: each sequence as if it were alone."""
    L, dk, dv = 70, 64, 128
    t = D._inputs(B, L, H, H, dk, dv, seed=H)
    out, S, _ = D._run(t, B, L, H, H, dk, dv)
    for b in range(B):
        one = {k: (v[b * L:(b + 1) * L] if k in "xz" else v[b:b + 1] if k == "S" else v) for k, v in t.items()}
        o, s, _ = D._run(one, 1, L, H, H, dk, dv)
        assert torch.equal(out[b * L:(b + 1) * L], o) and torch.equal(S[b], s[0])


@pytest.mark.parametrize("dv", [80, 128])
def test_heads_over_two_ctas_for_many_blocks(dv):
    """The two CTAs of a head exchange a sum per token for every block: each row of each head is scaled by its own (a result is rounded to bf16, 2^-9 of it, against fp32), and a
    sequence's results do not depend on what runs beside it."""
    B, L, H, dk = 3, 64 * 66 + 5, 4, 64
    t = D._inputs(B, L, H, H, dk, dv, seed=dv)
    out, S, _ = D._run(t, B, L, H, H, dk, dv)
    want, _, _ = D._run(dict(t, x=t["x"].float(), z=t["z"].float()), B, L, H, H, dk, dv)
    off = (out.float() - want).view(B * L, H, dv).norm(dim=-1) / want.view(B * L, H, dv).norm(dim=-1)
    assert off.max() <= 2.0 ** -8
    for b in range(B):
        one = {k: (v[b * L:(b + 1) * L] if k in "xz" else v[b:b + 1] if k == "S" else v) for k, v in t.items()}
        o, s, _ = D._run(one, 1, L, H, H, dk, dv)
        assert torch.equal(out[b * L:(b + 1) * L], o) and torch.equal(S[b], s[0])


@pytest.mark.parametrize("B,H,G,dk,dv,L,zero", [(38, 4, 2, 64, 32, 64, 0), (38, 4, 4, 128, 32, 48, 1), (200, 2, 1, 64, 16, 49, 0), (100, 2, 2, 64, 80, 63, 0), (100, 2, 1, 128, 128, 64, 0), (26, 2, 2, 64, 192, 64, 0), (38, 2, 2, 128, 144, 51, 1), (256, 2, 2, 128, 128, 33, 0),
                                                 (37, 4, 4, 64, 32, 64, 0), (75, 2, 2, 64, 128, 64, 0)])
def test_a_single_block_on_many_sms(B, H, G, dk, dv, L, zero):
    """Calls of one block with more CTAs than the chip takes at once, which have a kernel of their own (and, last, two that have not): the bounds of the blocks' other forms."""
    t = D._inputs(B, L, H, G, dk, dv, seed=L + dv)
    out, S, nb = D._run(t, B, L, H, G, dk, dv, zero, ldo=H * dv + 8)
    assert nb > 4 * B * L * H * dv                                              # the block form was taken
    want, state = D._oracle(t, B, L, H, G, dk, dv, zero)
    assert (out[:, :H * dv].double() - want).norm() <= 2.2e-3 * want.norm()
    assert (S.double() - state).norm() <= 1e-6 * state.norm()
    assert not out[:, H * dv:].any()
    odd = dict(t, z=torch.nn.functional.pad(t["z"], (0, 3)).contiguous())      # gate rows that start anywhere: another norm kernel, whose sums of squares run in another order
    assert (D._run(odd, B, L, H, G, dk, dv, zero)[0].double() - want).norm() <= 2.2e-3 * want.norm()
    none, _, _ = D._run(t, B, L, H, G, dk, dv, 1, state=False)
    assert torch.equal(none, D._run(t, B, L, H, G, dk, dv, 1)[0])


@pytest.mark.parametrize("dk,dv", [(64, 32), (128, 128)])
@pytest.mark.parametrize("what", ["v", "k", "q", "state"])
def test_what_is_not_finite_in_a_single_block(dk, dv, what):
    """The same as in the scan: what is behind the token, and only that, in its head; the other heads keep their bits."""
    B, L, H, at = 110, 64, 2, 20
    t = D._inputs(B, L, H, H, dk, dv, seed=5)
    clean, _, _ = D._run(t, B, L, H, H, dk, dv)
    bad = {k: v.clone() for k, v in t.items()}
    if what == "state":
        bad["S"][0, 0, 3, dv - 1] = math.inf
        at = 0
    else:
        bad["x"][at, {"q": 0, "k": H * dk, "v": 2 * H * dk + dv - 2}[what] + 1] = math.nan
    out, _, _ = D._run(bad, B, L, H, H, dk, dv)
    assert (out[:at].float() - clean[:at].float()).norm() <= 1e-4 * clean[:at].float().norm()
    assert torch.equal(out[:, dv:], clean[:, dv:]) and torch.equal(out[L:], clean[L:])
    step = D._run(dict(bad, x=bad["x"].float(), z=bad["z"].float()), B, L, H, H, dk, dv)[0]
    assert torch.equal(torch.isfinite(out.float()), torch.isfinite(step))
