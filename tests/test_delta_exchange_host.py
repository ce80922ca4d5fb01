"""The exchange of sums between the two CTAs that share a head of the gated delta scan, as a model whose orders are all tried."""
import os
import re

import pytest

SOURCE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "evo_b200", "csrc", "delta_block.cu")


def _first_fault(places, warps, blocks):
    """Two CTAs with `warps` read-out warps of one parity and `blocks` blocks.  A warp's steps of a block: meet the others (of its CTA); the first warp expects the block's bytes at the
    barrier of its place; meet; send a sum to the other CTA, where it arrives at any later time, in any order; wait for the barrier's phase; read.  Returns what goes wrong in some order
    of these, or None.  A barrier is (phase, arrivals to come, bytes to come); a wait sees the parity of the phase only, as an mbarrier's does."""
    MEET, EXPECT, MEET2, SEND, WAIT, READ = range(6)
    barrier = (0, 1, 0)
    start = (tuple((0, MEET) for _ in range(2 * warps)), tuple(barrier for _ in range(2 * places)), tuple(-1 for _ in range(2 * places * warps)), frozenset())

    def settle(b):
        phase, pending, tx = b
        return (phase + 1, 1, 0) if pending == 0 and tx == 0 else b

    def put(t, i, v):
        return t[:i] + (v,) + t[i + 1:]

    seen, todo = {start}, [start]
    while todo:
        pcs, bars, slots, flying = todo.pop()
        after = []
        for w, (n, step) in enumerate(pcs):
            if n == blocks:
                continue
            cta, me = divmod(w, warps)
            at = cta * places + n % places
            if step in (MEET, MEET2):                                # all go on when the last one is there
                first = cta * warps
                if all(pcs[first + i] == (n, step) for i in range(warps)):
                    p = pcs
                    for i in range(warps):
                        p = put(p, first + i, (n, step + 1))
                    after.append((p, bars, slots, flying))
            elif step == EXPECT:
                b = bars
                if me == 0:
                    phase, pending, tx = bars[at]
                    if pending != 1:
                        return "a phase is expected twice"
                    b = put(bars, at, settle((phase, 0, tx + warps)))
                after.append((put(pcs, w, (n, MEET2)), b, slots, flying))
            elif step == SEND:
                after.append((put(pcs, w, (n, WAIT)), bars, slots, flying | {(1 - cta, me, n)}))
            elif step == WAIT:
                if bars[at][0] % 2 != n // places % 2:
                    after.append((put(pcs, w, (n, READ)), bars, slots, flying))
            else:
                if slots[at * warps + me] != n:
                    return f"block {n} reads the sum of block {slots[at * warps + me]}"
                after.append((put(pcs, w, (n + 1, MEET)), bars, slots, flying))
        for cta, me, n in flying:
            at = cta * places + n % places
            phase, pending, tx = bars[at]
            after.append((pcs, put(bars, at, settle((phase, pending, tx - 1))), put(slots, at * warps + me, n), flying - {(cta, me, n)}))
        if not after and any(n < blocks for n, _ in pcs):
            return "nobody goes on"
        for s in after:
            if s not in seen:
                seen.add(s)
                todo.append(s)
    return None


@pytest.mark.parametrize("warps,blocks", [(1, 6), (2, 5)])
def test_no_order_of_the_exchange_loses_a_sum(warps, blocks):
    """With as many places as the kernel has; one would lose sums, which shows that the model sees it."""
    places = int(re.search(r"NORM_TURNS = (\d+)", open(SOURCE).read()).group(1))
    assert _first_fault(places, warps, blocks) is None
    assert _first_fault(1, warps, blocks) is not None
