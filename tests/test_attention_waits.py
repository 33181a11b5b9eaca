"""The waits at the end of the attention forward's kernel, explored on the CPU over every interleaving.

A wait on an mbarrier names a phase by its parity only, so it is sound while the waiter can meet the barrier in at
most two states.  The model below holds what the kernel's softmax warps and its tensor core may do in any order;
the wait itself is read from the source.
"""
import re
from pathlib import Path

import pytest

SRC = (Path(__file__).resolve().parent.parent / "rust_trainer_b200" / "csrc" / "attention_tc.cu").read_text()
WARPS = 2  # four behave as two do: the fastest and the slowest


def explore(ntiles, end_waits):
    """Problems ("stuck", "early") that some interleaving of the warps and the products P.V reaches.  `end_waits`:
    (barrier, parity) in order, barrier "pv" (one phase per product) or "last" (one phase, after the last product)."""
    found, seen, todo = set(), set(), [((0,) * WARPS, 0)]
    while todo:
        state = todo.pop()
        if state in seen:
            continue
        seen.add(state)
        at, done = state  # a warp's next tile, or ntiles + waits passed; products completed
        nxt = []
        if done < ntiles and all(a > done for a in at):  # every warp has left its P: the product may complete
            nxt.append((at, done + 1))
        for w, a in enumerate(at):
            if a < ntiles:
                go = a < 2 or done >= a - 1  # scores n come after product n - 2
            elif a < ntiles + len(end_waits):
                barrier, parity = end_waits[a - ntiles]
                phase = done if barrier == "pv" else int(done == ntiles)
                go = phase % 2 != parity
            else:
                if done < ntiles:
                    found.add("early")
                go = False
            if go:
                nxt.append((at[:w] + (a + 1,) + at[w + 1:], done))
        if not nxt and any(a < ntiles + len(end_waits) for a in at):
            found.add("stuck")
        todo += nxt
    return found


@pytest.mark.parametrize("ntiles", [1, 2, 3, 4, 5, 6])
def test_the_end_of_the_forward_neither_hangs_nor_reads_early(ntiles):
    kernel = SRC[SRC.index("attn_fwd_tc_kernel(const"):SRC.index("int fwd_tc_impl(")]
    end = kernel[kernel.index("if (lane == 0) mbar_arrive(&p_full[b]);"):kernel.index("// O / l as f16")]
    waits = re.findall(r"mbar_wait\(([^,]+), ([^,]+), status", end)
    assert waits == [("o_done", "0")] and kernel.count("umma_commit(o_done)") == 1
    assert explore(ntiles, [("last", 0)]) == set()


@pytest.mark.parametrize("ntiles", [3, 4, 5])
def test_the_model_tells_bad_ends_apart(ntiles):
    last, before = (ntiles - 1) & 1, ntiles & 1
    assert explore(ntiles, [("pv", last)]) == {"early"}
    assert explore(ntiles, [("pv", before), ("pv", last)]) == {"stuck"}
