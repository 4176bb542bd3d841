"""The barriers of the attention backward kernel, walked through every interleaving.

The kernel's roles (copies, products, the threads of P and dS, those of dQ) meet at mbarriers whose waits name a parity.  A wait is
lost when its phase is followed by another before the waiter has looked: it then waits for a phase that needs the waiter itself.
Here every role is the list of its barrier operations -- the P and dS threads' as the kernel's source has them -- and a search
over all orders looks for a state in which nobody can go on.
"""
import re
from pathlib import Path

import pytest

SOURCE = Path(__file__).resolve().parent.parent / "arctic_platform_b200" / "csrc" / "attention_bwd.cu"
WARPS = 2                     # of P and dS: one that is held up and one that is not
ARRIVALS = {"q_full0": 1, "q_full1": 1, "q_empty0": 1, "q_empty1": 1, "do_full": 1, "do_empty": 1, "s_full": 1, "p_full": WARPS,
            "dp_full": 1, "ds_full": WARPS, "dq_full": 1, "dq_read": 1}


def _order_of_p_and_ds():
    """``[("wait" | "arrive", barrier), ...]`` of one tile, in the order of the source."""
    text = SOURCE.read_text()
    begin = text.index("P and dS: 64 columns of every tile per group")
    body = text[begin:text.index("// dK (first group) and dV (second) of this block", begin)]
    ops = [("wait" if w else "arrive", w or a) for w, a in re.findall(r"\bwait\(&?(\w+)|mbar_arrive\((\w+)\)", body)]
    assert sorted(ops) == sorted([("wait", "q_full"), ("wait", "s_full"), ("arrive", "p_full"), ("wait", "do_full"),
                                  ("wait", "dp_full"), ("arrive", "ds_full")])
    return ops


def _roles(tiles, order):
    """Operations of every role over ``tiles`` tiles: ("w", barrier, parity) and ("a", barrier).  A copy or a product is done as soon as
    it is issued -- the earliest that its barrier can move on."""
    q = lambda name, i: "%s%d" % (name, i & 1)
    copies, products, dq = [], [], []
    for i in range(tiles):
        copies += [("w", q("q_empty", i), ((i >> 1) & 1) ^ 1), ("a", q("q_full", i)), ("w", "do_empty", (i & 1) ^ 1), ("a", "do_full")]
        dq += [("w", "dq_full", i & 1), ("a", "dq_read")]
    products += [("w", "q_full0", 0), ("a", "s_full"), ("w", "do_full", 0), ("a", "dp_full"), ("w", "p_full", 0), ("a", "do_empty")]
    for i in range(tiles):
        more = i + 1 < tiles
        if more:
            products += [("w", q("q_full", i + 1), ((i + 1) >> 1) & 1), ("a", "s_full")]
        products += [("w", "ds_full", i & 1), ("a", "dq_full"), ("a", q("q_empty", i))]
        if more:
            products += [("w", "do_full", (i + 1) & 1), ("w", "dq_read", i & 1), ("a", "dp_full"), ("w", "p_full", (i + 1) & 1),
                         ("a", "do_empty")]
    worker = []
    for i in range(tiles):
        for kind, name in order:
            bar, parity = (q(name, i), (i >> 1) & 1) if name == "q_full" else (name, i & 1)
            worker.append(("w", bar, parity) if kind == "wait" else ("a", bar))
    return [copies, products, dq] + [worker] * WARPS


def _stuck(roles):
    """A reachable state in which somebody is left and nobody can go on, or None."""
    names = sorted(ARRIVALS)
    place = {n: k for k, n in enumerate(names)}
    start = ((0,) * len(roles), ((0, 0),) * len(names))       # next operation per role; (phases over, arrivals of the present one)
    seen, todo = {start}, [start]
    while todo:
        at, bars = todo.pop()
        moved = False
        for r, ops in enumerate(roles):
            if at[r] == len(ops):
                continue
            op = ops[at[r]]
            k = place[op[1]]
            over, count = bars[k]
            if op[0] == "w":
                if over % 2 == op[2]:
                    continue                                  # the phase of this parity is not over
                nxt = bars
            else:
                count += 1
                new = (over + 1, 0) if count == ARRIVALS[op[1]] else (over, count)
                nxt = bars[:k] + (new,) + bars[k + 1:]
            moved = True
            state = (at[:r] + (at[r] + 1,) + at[r + 1:], nxt)
            if state not in seen:
                seen.add(state)
                todo.append(state)
        if not moved and any(at[r] < len(ops) for r, ops in enumerate(roles)):
            return [ops[at[r]] if at[r] < len(ops) else "done" for r, ops in enumerate(roles)]
    return None


@pytest.mark.parametrize("tiles", [1, 2, 3, 5])
def test_no_wait_of_the_kernel_can_be_lost(tiles):
    assert _stuck(_roles(tiles, _order_of_p_and_ds())) is None


def test_the_search_sees_a_lost_wait():
    """P published before dO has been seen: the buffer may be filled again in between."""
    order = [("wait", "q_full"), ("wait", "s_full"), ("arrive", "p_full"), ("wait", "do_full"), ("wait", "dp_full"), ("arrive", "ds_full")]
    stuck = _stuck(_roles(3, order))
    assert stuck is not None and any(op[:2] == ("w", "do_full") for op in stuck)
