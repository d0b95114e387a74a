"""The hand-overs of a seven-warp team of a batch (seq_unit), as a model on the
host: any interleaving of the warps, barriers that open at two arrivals.  The
order of a row's two arrivals, and whether a row may skip the wait for the early
one, are read from the kernel's source."""
import random
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "sptrsv_b200" / "csrc"
W, H = 7, 4


def _row(r, rows, kind, form):
    """What row r's warp does: (op, argument) with sync and arrive at a barrier,
    read of a range of rows and store of this one."""
    me, late, middle, in_turn = r % W, *kind
    order, waits = form
    ops, before = [("read", (0, r - W))], []
    if r >= H:
        if middle and not in_turn:
            ops += [("sync", 8 + me), ("read", (r - 6, r - H))]
        elif waits:
            before = [("sync", 8 + me)]
        else:
            ops += [("arrive", 8 + me)]
    turn = before + ([("sync", 1 + me)] if r > 0 else [])
    if in_turn:
        ops += turn + [("read", (0, r - 1)), ("store", r)]
    elif late:
        ops += turn + [("read", (r - H + 1, r - 1)), ("store", r)]
    else:
        ops += [("store", r)] + turn
    hand = {"next": [("arrive", 1 + (me + 1) % W)] if r + 1 < rows else [],
            "ahead": [("arrive", 8 + (me + H) % W)] if r + H < rows else []}
    return ops + hand[order[0]] + hand[order[1]]


def _run(seed, form, rows=40):
    """Rows read before they were stored; None when the warps stop."""
    rng = random.Random(seed)
    kinds = [(rng.random() < 0.5, rng.random() < 0.5, rng.random() < 0.1) for _ in range(rows)]
    prog = [[op for r in range(w, rows, W) for op in _row(r, rows, kinds[r], form)] for w in range(W)]
    speed = [rng.choice((1, 1, 1, 30)) for _ in range(W)]  # now and then a warp that is held up
    at, count, waits, stored, early = [0] * W, {}, {}, set(), 0
    while True:
        able = [w for w in range(W) if at[w] < len(prog[w]) and w not in waits]
        if not able:
            return early if all(at[w] == len(prog[w]) for w in range(W)) else None
        w = rng.choices(able, [1 / speed[v] for v in able])[0]
        op, arg = prog[w][at[w]]
        at[w] += 1
        if op == "store":
            stored.add(arg)
        elif op == "read":
            early += any(q >= 0 and q not in stored for q in range(max(0, arg[0]), arg[1] + 1))
        else:
            if op == "sync":
                waits[w] = arg
            count[arg] = count.get(arg, 0) + 1
            if count[arg] == 2:
                count[arg] = 0
                waits = {v: b for v, b in waits.items() if b != arg}


def _source_form():
    """(order of a row's two arrivals, whether every row waits for its early hand-over)"""
    text = (CSRC / "batch.cu").read_text()
    body = text[text.index("void seq_unit("):text.index("before the team's next unit")]
    order = re.findall(r'barrier\.cta\.arrive %0, 64;" ::"r"\((next|ahead)\)', body)
    early = re.findall(r'barrier\.cta\.(\w+) %0, 64;" ::"r"\(8 \+ tw\)', body)
    assert sorted(order) == ["ahead", "next"] and len(early) >= 3
    return tuple(order), set(early) == {"sync"}


def test_no_row_is_read_before_it_is_stored():
    form = _source_form()
    assert [_run(s, form) for s in range(600)] == [0] * 600


@pytest.mark.parametrize("order", [("next", "ahead"), ("ahead", "next")])
def test_the_model_tells_the_safe_forms_from_the_other(order):
    assert any(_run(s, (order, False)) != 0 for s in range(600)) == (order[0] == "next")
    assert all(_run(s, (order, True)) == 0 for s in range(200))
