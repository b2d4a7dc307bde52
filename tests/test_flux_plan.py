"""A model of the row waits between a step's passes on the flux pass: the
single grid's (tile_begin, lsh_kernels.cuh) and the queue's (item_rows and
producer_rows, lsh_queue.cuh), which are the same rows.  For every two tiles
of different passes that touch one row of an array, one of them writing, a
chain of waits has to order them, also over a stage's end, where slopes, edge
planes, marks and the state are used again."""
import pytest

T = 4  # rows of a tile


def passes(order):
    return ["flux", "update"] if order == 1 else ["slopes", "flux", "update"] * 2


def tile_rows(op, ny):
    return ny // T + 1 if op == "flux" else (ny + T - 1) // T  # edge rows 0 .. ny


def rows(lo, hi, n):
    return set(range(max(lo, 0), min(hi, n - 1) + 1))


def touched(op, stage, order, t, ny):
    """(reads, writes): array name -> rows.  E: edge rows; M: marks; D: the limiter's depths."""
    src = "Y" if stage else "X"
    dst = "X" if order == 1 or stage else "Y"
    depth = "D" if order == 1 else src
    a, b = T * t, T * t + T - 1
    if op == "slopes":
        return {src: rows(a - 1, b + 1, ny)}, {"S": rows(a, b, ny)}
    if op == "flux":
        w = {"E": rows(a, b, ny + 1), "M": rows(a - 1, b, ny)}
        if order == 1:
            w["D"] = rows(a, b, ny)
        return {src: rows(a - 1, b, ny), "S": rows(a - 1, b, ny)}, w
    # the limiter's partial sums reach the edges of the cells above and below
    r = {"E": rows(a - 1, b + 2, ny + 1), "M": rows(a - 2, b + 2, ny), "S": rows(a, b, ny), "X": rows(a, b, ny)}
    r[src] = rows(a, b, ny)
    r[depth] = r[depth] | rows(a - 2, b + 2, ny) if depth in r else rows(a - 2, b + 2, ny)
    return r, {dst: rows(a, b, ny)}


def waits(op, t, producer_rows, after_update):
    """The producer's tile rows that tile row t of `op` waits for."""
    after = {"slopes": 1, "flux": 0, "update": after_update}[op]
    return range(max(t - 1, 0), min(t + after, producer_rows - 1) + 1)


def unordered(order, ny, after_update=1):
    ops = passes(order)
    done = []  # done[p][t]: every (pass, tile row) finished before it starts
    for p, op in enumerate(ops):
        cur = []
        for t in range(tile_rows(op, ny)):
            s = set()
            if p:
                for r in waits(op, t, tile_rows(ops[p - 1], ny), after_update):
                    s |= done[p - 1][r] | {(p - 1, r)}
            cur.append(s)
        done.append(cur)
    acc = [[touched(op, p // 3 if order == 2 else 0, order, t, ny) for t in range(tile_rows(op, ny))]
           for p, op in enumerate(ops)]
    bad = 0
    for q in range(len(ops)):
        for u, (ru, wu) in enumerate(acc[q]):
            for p in range(q):
                for t, (rt, wt) in enumerate(acc[p]):
                    clash = any(wt.get(k, set()) & (ru.get(k, set()) | wu.get(k, set())) for k in wt)
                    clash |= any(rt.get(k, set()) & wu.get(k, set()) for k in wu)
                    bad += clash and (p, t) not in done[q][u]
    return bad


@pytest.mark.parametrize("order", [1, 2])
@pytest.mark.parametrize("ny", [1, 3, 4, 5, 8, 17, 32, 33])
def test_waits_order_every_conflict(order, ny):
    assert unordered(order, ny) == 0


@pytest.mark.parametrize("order", [1, 2])
def test_a_missing_row_is_found(order):
    assert unordered(order, 17, after_update=0) > 0
