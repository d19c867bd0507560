"""The barriers of the attention forward with alternating score regions (heads wider than 64 channels), as a model: every
interleaving of the MMA-issuing thread, the tensor core and two softmax warps.  A wait by parity returns when the phase now
open has the other parity, so it must never be possible that the phase it means is two behind (it would never return) or
not reached yet (it would return at once)."""
import pytest


def explore(ntiles, two_done, rescale):
    """States that go wrong: ("lost", ...) for a deadlock, ("early", ...) for a wait that returns before its phase.
    ``two_done``: value products complete on a barrier per score region; else on one, and the epilogue waits for the last
    phase but one first.  ``rescale``: every tile raises the maximum, so each warp waits for the product before it."""
    def issuer():
        ops = [("issue", "S", 0)]
        for j in range(ntiles):
            if j + 1 < ntiles:
                ops.append(("issue", "S", j + 1))
            ops += [("wait", "p", j), ("issue", "O", j)]
        return ops

    def warp():
        ops = []
        for j in range(ntiles):
            ops.append(("wait", "s", j))
            if rescale and j:
                ops.append(("wait", "o", j - 1))
            ops.append(("arrive", "p", j))
        if not two_done and ntiles > 1:
            ops.append(("wait", "o", ntiles - 2))
        return ops + [("wait", "o", ntiles - 1)]

    progs = [issuer(), warp(), warp()]
    alternates = {"s": True, "p": True, "o": two_done}
    place = lambda kind, j: (kind, j & 1, j >> 1) if alternates[kind] else (kind, 0, j)
    need = {"s": 1, "p": 2, "o": 1}
    # state: program counters, products retired, arrivals at each barrier
    start = ((0, 0, 0), 0, ())
    seen, stack, wrong = {start}, [start], set()
    while stack:
        pcs, retired, arr = stack.pop()
        count = dict(arr)
        queue = [op for op in progs[0][:pcs[0]] if op[0] == "issue"]
        after = []
        if retired < len(queue):  # the tensor core works in order; each product's commit arrives on its barrier
            _, kind, j = queue[retired]
            b = place("s" if kind == "S" else "o", j)[:2]
            after.append((pcs, retired + 1, tuple(sorted({**count, b: count.get(b, 0) + 1}.items()))))
        for i, prog in enumerate(progs):
            if pcs[i] == len(prog):
                continue
            op, kind, j = prog[pcs[i]]
            nxt = tuple(pc + (k == i) for k, pc in enumerate(pcs))
            if op == "issue":
                after.append((nxt, retired, arr))
            elif op == "arrive":
                b = place(kind, j)[:2]
                after.append((nxt, retired, tuple(sorted({**count, b: count.get(b, 0) + 1}.items()))))
            else:
                *b, phase = place(kind, j)
                done = count.get(tuple(b), 0) // need[kind]  # phases completed = index of the one now open
                if done % 2 != phase % 2:
                    if done <= phase:
                        wrong.add(("early", kind, j))
                    after.append((nxt, retired, arr))
        if not after and any(pc < len(p) for pc, p in zip(pcs, progs)):
            wrong.add(("lost", *[p[pc][1:] for pc, p in zip(pcs, progs) if pc < len(p)]))
        for s in after:
            if s not in seen:
                seen.add(s)
                stack.append(s)
    return wrong


@pytest.mark.parametrize("rescale", [False, True])
@pytest.mark.parametrize("ntiles", [1, 2, 3, 4, 5, 6])
def test_no_wait_is_lost_or_early(ntiles, rescale):
    assert explore(ntiles, True, rescale) == set()


def test_the_model_sees_what_one_barrier_would_do():
    assert any(w[0] == "lost" for w in explore(3, False, False))


def explore_any_order(ntiles, wide, rescale, two_done=True):
    """The same with commits of their own: a commit arrives when the products queued before it are over, after the commits with fewer
    products before them; those with the same products before them arrive in any order.  ``wide``: heads of more than 64
    channels, whose score regions alternate; else the program of 64 channels, which queues the next scores behind the value
    products and commits both after.  Besides lost and early waits, ("touch", j): a warp may read or rescale the output of tile j
    while its product is under way."""
    def issuer():
        ops = [("issue", "S", 0), ("commit", "s", 0)]
        for j in range(ntiles):
            nxt = [("issue", "S", j + 1), ("commit", "s", j + 1)] if j + 1 < ntiles else []
            ops += (nxt if wide else []) + [("wait", "p", j), ("issue", "O", j)] + ([] if wide else nxt) + [("commit", "o", j)]
        return ops

    def warp():
        ops = []
        for j in range(ntiles):
            ops.append(("wait", "s", j))
            if rescale and j:
                ops += ([("wait", "o", j - 1)] if wide else []) + [("touch", "O", j - 1)]
            ops.append(("arrive", "p", j))
        return ops + [("wait", "o", ntiles - 1), ("touch", "O", ntiles - 1)]

    progs = [issuer(), warp(), warp()]
    alternates = {"s": wide, "p": wide, "o": two_done}
    place = lambda kind, j: (kind, j & 1, j >> 1) if alternates[kind] else (kind, 0, j)
    need = {"s": 1, "p": 2, "o": 1}
    start = ((0, 0, 0), 0, frozenset(), ())
    seen, stack, wrong = {start}, [start], set()
    while stack:
        pcs, retired, arrived, arr = stack.pop()
        count = dict(arr)
        add = lambda b: tuple(sorted({**count, b: count.get(b, 0) + 1}.items()))
        done = progs[0][:pcs[0]]
        queue = [op for op in done if op[0] == "issue"]
        after = []
        if retired < len(queue):
            after.append((pcs, retired + 1, arrived, arr))
        covers = {i: sum(o[0] == "issue" for o in done[:i]) for i, o in enumerate(done) if o[0] == "commit"}
        for i, (op, kind, j) in enumerate(done):
            if op == "commit" and i not in arrived and retired >= covers[i] and all(k in arrived for k in covers if covers[k] < covers[i]):
                after.append((pcs, retired, arrived | {i}, add(place(kind, j)[:2])))
        for i, prog in enumerate(progs):
            if pcs[i] == len(prog):
                continue
            op, kind, j = prog[pcs[i]]
            nxt = tuple(pc + (k == i) for k, pc in enumerate(pcs))
            if op == "wait":
                *b, phase = place(kind, j)
                over = count.get(tuple(b), 0) // need[kind]
                if over % 2 != phase % 2:
                    if over <= phase:
                        wrong.add(("early", kind, j))
                    after.append((nxt, retired, arrived, arr))
            elif op == "touch":
                if ("issue", "O", j) not in queue[:retired]:
                    wrong.add(("touch", j))
                after.append((nxt, retired, arrived, arr))
            else:
                after.append((nxt, retired, arrived, add(place(kind, j)[:2]) if op == "arrive" else arr))
        if not after and any(pc < len(p) for pc, p in zip(pcs, progs)):
            wrong.add(("lost", *[p[pc][1:] for pc, p in zip(pcs, progs) if pc < len(p)]))
        for s in after:
            if s not in seen:
                seen.add(s)
                stack.append(s)
    return wrong


@pytest.mark.parametrize("rescale", [False, True])
@pytest.mark.parametrize("wide", [False, True])
@pytest.mark.parametrize("ntiles", [1, 2, 3, 4, 5])
def test_commits_that_arrive_in_any_order(ntiles, wide, rescale):
    assert explore_any_order(ntiles, wide, rescale) == set()


def test_one_barrier_for_the_value_products_of_64_channels_would_be_overtaken():
    assert explore_any_order(3, False, True, two_done=False)
