"""The barriers of the kernel for clusters of SM pairs (habitat_b200/csrc/mlp_pairs.cu), as a model: every order in which
the roles of a block can run and copies and commits can land, for a block with rows of its own for what goes out.

A wait on a barrier's parity passes while the phase under way has the other parity, so a role that sleeps through two
phases waits for a third one.  No order may leave the roles waiting, and nothing may still be on its way when all have
ended: the barriers may start over then, or the shared memory go to another block."""
import pytest

SLOTS, QUARTERS = 2, 2       # of the ring; of a layer's input, each used with a slot of weights


def _roles(layers, looked_from=1, last_slots=True):
    """What each role does, in order: ("wait", barrier, phase), ("arrive", barrier), or ("later", barrier) for an arrival
    that comes when a copy has landed or the MMAs have ended.  looked_from: the first layer whose output is announced
    to the warps that look at what has come.  last_slots: the producer sees every slot freed before it ends."""
    n_layers, loads = layers + 1, 1 + layers * QUARTERS
    producer, issuer, loader, epilogue, look = [], [], [], [], []
    for n in range(loads):
        if n >= SLOTS:
            producer.append(("wait", "empty%d" % (n % SLOTS), n // SLOTS - 1))
        producer.append(("later", "full%d" % (n % SLOTS)))
    for n in range(max(loads, SLOTS), loads + SLOTS if last_slots else 0):
        producer.append(("wait", "empty%d" % (n % SLOTS), n // SLOTS - 1))
    n = 0
    for L in range(n_layers):
        for q in range(1 if L == 0 else QUARTERS):
            if L > 0:
                issuer.append(("wait", "act%d" % q, L - 1))
            issuer += [("wait", "full%d" % (n % SLOTS), n // SLOTS), ("later", "empty%d" % (n % SLOTS))]
            n += 1
        issuer.append(("later", "acc"))
        epilogue.append(("wait", "acc", L))
        if L >= looked_from:
            epilogue.append(("arrive", "out"))
            look.append(("wait", "out", L - looked_from))
        if L > 0:
            look.append(("arrive", "seen"))
        if L < layers:
            epilogue += [("later", "signal%d.%d" % (L & 1, q)) for q in range(QUARTERS)]
            loader.append(("wait", "acc", L))
            if L > 0:
                loader.append(("wait", "seen", L - 1))
            for q in range(QUARTERS):
                loader += [("wait", "signal%d.%d" % (L & 1, q), L // 2), ("later", "act%d" % q)]
    return producer, issuer, loader, epilogue, look


def _fault(roles):
    """A state from which nothing can go on although some role has not ended, or in which all have ended and an arrival is
    still to come; else None."""
    start = ((0,) * len(roles), (), ())
    seen, todo = {start}, [start]
    while todo:
        at, phases, coming = todo.pop()
        done = dict(phases)
        steps = []
        for i, ops in enumerate(roles):
            if at[i] == len(ops):
                continue
            op = ops[at[i]]
            if op[0] == "wait" and (done.get(op[1], 0) & 1) == (op[2] & 1):
                continue
            moved = at[:i] + (at[i] + 1,) + at[i + 1:]
            if op[0] == "arrive":
                steps.append((moved, {**done, op[1]: done.get(op[1], 0) + 1}, coming))
            else:
                steps.append((moved, done, tuple(sorted(coming + (op[1],))) if op[0] == "later" else coming))
        for bar in set(coming):
            left = list(coming)
            left.remove(bar)
            steps.append((at, {**done, bar: done.get(bar, 0) + 1}, tuple(left)))
        if all(a == len(ops) for a, ops in zip(at, roles)):
            if coming:
                return at, coming
        elif not steps:
            return at, ()
        for moved, done, left in steps:
            state = (moved, tuple(sorted(done.items())), left)
            if state not in seen:
                seen.add(state)
                todo.append(state)
    return None


@pytest.mark.parametrize("layers", [1, 2, 3, 4])
def test_every_order_ends_with_nothing_on_its_way(layers):
    assert _fault(_roles(layers)) is None


def test_an_announcement_that_nobody_answers_can_be_missed():
    """The output of fc1 is not announced: nothing waits for a look at it, so the next announcement could come first."""
    assert _fault(_roles(3, looked_from=0)) is not None


def test_commits_of_the_last_slots_can_come_late():
    """The last layer's MMAs have ended when its commit is there, but the commits that free its slots may come after it."""
    at, coming = _fault(_roles(2, last_slots=False))
    assert coming and all(bar.startswith("empty") for bar in coming)


@pytest.mark.parametrize("layers", range(1, 10))
@pytest.mark.parametrize("fence", ["odd layers", "none"])
def test_rows_are_ordered_before_their_place_is_read_again(layers, fence):
    """Without releases a load may find the rows of an earlier use of its place.  It must not find those of two uses ago, which
    carry the same parity: the rows of the use in between have to be ordered before it.  A fence after exchange u and
    the arrival for a later one order what was written up to u; the loader waits for the arrivals of each exchange."""
    fenced = [u for u in range(layers) if fence == "odd layers" and u % 2 == 1 and u + 2 < layers + 1]
    for u in range(layers - 2):                       # written in exchange u, the place is read again in u + 2
        ordered = any(u <= f < f + 1 <= u + 2 for f in fenced)
        assert ordered == (fence == "odd layers"), u
