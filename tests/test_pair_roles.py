"""A CPU model of pair_main's waits (csrc/aodmao2rho_split_pair.cu): twelve gather
warps in three groups that run on over the ends of items, eight epilogue warps, the MMA
issuer, the phi loader and the item drawer as generators over mbarriers, under random
schedules.  A wait of parity P passes when the barrier's current phase has the other
parity; the model asserts that this is always the same as the wanted phase being
complete (no aliasing), that ring slots and stages hold what their readers expect, and
that every role ends."""
import random

import pytest

NG, STAGES, RING, AHEAD, EPI = 3, 3, 4, 2, 8


class Bar:
    def __init__(self, n):
        self.n, self.count, self.phase = n, 0, 0

    def arrive(self):
        self.count += 1
        assert self.count <= self.n
        if self.count == self.n:
            self.count, self.phase = 0, self.phase + 1

    def passes(self, want):  # a wait for the end of phase `want`, by its parity
        ok = (self.phase & 1) != (want & 1)
        assert ok == (self.phase > want), "a parity named another phase"
        return ok


def run(items, seed):
    rnd = random.Random(seed)
    full_phi, empty = [Bar(1) for _ in range(STAGES)], [Bar(1) for _ in range(STAGES)]
    full_d = [Bar(4) for _ in range(STAGES)]
    acc_full, acc_empty = Bar(1), Bar(EPI)
    started, ifull = [Bar(1) for _ in range(RING)], [Bar(1) for _ in range(RING)]
    iempty = [Bar(4 * NG + EPI + 2) for _ in range(RING)]
    ring, phi, d = [None] * RING, [None] * STAGES, [set() for _ in range(STAGES)]

    def wait(bar, want):
        while not bar.passes(want):
            yield

    def item(n):
        yield from wait(ifull[n % RING], n // RING)
        number, chunks = ring[n % RING]
        assert number == n
        iempty[n % RING].arrive()
        return chunks

    def gather(group, warp):
        state = dict(base=0, nch=0, n=0, more=True)

        def advance(q):
            while q >= state["base"] + state["nch"]:
                state["base"] += state["nch"]
                chunks = yield from item(state["n"])
                state["n"] += 1
                if chunks is None:
                    state["more"] = False
                    return
                state["nch"] = chunks

        q = group
        yield from advance(q)
        live = state["more"]
        if live:
            yield from advance(q + NG)
        while live:
            s = q % STAGES
            if q >= STAGES:
                yield from wait(empty[s], q // STAGES - 1)
            live = state["more"]
            yield
            d[s].add((q, warp))
            full_d[s].arrive()
            q += NG
            if live:
                yield from advance(q + NG)

    def epilogue():
        n = 0
        while (yield from item(n)) is not None:
            yield from wait(acc_full, n)
            yield
            acc_empty.arrive()
            n += 1

    def mma():
        n = seq = 0
        while True:
            chunks = yield from item(n)
            if chunks is None:
                return
            if n > 0:
                yield from wait(acc_empty, n - 1)
            for _ in range(chunks):
                s = seq % STAGES
                yield from wait(full_phi[s], seq // STAGES)
                yield from wait(full_d[s], seq // STAGES)
                assert phi[s] == seq and d[s] == {(seq, w) for w in range(4)}
                yield
                d[s] = set()
                empty[s].arrive()
                seq += 1
            acc_full.arrive()
            n += 1

    def load():
        n = seq = 0
        while True:
            chunks = yield from item(n)
            if chunks is None:
                return
            started[n % RING].arrive()
            for _ in range(chunks):
                s = seq % STAGES
                if seq >= STAGES:
                    yield from wait(empty[s], seq // STAGES - 1)
                yield
                phi[s] = seq
                full_phi[s].arrive()
                seq += 1
            n += 1

    def draw():
        n = 0
        while True:
            if n >= AHEAD:
                yield from wait(started[(n - AHEAD) % RING], (n - AHEAD) // RING)
            if n >= RING:
                yield from wait(iempty[n % RING], n // RING - 1)
            chunks = items[n] if n < len(items) else None
            ring[n % RING] = (n, chunks)
            ifull[n % RING].arrive()
            if chunks is None:
                return
            n += 1

    roles = [gather(w // 4, w % 4) for w in range(4 * NG)] + [epilogue() for _ in range(EPI)]
    roles += [mma(), load(), draw()]
    speed = [rnd.choice([1, 1, 5, 30]) for _ in roles]
    live, steps = list(range(len(roles))), 0
    while live:
        i = rnd.choices(live, [speed[j] for j in live])[0]
        try:
            next(roles[i])
        except StopIteration:
            live.remove(i)
        steps += 1
        assert steps < 4000 * (sum(items) + 10), "stuck"


@pytest.mark.parametrize("most", [1, 3, 14])  # chunks of an item
def test_every_role_ends(most):
    for seed in range(40):
        rnd = random.Random(seed)
        run([rnd.randint(1, most) for _ in range(rnd.randint(0, 20))], seed)
