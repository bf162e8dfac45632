"""CPU model of the attention kernel's pipeline (full tiles): its warps as generators that wait on barriers and arrive on them, in the order of
the kernel's loops.  A list of units that stops the model would make the kernel's bounded waits give up.  What it shows: V may be loaded two blocks
behind K as long as all of it is loaded before the producer publishes a unit without keys, or the end."""
import random

import pytest

RING = 4                                           # unit descriptors


class Bar:
    """An mbarrier: a phase completes at `count` arrivals; a wait for parity p passes once a phase of parity p is the last completed one."""
    def __init__(self, count):
        self.count, self.got, self.phase = count, 0, 0

    def arrive(self):
        self.got += 1
        if self.got == self.count:
            self.got, self.phase = 0, self.phase + 1


class Ring:
    """A place in a ring of stages, with the parity that goes with it."""
    def __init__(self, n, parity):
        self.n, self.i, self.parity = n, 0, parity

    def step(self):
        self.i += 1
        if self.i == self.n:
            self.i, self.parity = 0, self.parity ^ 1


def ends(units, lag, drain, stages=4):
    """units: (key blocks of tile 0, of tile 1, tiles).  lag: blocks V is loaded behind K; drain: pending V is loaded before a unit without keys
    and the end are published.  True when every warp gets to its end."""
    def bars(n, count=1):
        return [Bar(count) for _ in range(n)]
    q_full, q_free, k_full, k_free, v_full, v_free = bars(2), bars(2, 2), bars(stages), bars(stages, 2), bars(stages), bars(stages)
    s_full, s_free, maxima, p_full, pv_done, o_scaled = bars(8), [bars(2), bars(1)], bars(8), bars(8), bars(8), bars(8)
    published, finished = bars(RING), bars(RING, 8)
    ring = [None] * RING

    def until(bar, parity):
        while bar.phase & 1 == parity:
            yield

    def producer():
        k_at, v_at, pending, nq = Ring(stages, 1), Ring(stages, 1), 0, 0

        def load_v():
            yield from until(v_free[v_at.i], v_at.parity)
            v_full[v_at.i].arrive()
            v_at.step()
        for k, u in enumerate(units + [None]):
            if drain and (u is None or u[0] + u[1] == 0):
                for _ in range(pending):
                    yield from load_v()
                pending = 0
            yield from until(finished[k % RING], k // RING & 1 ^ 1)
            ring[k % RING] = u
            published[k % RING].arrive()
            if u is None:
                for _ in range(pending):
                    yield from load_v()
                return
            if u[0] + u[1] == 0:
                continue
            yield from until(q_free[nq & 1], nq >> 1 & 1 ^ 1)
            q_full[nq & 1].arrive()
            nq += 1
            for _ in range(max(u[0], u[1])):
                yield from until(k_free[k_at.i], k_at.parity)
                k_full[k_at.i].arrive()
                if pending == lag:
                    yield from load_v()
                else:
                    pending += 1
                k_at.step()

    def walk(body, early):
        """A consumer: unit after unit; `early`: it lets go of the descriptor before it works on the unit."""
        base, i = 0, 0
        while True:
            yield from until(published[i % RING], i // RING & 1)
            u = ring[i % RING]
            if u is None:
                return
            two = 1 if u[2] == 2 else 0
            if early:
                finished[i % RING].arrive()
            yield from body(u, base, u[0] + u[1], two, u[1] - u[0] if two else 0)
            if not early:
                finished[i % RING].arrive()
            base, i = base + u[0] + u[1], i + 1

    def scores(half):
        k_at, buf, units_seen = Ring(stages, 0), Ring(2 - half, 1), [0]

        def body(u, base, ns, two, d):
            if ns == 0:
                return
            n = units_seen[0]
            yield from until(q_full[n & 1], n >> 1 & 1)
            for s in range(ns):
                t = s + d & two
                if t == 0 or s == 0:
                    yield from until(k_full[k_at.i], k_at.parity)
                yield from until(s_free[half][buf.i], buf.parity)
                s_full[2 * (base + s & 3) + half].arrive()
                if s == ns - 1:
                    q_free[n & 1].arrive()
                buf.step()
                if t == two:
                    k_free[k_at.i].arrive()
                    k_at.step()
            units_seen[0] += 1
        return walk(body, True)

    def products():
        v_at = Ring(stages, 0)

        def body(u, base, ns, two, d):
            for s in range(ns):
                t, sg = s + d & two, base + s
                if t == 0 or s == 0:
                    yield from until(v_full[v_at.i], v_at.parity)
                yield from until(o_scaled[sg & 7], sg >> 3 & 1)
                pv_done[sg & 7].arrive()
                if t == two:
                    v_free[v_at.i].arrive()
                    v_at.step()
        return walk(body, True)

    def softmax(group):
        def body(u, base, ns, two, d):
            for sg in range(base + (group - base) % 4, base + ns, 4):
                if sg >= 6:
                    yield from until(pv_done[sg - 6 & 7], sg - 6 >> 3 & 1)
                for half in (0, 1):
                    yield from until(s_full[2 * group + half], sg >> 2 & 1)
                    s_free[half][sg % (2 - half)].arrive()
                if sg - base > two:
                    yield from until(maxima[sg - 1 - two & 7], sg - 1 - two >> 3 & 1)
                maxima[sg & 7].arrive()
                p_full[sg & 7].arrive()
        return walk(body, False)

    def rescale():
        def body(u, base, ns, two, d):
            for sg in range(base, base + ns):
                yield from until(p_full[sg & 7], sg >> 3 & 1)
                if sg - base > two:
                    yield from until(pv_done[sg - 1 - two & 7], sg - 1 - two >> 3 & 1)
                o_scaled[sg & 7].arrive()
            for t in range(u[2]):
                if u[t]:
                    last = base + (2 * (max(u[0], u[1]) - 1) + t - d if two else u[t] - 1)
                    yield from until(pv_done[last & 7], last >> 3 & 1)
        return walk(body, False)

    every = [b for g in (q_full, q_free, k_full, k_free, v_full, v_free, s_full, *s_free, maxima, p_full, pv_done, o_scaled, published, finished) for b in g]
    running, before = [producer(), scores(0), scores(1), products(), rescale(), *(softmax(g) for g in range(4))], None
    while running:
        now = (len(running), [(b.phase, b.got) for b in every])
        if now == before:
            return False
        before, still = now, []
        for w in running:
            for _ in range(32):
                if next(w, "end") == "end":
                    break
            else:
                still.append(w)
        running = still
    return True


EMPTY, ONE, PAIR = (0, 0, 2), (1, 0, 1), (5, 6, 2)


@pytest.mark.parametrize("units", [[PAIR, EMPTY, EMPTY, EMPTY], [ONE, EMPTY, ONE, EMPTY, ONE], [PAIR, PAIR] + 6 * [EMPTY]])
def test_units_without_keys_stop_a_producer_that_holds_v_back(units):
    assert ends(units, 0, False) and ends(units, 2, True)
    assert not ends(units, 2, False)


@pytest.mark.parametrize("stages", [4, 5])
def test_no_list_of_units_stops_the_pipeline(stages):
    r = random.Random(stages)

    def unit():
        if r.random() < 0.45:
            return (0, 0, r.choice((1, 2)))
        a = r.choice((0, 1, 1, 2, 5, 9))
        return (max(a, 1), 0, 1) if r.random() < 0.5 else (a, max(a, 1) if r.random() < 0.5 else a + 1, 2)
    for _ in range(300):
        units = [unit() for _ in range(r.randint(1, 14))]
        assert ends(units, 2, True, stages), units
