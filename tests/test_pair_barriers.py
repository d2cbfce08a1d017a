"""The barriers between the roles of the tensor-core prefill kernel (csrc/prefill_tcgen05.cu), as a model of its own on the CPU: a CTA takes over one tile pair
after the other, and its two producers, the issuer and the two softmax warpgroups run on across them. Each role is a coroutine that makes the kernel's waits
and arrivals in the kernel's order; roles, copies and products are interleaved at random. A run checks that

* every wait is satisfied by the phase that it is for (a barrier keeps the parity of its phase only), and no role waits for good;
* no phase gets an arrival too many (which the hardware takes for an error while bytes are missing);
* what a product or a softmax step reads is what was meant for it;
* where a role gives up, at any point, every copy has landed when the last role has ended, and no producer's wait for its last copies is left without an end.

Mistakes planted in the model (never in the kernel) show that it finds them."""
import random

import pytest

MISTAKES = {
    "two entries of step_done": "a producer that falls behind finds the phase that it waits for gone",
    "O shares the barrier of S": "the next pair's first scores come on the phase that O's look is for",
    "counters of the next pair": "after a finished pair, the waits for the last copies look at phases of steps that never come",
    "no arrivals for the other ring": "a copy's phase lacks the arrival of the producer that gave up",
    "arrivals out of turn": "an arrival for step x while step x - 2 still lacks bytes",
    "no waits after an abort": "a copy is in flight when the CTA ends",
}


class Stuck(AssertionError):
    pass


class Bar:
    def __init__(self, arrivals):
        self.arrivals = self.pending = arrivals
        self.missing = 0       # copies that have not landed
        self.phase = 0         # phases completed

    def _turn(self):
        if self.pending == 0 and self.missing == 0:
            self.phase += 1
            self.pending = self.arrivals

    def arrive(self, copies=0):
        assert self.pending > 0, "an arrival too many"
        self.pending -= 1
        self.missing += copies
        self._turn()

    def land(self):
        self.missing -= 1
        self._turn()

    def done(self, n):   # try_wait.parity for completion number n
        return (self.phase & 1) != (n & 1)


class Cta:
    def __init__(self, pairs, seed, fault=False, mistake=None):
        assert mistake is None or mistake in MISTAKES
        self.pairs, self.rng, self.mistake, self.fault = pairs, random.Random(seed), mistake, fault
        self.n_done = 2 if mistake == "two entries of step_done" else 4
        two = lambda n: [Bar(n), Bar(n)]
        self.item_full, self.item_empty, self.q_full, self.step_full = two(1), two(4), two(1), two(2)
        self.s_full, self.o_full, self.p0, self.p1 = two(1), two(1), two(1), two(1)
        if mistake == "O shares the barrier of S":
            self.o_full = self.s_full
        self.k_first, self.answered, self.v_tail, self.drain = Bar(1), Bar(1), Bar(1), Bar(1)
        self.step_done = [Bar(1) for _ in range(self.n_done)]
        self.item, self.q, self.k, self.v, self.s, self.o = ([None, None] for _ in range(6))
        self.copies, self.products, self.written = [], [], []
        self.abort = False

    # -- what the roles are made of
    def wait(self, bar, n, tight=True):
        """False: given up. A wait that could run out may do so whenever a fault is wanted."""
        while not bar.done(n):
            if self.abort:
                return False
            if self.fault and self.rng.random() < self.give_up:
                self.abort = True
                return False
            yield
        assert self.abort or not tight or bar.phase == n + 1, ("another phase", n, bar.phase)
        return True

    def copy(self, bar, landed=lambda: None):
        bar.arrive(copies=1)
        self.copies.append((bar, landed))

    def last_copies(self, alive, given, others, left_out=0):
        """The end of a producer: where somebody has given up, its last copies, and the arrivals that the other ring's producer may wait for."""
        if alive:
            alive = yield from self.wait(self.drain, 0)
        if alive and not self.abort or self.mistake == "no waits after an abort":
            return
        for bar, n in others:
            while not bar.done(n):
                yield
        for x in ([left_out - 1] if left_out > 0 else []) + [given, given + 1]:
            while x >= 2 and not self.step_full[x & 1].done((x - 2) >> 1) and self.mistake != "arrivals out of turn":
                yield
            if self.mistake != "no arrivals for the other ring":
                self.step_full[x & 1].arrive()
            yield

    # -- roles
    def k_producer(self):
        g = commits = given = firsts = requests = answers = 0
        free, used, scores, loads = [-1, -1], [False, False], [0, 0], [0, 0]
        first_s, owed, alive, left_out = -1, False, True, 0
        freed = lambda c: self.wait(self.step_done[c % self.n_done], c // self.n_done)
        for it in range(len(self.pairs) + 1):
            e = it & 1
            if owed:
                c = free[g & 1]
                if c < 0 or self.step_done[c % self.n_done].done(c // self.n_done):
                    self.step_full[(g - 1) & 1].arrive()
                    given, owed = g, False
            yield
            if it > 0:
                if requests == answers:
                    self.copy(self.answered)
                    requests += 1
                if it >= 2:
                    alive = yield from self.wait(self.item_empty[e], (it >> 1) - 1)
                if alive:
                    alive = yield from self.wait(self.answered, answers)
                if not alive:
                    break
                answers += 1
            n = (0, 0) if it == len(self.pairs) else self.pairs[it]
            self.item[e] = n if it < len(self.pairs) else "end"
            self.item_full[e].arrive()
            yield
            if owed:
                if free[g & 1] >= 0:
                    alive = yield from freed(free[g & 1])
                if not alive:
                    break
                self.step_full[(g - 1) & 1].arrive()
                given, owed = g, False
            if it == len(self.pairs):
                break
            steps = max(n)
            if steps == 0:
                self.copy(self.answered)
                requests += 1
                continue
            if first_s >= 0:
                alive = yield from freed(first_s)
            for j in range(steps):
                s = (g + j) & 1
                if alive and free[s] >= 0:
                    alive = yield from freed(free[s])
                if not alive:
                    break

                def land(s=s, it=it, j=j):
                    self.k[s] = (it, j)
                skip = self.fault and left_out == 0 and self.rng.random() < self.give_up   # (the test hook)
                if skip:
                    left_out = g + j if j > 0 else 0
                else:
                    self.copy(self.k_first if j == 0 else self.step_full[s ^ 1], land)
                free[s] = commits + j
                if j == 0:
                    firsts += not skip
                    for t in (1, 0):
                        yield
                        if used[t] and alive:
                            alive = yield from self.wait(self.s_full[t], scores[t] - 1)
                        if n[t] > 0 and alive:
                            def land_q(t=t, it=it):
                                self.q[t] = it
                            self.copy(self.q_full[t], land_q)
                            loads[t] += 1
                else:
                    given = g + j
                yield
                if not alive:
                    break
            if not alive:
                break
            owed = True
            first_s = commits if steps == 1 else -1
            for t in (0, 1):
                used[t] = n[t] > 0
                scores[t] += n[t]
            commits, g = commits + steps + 1, g + steps
            last_steps = steps
        if self.mistake == "counters of the next pair" and not alive and commits:
            given = g + last_steps - 1
        others = [(self.answered, answers)] if answers != requests else []
        others += [(self.q_full[t], loads[t] - 1) for t in (0, 1) if loads[t]] + ([(self.k_first, firsts - 1)] if firsts else [])
        yield from self.last_copies(alive, given, others, left_out)

    def v_producer(self):
        g = commits = given = tails = it = 0
        free, alive, pending = [-1, -1], True, False
        while alive:
            alive = yield from self.wait(self.item_full[it & 1], it >> 1)
            if not alive:
                break
            n = self.item[it & 1]
            self.item_empty[it & 1].arrive()
            if n == "end":
                break
            steps = max(n)
            tail = self.rng.random() < 0.5
            for j in range(steps):
                s = (g + j) & 1
                if free[s] >= 0:
                    alive = yield from self.wait(self.step_done[free[s] % self.n_done], free[s] // self.n_done)
                if not alive:
                    break

                def land(s=s, it=it, j=j):
                    self.v[s] = (it, j)
                fix = tail and j == steps - 1
                self.copy(self.v_tail if fix else self.step_full[s], land)
                free[s] = commits + j + 1
                yield
                if fix:
                    pending = True
                    alive = yield from self.wait(self.v_tail, tails)
                    if not alive:
                        break
                    pending = False
                    tails += 1
                    self.step_full[s].arrive()
                given = g + j + 1
            if steps and alive:
                commits, g = commits + steps + 1, g + steps
            it += 1
        yield from self.last_copies(alive, given, [(self.v_tail, tails)] if pending else [])

    def issuer(self):
        yield from self.issue()
        self.products.append(self.drain.arrive)

    def issue(self):
        g = done = firsts = it = 0
        loads, steps = [0, 0], [0, 0]

        def product(check):
            self.products.append(lambda: self.abort or check())

        def commit(bar):
            self.products.append(bar.arrive)

        def scores(t, item, j, s):
            def check():
                assert self.q[t] == item and self.k[s] == (item, j), (self.q, self.k, item, j)
                assert self.s[t] is None or self.s[t][0] == "used", self.s[t]
                self.s[t] = ("s", item, j)
            product(check)

        def values(t, item, j, s, last):
            def check():
                assert self.v[s] == (item, j) and self.s[t] == ("p", item, j), (self.v, self.s, item, j)
                if last:
                    self.o[t], self.s[t] = (item, j), ("used",)
            product(check)

        while True:
            if not (yield from self.wait(self.item_full[it & 1], it >> 1)):
                return
            n = self.item[it & 1]
            self.item_empty[it & 1].arrive()
            if n == "end":
                return
            if max(n) > 0:
                for t in (0, 1):
                    if n[t] <= 0:
                        continue
                    for bar, x in ((self.q_full[t], loads[t]), (self.k_first, firsts)):
                        if not (yield from self.wait(bar, x)):
                            return
                    loads[t] += 1
                    scores(t, it, 0, g & 1)
                    commit(self.s_full[t])
                    yield
                firsts += 1
                commit(self.step_done[done % self.n_done])
                done += 1
            for j in range(max(n)):
                s = g & 1
                if not (yield from self.wait(self.step_full[s], g >> 1)):
                    return
                for t in (0, 1):
                    if j >= n[t]:
                        continue
                    for half, bar in enumerate((self.p0[t], self.p1[t])):
                        if not (yield from self.wait(bar, steps[t])):
                            return
                        values(t, it, j, s, half == 1)
                        yield
                    steps[t] += 1
                    if j + 1 < n[t]:
                        scores(t, it, j + 1, s ^ 1)
                    commit(self.s_full[t] if j + 1 < n[t] else self.o_full[t])
                    yield
                commit(self.step_done[done % self.n_done])
                done += 1
                g += 1
            it += 1

    def softmax(self, t):
        steps = tiles = it = 0
        while True:
            if not (yield from self.wait(self.item_full[it & 1], it >> 1)):
                return
            n = self.item[it & 1]
            yield
            self.item_empty[it & 1].arrive()
            if n == "end":
                return
            for j in range(n[t]):
                if not (yield from self.wait(self.s_full[t], steps)):
                    return
                steps += 1
                assert self.abort or self.s[t] == ("s", it, j), (self.s[t], it, j)
                yield
                self.s[t] = ("p", it, j)
                self.p0[t].arrive()
                yield
                self.p1[t].arrive()
                yield
            if n[t] > 0:
                x = steps if self.mistake == "O shares the barrier of S" else tiles
                if not (yield from self.wait(self.o_full[t], x)):
                    return
                tiles += 1
                steps += self.mistake == "O shares the barrier of S"
                for _ in range(self.rng.randint(0, 6)):   # the epilogue
                    yield
                assert self.abort or self.o[t] == (it, n[t] - 1)
                self.written.append((it, t))
            it += 1

    def run(self):
        r = self.rng
        self.give_up = r.choice([0.02, 0.005, 0.001])
        roles = [self.k_producer(), self.v_producer(), self.issuer(), self.softmax(0), self.softmax(1)]
        # 4 arrivals on item_empty: V producer, issuer, two softmax warpgroups
        speed = [r.choice([1, 1, 3, 10]) for _ in roles]
        landing, computing = r.choice([1, 1, 5, 20]), r.choice([1, 1, 5, 20])
        turns = 0
        while roles:
            turns += 1
            if turns > 100_000:
                raise Stuck(f"{len(roles)} roles wait for good, {len(self.copies)} copies in flight")
            what = r.choices(range(len(roles) + 2), speed + [landing * bool(self.copies), computing * bool(self.products)])[0]
            if what < len(roles):
                try:
                    next(roles[what])
                except StopIteration:
                    roles.pop(what)
                    speed.pop(what)
            elif what == len(roles):
                bar, landed = self.copies.pop(r.randrange(len(self.copies)))
                landed()
                bar.land()
            else:
                self.products.pop(0)()
        assert not self.copies, "copies in flight at the end of the CTA"
        if not self.abort:
            assert sorted(self.written) == [(i, t) for i, n in enumerate(self.pairs) for t in (0, 1) if n[t] > 0]


def _pairs(seed):
    r = random.Random(1000 + seed)
    most, least = r.choice([1, 2, 3, 6]), r.choice([0, 1, 1])
    pairs = []
    for _ in range(r.randint(1, 9)):
        a = r.randint(least, most)
        pairs.append((a, r.choice([a, a, max(0, a - 1), 0])))
    return pairs


def _run(seed, **how):
    Cta(_pairs(seed), seed, **how).run()


@pytest.mark.parametrize("fault", [False, True])
def test_every_wait_ends_with_its_own_phase_and_no_copy_is_left(fault):
    for seed in range(1500):
        _run(seed, fault=fault)


@pytest.mark.parametrize("mistake", MISTAKES)
def test_the_model_finds_a_planted_mistake(mistake):
    # mistakes at the end of the producers show where a role gives up
    fault = mistake not in ("two entries of step_done", "O shares the barrier of S")
    found = 0
    for seed in range(1500):
        try:
            _run(seed, fault=fault, mistake=mistake)
        except AssertionError:
            found += 1
            if found == 3:
                return
    raise AssertionError(f"{mistake}: {MISTAKES[mistake]}: found {found} times")
