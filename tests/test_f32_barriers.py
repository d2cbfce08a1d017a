"""The barriers between the warps of the f32 kernel on the tensor cores (csrc/tile_f32_tcgen05.cu), as a model on the CPU: worker warps (three quads of rows, two parts of
keys and columns; the first two also write a tile's mask) and the issuer are coroutines that make the kernel's waits, arrivals and accesses in the kernel's order, and
they and the products are interleaved at random. A product reads its operands at its begin and at its end; products into one sum end in the order in which
they were issued, others in any. Checked: every wait is satisfied by the phase that it is for, no role waits for good, also where a wait runs out, and whatever is read, in shared memory and in tensor
memory, is what was meant for that tile. How many buffers there are is read from the source; mistakes planted in the model show that it finds them."""
import random
import re
from pathlib import Path

import pytest

SOURCE = (Path(__file__).resolve().parent.parent / "luma_b200" / "csrc" / "tile_f32_tcgen05.cu").read_text()
QUADS, PARTS = 3, 2
WARPS = QUADS * PARTS
WRITERS = 2
WAITS_FOR_O = "wait(o_full, phase, 65)" in SOURCE
MISTAKES = {
    "one buffer for the maxima": "a warp of the quad runs on and writes the next tile's maximum where another has not read this one's",
    "two buffers for the mask": "the warps that bring the next tile's mask are behind what others did two tiles ago only",
    "scores without a wait for O": "at head size 128 the third sum of the scores lies over the weights, whose product may still run",
    "a tile's K before its scores are there": "the planes are written again under the product that reads them",
}


def _buffers(name):
    found = re.search(rf"constexpr int {name} = (\d+);", SOURCE)
    return int(found.group(1)) if found else 1


class Bar:
    def __init__(self, arrivals):
        self.arrivals = self.pending = arrivals
        self.phase = 0

    def arrive(self):
        self.pending -= 1
        if self.pending == 0:
            self.phase += 1
            self.pending = self.arrivals

    def done(self, n):   # try_wait.parity for completion number n
        return (self.phase & 1) != (n & 1)


class Cta:
    def __init__(self, n, over, seed, fault=False, mistake=None):
        assert mistake is None or mistake in MISTAKES
        self.n, self.over, self.fault, self.mistake, self.rng = n, over, fault, mistake, random.Random(seed)
        self.reds = 1 if mistake == "one buffer for the maxima" else _buffers("kMaxBuffers")
        self.s_full, self.o_full = Bar(1), Bar(1)
        self.k_ready, self.s_free, self.pv_ready = Bar(WARPS), Bar(WARPS), Bar(WARPS)
        self.quad_at = [0] * WARPS                       # barriers of its quad that a warp has come to
        self.k, self.v = [None] * WARPS, [None] * WARPS  # the tile whose rows a warp has laid down
        self.red = [[[None] * PARTS for _ in range(QUADS)] for _ in range(self.reds)]
        self.masks = 2 if mistake == "two buffers for the mask" else _buffers("kMaskBuffers")
        self.vis = [[None] * WRITERS for _ in range(self.masks)]
        self.s = [None, None]                            # the tile of the scores in tensor memory: first sums and third
        self.s_read = [None] * WARPS
        self.p = [None] * WARPS                          # weights
        self.o, self.o_read = None, [None] * WARPS
        self.products = []                               # [where to, check at begin and end, what it writes, begun], and commits
        self.abort = False

    def check(self, what, *say):
        assert self.abort or what, say

    def wait(self, bar, n):
        while not bar.done(n):
            if self.abort:
                return False
            if self.fault and self.rng.random() < 0.002:
                self.abort = True
                return False
            yield
        self.check(bar.phase == n + 1, "another phase", n, bar.phase)
        return True

    # -- products
    def product(self, to, reads, writes):
        self.products.append([to, reads, writes, False])

    def first_scores(self, j):
        def reads():
            self.check(all(x == j for x in self.k), "K", j, self.k)
            self.check(all(x == j - 1 for x in self.s_read) or j == 0, "scores over scores that have not been read", j, self.s_read)

        def writes():
            self.s[0] = j
        self.product("first scores", reads, writes)

    def small_scores(self, j):
        def reads():
            self.check(all(x == j for x in self.k), "K", j, self.k)
            self.check(all(x == j - 1 for x in self.s_read) or j == 0, "scores over scores that have not been read", j, self.s_read)
            self.check(not self.over or j == 0 or self.o == j - 1, "scores over weights that are still in use", j, self.o)

        def writes():
            self.s[1] = j
        self.product("small scores", reads, writes)
        self.products.append(self.s_full)

    def sums(self, j):
        def reads():
            self.check(all(x == j for x in self.v) and all(x == j for x in self.p), "V, P", j, self.v, self.p)
            self.check(all(x == j - 1 for x in self.o_read) or j == 0, "O over O that has not been read", j, self.o_read)

        def writes():
            self.o = j
        self.product("O", reads, writes)
        self.products.append(self.o_full)

    def compute(self):
        """A product begins or ends, or a commit behind products that have all ended arrives."""
        items = self.products
        if not isinstance(items[0], list):
            items.pop(0).arrive()
            return
        able, places = [], set()
        for i, x in enumerate(items):
            if isinstance(x, list) and x[0] not in places:
                places.add(x[0])
                able.append(i)
        i = self.rng.choice(able)
        _, reads, writes, begun = items[i]
        reads()
        if begun:
            writes()
            items.pop(i)
        else:
            items[i][3] = True

    # -- roles
    def issuer(self):
        if not (yield from self.wait(self.k_ready, 0)):
            return
        self.first_scores(0)
        self.small_scores(0)
        for j in range(self.n):
            more = j + 1 < self.n
            if not self.over and more:
                for bar, x in ((self.k_ready, j + 1), (self.s_free, j)):
                    if not (yield from self.wait(bar, x)):
                        return
                self.first_scores(j + 1)
                yield
                self.small_scores(j + 1)
                yield
            if not (yield from self.wait(self.pv_ready, j)):
                return
            self.sums(j)
            yield
            if self.over and more:
                if not (yield from self.wait(self.k_ready, j + 1)):
                    return
                self.first_scores(j + 1)
                yield
                if WAITS_FOR_O and self.mistake != "scores without a wait for O" and not (yield from self.wait(self.o_full, j)):
                    return
                self.small_scores(j + 1)
                yield

    def quad_barrier(self, w):
        self.quad_at[w] += 1
        while min(self.quad_at[w % QUADS::QUADS]) < self.quad_at[w]:
            yield

    def worker(self, w):
        quad, part = w % QUADS, w // QUADS
        self.k[w] = 0
        if w < WRITERS:
            self.vis[0][w] = 0
        yield
        self.k_ready.arrive()
        for j in range(self.n):
            if self.mistake == "a tile's K before its scores are there" and j + 1 < self.n:
                self.k[w] = j + 1
            yield from self.wait(self.s_full, j)
            self.check(self.s == [j, j], "scores", j, self.s)
            yield
            self.check(self.s == [j, j], "scores", j, self.s)
            self.s_read[w] = j
            if not self.over:
                self.s_free.arrive()
            yield
            if j + 1 < self.n:
                if w < WRITERS:
                    self.vis[(j + 1) % self.masks][w] = j + 1
                self.k[w] = j + 1
                yield
                self.k_ready.arrive()
            yield
            self.check(self.vis[j % self.masks] == [j] * WRITERS, "mask", j, self.vis)
            yield
            self.check(self.vis[j % self.masks] == [j] * WRITERS, "mask", j, self.vis)
            red = self.red[j % self.reds][quad]
            red[part] = j
            yield from self.quad_barrier(w)
            for x in range(PARTS):
                yield
                self.check(red[x] == j, "maxima", j, red)
            if j > 0:
                yield from self.wait(self.o_full, j - 1)
                self.check(self.o == j - 1, "O", j, self.o)
                yield
                self.o_read[w] = j - 1
            self.v[w] = j
            yield
            self.check(not self.over or all(x == j for x in self.s_read[quad::QUADS]), "weights over scores", j)
            self.p[w] = j
            yield
            self.pv_ready.arrive()
        yield from self.wait(self.o_full, self.n - 1)
        self.check(self.o == self.n - 1, "O", self.n - 1, self.o)
        self.o_read[w] = self.n - 1
        yield from self.quad_barrier(w)

    def run(self):
        roles = [self.worker(w) for w in range(WARPS)] + [self.issuer()]
        speed = [self.rng.choice([1, 1, 5, 30]) for _ in roles]
        computing = self.rng.choice([1, 5, 30])
        turns = 0
        while roles:
            turns += 1
            assert turns < 200_000, f"{len(roles)} roles wait for good"
            i = self.rng.choices(range(len(roles) + 1), speed + [computing * bool(self.products)])[0]
            if i == len(roles):
                self.compute()
                continue
            try:
                next(roles[i])
            except StopIteration:
                roles.pop(i)
                speed.pop(i)
        assert self.abort or self.o_read == [self.n - 1] * WARPS


@pytest.mark.parametrize("fault", [False, True])
@pytest.mark.parametrize("over", [False, True])
def test_every_tile_is_read_as_it_was_written(over, fault):
    for seed in range(400):
        Cta(1 + seed % 7, over, seed, fault).run()


@pytest.mark.parametrize("mistake", MISTAKES)
def test_the_model_finds_a_planted_mistake(mistake):
    found = 0
    for seed in range(1500):
        try:
            Cta(5, mistake == "scores without a wait for O", seed, mistake=mistake).run()
        except AssertionError:
            found += 1
            if found == 3:
                return
    raise AssertionError(f"{mistake}: {MISTAKES[mistake]}: found {found} times")


def test_weights_over_scores_are_stored_behind_a_fence():
    """At head size 128 a warp's weights go over the scores that the other warps of its rows have loaded: loads, tcgen05.fence::before_thread_sync, barrier,
    tcgen05.fence::after_thread_sync, stores, in the first tile as well (the later ones have the fence of their wait for O besides)."""
    loop = SOURCE[SOURCE.index("wait_warp(s_full, phase, 70);"):SOURCE.index("tell(pv_ready);")]
    at = [loop.index(x) for x in ("tc_ld16(mine + part * kKeys, sc);", "tc_fence_before();", "barrier.cta.sync %0, 128;", "if (S::kOver) tc_fence_after();", "if (j > 0) {", "tc_st8(")]
    assert at == sorted(at)


@pytest.mark.parametrize("d", [32, 64, 128])
def test_products_that_share_columns_have_the_same_accumulator_and_shape(d):
    """The order of issue is promised for products of one accumulator and shape only. From the source: first column and columns of every product, for each head size."""
    plan = SOURCE[SOURCE.index("struct Plan {"):]
    plan = plan[:plan.index("};")]
    env = dict(D=d, kN=64, kM=128, tmem=0)
    for name, value in re.findall(r"(k[A-Z]\w*) = ([^,;]+)[,;]", plan):
        value = re.sub(r"(.+) \? (.+) : (.+)", r"(\2) if (\1) else (\3)", value.replace("/", "//"))
        if name in ("kHalves", "kCols", "kOver", "kP", "kO", "kOrders"):
            env[name] = eval(value, {}, env)
    found = 0
    for function in ("issue_scores", "issue_sums"):
        body = SOURCE[SOURCE.index(f"__noinline__ void {function}("):]
        body = body[:body.index("__syncwarp();")].replace("S::", "")
        places = dict(re.findall(r"(\w+) = (tmem[^,;]*)[,;]", body))
        shapes = set()
        for to, columns in re.findall(r"tc_mma_[st]s\((\w+), .*?make_idesc<__nv_bfloat16>\(\w+, ([^)]*)\)", body):
            shapes.add((eval(places[to], {}, env), eval(columns, {}, env)))
            found += 1
        shapes = sorted(shapes)
        assert all(a + n <= b for (a, n), (b, _) in zip(shapes, shapes[1:])), (function, shapes)
        assert all(a + n <= 512 for a, n in shapes)
    if d == 128:   # the weights over the third sum alone, and not over O
        assert 2 * 64 <= env["kP"] and env["kP"] + 3 * 64 // 2 <= env["kO"]
    assert found == 8
