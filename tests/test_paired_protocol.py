"""The barriers of the paired kernel (csrc/paired_heads.cu) as a model: every warp role and every asynchronous unit (copies, MMAs with
their commits) is a process of its own that may be held back for as long as the others can run.  The model keeps what each buffer
holds, so it finds a wait that misses its phase (deadlock), one that passes too early or a buffer that is overwritten too soon
(wrong content), and an arrival too many.  Ring sizes and whether the score issuers share barriers are read from the kernel's source."""
import os
import random
import re
from collections import deque

import pytest

SRC = open(os.path.join(os.path.dirname(__file__), "..", "opfoundry_b200", "csrc", "paired_heads.cu")).read()


def _const(name):
    return int(re.search(r"constexpr int (?:[^;]*, )?%s = (\d+)" % name, SRC).group(1))


STAGES, Q_STAGES, MAX_RING = _const("kStages"), _const("kQStages"), _const("kMaxRing")
# a score issuer has the landing barriers of its own tiles to itself (else it has to look at those of the other's tiles too)
OWN_BARRIERS = "uint64_t tile_ready[2][kStages]" in SRC


class Bar:
    def __init__(self, count):
        self.count = self.pending = count
        self.phase = self.tx = 0

    def _check(self):
        assert self.pending >= 0, "an arrival too many"
        if self.pending == 0 and self.tx == 0:
            self.phase, self.pending = self.phase + 1, self.count

    def arrive(self, n=1):
        self.pending -= n
        self._check()

    def landed(self, n=1):
        self.tx -= n
        self._check()

    def passes(self, parity):
        return (self.phase & 1) != parity


class Ring:
    def __init__(self, bits=0):
        self.s, self.bits = 0, bits

    def ph(self):
        return (self.bits >> self.s) & 1

    def skip(self, n):
        self.s = (self.s + n) % STAGES

    def next(self):
        self.bits ^= 1 << self.s
        self.skip(1)


class Pair:
    """A pair of CTAs over `items` (tiles of each item).  A process yields (barrier, parity) to wait or None between two steps."""

    def __init__(self, items, own_barriers, rng):
        self.items, self.own_barriers, self.rng = items, own_barriers, rng
        bars = lambda n, count: [[Bar(count) for _ in range(n)] for _ in range(2)]
        self.kv_full, self.kv_empty, self.peer_late, self.dead, self.late_full = bars(STAGES, 8 * 33), bars(STAGES, 1), bars(STAGES, 1), bars(STAGES, 1), bars(STAGES, 4 * 32)
        self.tile_ready = bars(STAGES, 2)   # CTA 0's, by the issuer that takes the tile
        if not own_barriers:
            self.tile_ready[1] = self.tile_ready[0]
        self.s_full, self.s_empty, self.p_full, self.pv_done = bars(2, 1), bars(2, 8), bars(2, 8), bars(2, 1)
        self.m_bar = [[[Bar(2) for _ in range(2)] for _ in range(MAX_RING)] for _ in range(2)]
        self.q_stage = bars(2, 8)
        one = lambda count: [Bar(count) for _ in range(2)]
        self.q_smem, self.q_copied, self.q_full, self.q_empty, self.o_full, self.o_free, self.e_bar, self.l_free = (
            one(1), one(4), one(8), one(2), one(1), one(8), one(8), one(4))
        # what the buffers hold
        self.keep = [[[None] * 8 for _ in range(STAGES)] for _ in range(2)]    # the CTA's own columns of its rows, by loader warp
        self.other = [[[None] * 8 for _ in range(STAGES)] for _ in range(2)]   # the other column blocks: its rows, later the late rows
        self.rows = [[[None] * 8 for _ in range(STAGES)] for _ in range(2)]    # mask and late rows
        self.q_t, self.q_s = [[None] * 4 for _ in range(2)], [None, None]
        self.score, self.prob, self.acc = [[None, None], [None, None]], [[[None] * 4, [None] * 4] for _ in range(2)], [None, None]
        self.post = [[[[None] * 2 for _ in range(2)] for _ in range(MAX_RING)] for _ in range(2)]
        self.sums = [[None] * 8 for _ in range(2)]
        self.procs, self.queues = {}, []
        for c in range(2):
            for w in range(8):
                self.procs["softmax%d.%d" % (c, w)] = self.softmax(c, w)
                self.procs["loader%d.%d" % (c, w)] = self.loader(c, w, self.unit("copy%d.%d" % (c, w)), self.unit("tma%d.%d" % (c, w)) if w == 0 else None)
            for w in range(4):
                self.procs["q%d.%d" % (c, w)] = self.q_warp(c, w, self.unit("tmaq%d" % c) if w == 0 else None)
                self.procs["late%d.%d" % (c, w)] = self.late(c, w, self.unit("latecopy%d.%d" % (c, w)))
            self.procs["ready%d" % c] = self.passer(self.kv_full[c], self.tile_ready)
        self.procs["lateready1"] = self.passer(self.late_full[1], [self.peer_late[0]] * 2)
        self.procs["issuer0"], self.procs["issuer1"] = self.issuer(0, self.unit("score0")), self.issuer(1, self.unit("score1"))
        self.procs["pv"] = self.pv(self.unit("pvmma"))

    # ---- an asynchronous unit: takes its operations in order, each when it likes
    def unit(self, name):
        queue = deque()
        self.queues.append(queue)

        def run():
            while True:
                if not queue:
                    yield "idle"
                    continue
                for _ in queue[0]():
                    yield None
                queue.popleft()
                yield None
        self.procs["~" + name] = run()
        return queue

    def _tile(self, c, s, it, other):
        assert self.keep[c][s] == [("own", it)] * 8 and self.other[c][s] == [(other, it)] * 8, "a tile's rows are not there"

    def _commit(self, queue, bars):
        def op():
            for b in bars:
                b.arrive()
                yield
        queue.append(op)

    # ---- the warps
    def softmax(self, c, w):
        team, quad = w >> 2, w & 3
        h, rq = quad >> 1, quad & 1
        ring, base = Ring(), 0

        def follow(it):
            assert self.post[c][it % MAX_RING][0][rq] == it and self.post[c][it % MAX_RING][1][rq] == it, "maxima of another tile"
        for n, tiles in enumerate(self.items):
            ring.skip(Q_STAGES)
            for it in range(base, base + tiles):
                if (it & 1) == team:
                    ph2 = (it >> 1) & 1
                    yield self.kv_full[c][ring.s], ring.ph()
                    assert self.rows[c][ring.s] == [it] * 8, "mask of another tile"
                    yield self.s_full[c][team], ph2
                    assert self.score[c][team] == it, "scores of another tile"
                    yield None
                    assert self.score[c][team] == it, "scores overwritten"
                    self.s_empty[0][team].arrive()
                    if it > 0:
                        yield self.m_bar[c][(it - 1) % MAX_RING][rq], ((it - 1) // MAX_RING) & 1
                    self.post[c][it % MAX_RING][h][rq] = it
                    self.m_bar[c][it % MAX_RING][rq].arrive()
                    yield None
                    if it > base:
                        follow(it - 1)
                    yield self.m_bar[c][it % MAX_RING][rq], (it // MAX_RING) & 1
                    follow(it)
                    if it >= 2:
                        yield self.pv_done[c][team], ph2 ^ 1
                    self.prob[c][team][quad] = it
                    if it > base and self.rng.random() < 0.3:   # the reference moves: O is rescaled
                        yield self.pv_done[c][team ^ 1], ((it - 1) >> 1) & 1
                        assert self.acc[c] == (n, it - 1), "O is not that of the tile before"
                        yield None
                        assert self.acc[c] == (n, it - 1), "O changed under the rescaling"
                    self.p_full[0][team].arrive()
                ring.next()
            last = base + tiles - 1
            if (last & 1) != team:
                yield self.m_bar[c][last % MAX_RING][rq], (last // MAX_RING) & 1
                follow(last)
            if n > 0:
                yield self.l_free[c], (n - 1) & 1
            self.sums[c][w] = n
            self.e_bar[c].arrive()
            base += tiles

    def q_warp(self, c, i, tma):
        q_s = tiles_done = 0
        for n in range(len(self.items) + 1):
            if n < len(self.items):
                if n > 0:
                    yield self.q_empty[c], (n - 1) & 1
                if i == 0:
                    self.q_smem[c].tx += 1
                    self.q_smem[c].arrive()

                    def load(n=n):
                        yield
                        self.q_s[c] = n
                        self.q_smem[c].landed()
                    tma.append(load)
                yield self.q_stage[c][n & 1], (n >> 1) & 1
                stages = [(q_s + k) % STAGES for k in range(Q_STAGES)]
                for _ in range(2):
                    assert all(self.keep[c][s] == [("q", n)] * 8 for s in stages), "Q is not in its stages"
                    yield None
                self.q_t[c][i] = n
                self.q_copied[c].arrive()
                if i == 0:
                    yield self.q_copied[c], n & 1
                    for s in stages:
                        self.kv_empty[c][s].arrive()
                q_s = (q_s + Q_STAGES + self.items[n]) % STAGES
                yield self.q_smem[c], n & 1
                assert self.q_s[c] == n
                self.q_full[0].arrive()
            if n > 0:
                tiles_done += self.items[n - 1]
                yield self.e_bar[c], (n - 1) & 1
                assert self.sums[c] == [n - 1] * 8, "sums of another item"
                yield None
                assert self.sums[c] == [n - 1] * 8, "sums overwritten"
                self.l_free[c].arrive()
                yield self.o_full[c], (n - 1) & 1
                for _ in range(2):
                    assert self.acc[c] == (n - 1, tiles_done - 1), "O of another item"
                    yield None
                self.o_free[0].arrive()

    def issuer(self, par, mma):
        it, ring = 0, Ring()
        for n, tiles in enumerate(self.items):
            ring.skip(Q_STAGES)
            yield self.q_full[0], n & 1
            for _ in range(tiles):
                s, sb = ring.s, it & 1
                if sb == par or not self.own_barriers:
                    yield self.tile_ready[par][s], ring.ph()
                if sb == par:
                    if it >= 2:
                        yield self.s_empty[0][sb], ((it >> 1) & 1) ^ 1

                    def scores(it=it, n=n, s=s, sb=sb):
                        for _ in range(2):
                            for c in range(2):
                                self._tile(c, s, it, "own")
                                assert self.q_t[c] == [n] * 4 and self.q_s[c] == n, "Q of another item"
                            yield
                        self.score[0][sb] = self.score[1][sb] = it
                    mma.append(scores)
                    self._commit(mma, [self.s_full[c][sb] for c in range(2)])
                    self._commit(mma, [self.dead[c][s] for c in range(2)])
                it += 1
                if sb == par or not self.own_barriers:
                    ring.next()
                else:
                    ring.skip(1)
            self._commit(mma, self.q_empty)

    def pv(self, mma):
        it, ring, ready = 0, Ring(), [Ring(), Ring()]
        for n, tiles in enumerate(self.items):
            ring.skip(Q_STAGES)
            for t in range(tiles):
                s, sb, ph = ring.s, it & 1, ring.ph()
                bits = ready[sb if self.own_barriers else 0]
                yield self.tile_ready[sb][s], (bits.bits >> s) & 1
                bits.bits ^= 1 << s
                yield self.late_full[0][s], ph
                yield self.peer_late[0][s], ph
                if t == 0 and n > 0:
                    yield self.o_free[0], (n - 1) & 1
                yield self.p_full[0][sb], (it >> 1) & 1

                def product(it=it, n=n, t=t, s=s, sb=sb):
                    for _ in range(2):
                        for c in range(2):
                            self._tile(c, s, it, "late")
                            assert self.prob[c][sb] == [it] * 4, "P of another tile"
                            assert t == 0 or self.acc[c] == (n, it - 1)
                        yield
                    self.acc[0] = self.acc[1] = (n, it)
                mma.append(product)
                self._commit(mma, [self.kv_empty[c][s] for c in range(2)])
                self._commit(mma, [self.pv_done[c][sb] for c in range(2)])
                if t + 1 == tiles:
                    self._commit(mma, self.o_full)
                it += 1
                ring.next()

    def passer(self, src, dst):
        it, ring = 0, Ring()
        for tiles in self.items:
            ring.skip(Q_STAGES)
            for _ in range(tiles):
                yield src[ring.s], ring.ph()
                dst[it & 1][ring.s].arrive()
                it += 1
                ring.next()

    def loader(self, c, w, copies, tma):
        it, ring = 0, Ring((1 << STAGES) - 1)
        for n, tiles in enumerate(self.items):
            for i in range(Q_STAGES):
                s = ring.s
                yield self.kv_empty[c][s], ring.ph()
                if w == 0:
                    if i == 0:
                        self.q_stage[c][n & 1].tx += Q_STAGES

                    def load(n=n, s=s):
                        yield
                        self.keep[c][s] = [("q", n)] * 8
                        self.other[c][s] = [("q", n)] * 8
                        self.q_stage[c][n & 1].landed()
                    tma.append(load)
                ring.next()
            self.q_stage[c][n & 1].arrive()
            for _ in range(tiles):
                s = ring.s
                yield self.kv_empty[c][s], ring.ph()
                self.rows[c][s][w] = it

                def copy(it=it, s=s):
                    yield
                    self.keep[c][s][w] = self.other[c][s][w] = ("own", it)
                    yield
                    self.kv_full[c][s].arrive(32)
                copies.append(copy)
                yield None
                self.kv_full[c][s].arrive(1)
                it += 1
                ring.next()

    def late(self, c, w, copies):
        it, ring = 0, Ring()
        for tiles in self.items:
            ring.skip(Q_STAGES)
            for _ in range(tiles):
                s = ring.s
                yield self.kv_full[c][s], ring.ph()
                assert self.rows[c][s][2 * w:2 * w + 2] == [it] * 2, "late rows of another tile"
                yield self.dead[c][s], ring.ph()

                def copy(it=it, s=s):
                    yield
                    self.other[c][s][2 * w:2 * w + 2] = [("late", it)] * 2
                    yield
                    self.late_full[c][s].arrive(32)
                copies.append(copy)
                it += 1
                ring.next()

    # ---- runs to the end with `slow` held back whenever anything else can run; None: no process is favoured
    def run(self, slow=None):
        state = {name: next(p) for name, p in self.procs.items()}
        done = set()

        def step(name):
            want = state[name]
            if name in done or (want not in (None, "idle") and not want[0].passes(want[1])):
                return False
            try:
                state[name] = next(self.procs[name])
            except StopIteration:
                done.add(name)
                return True
            return not (want == "idle" and state[name] == "idle")
        names = list(self.procs)
        while True:
            self.rng.shuffle(names)
            moved = False
            for name in names:
                if name != slow:
                    for _ in range(self.rng.choice((1, 1, 2, 6))):
                        if not step(name):
                            break
                        moved = True
            if not moved and not (slow and step(slow)):
                break
        stuck = sorted(n for n in self.procs if n not in done and n[0] != "~")
        assert not stuck and not any(self.queues), "deadlock: %s" % stuck


LISTS = [[1] * 9, [2] * 6, [3, 1, 2, 5, 1, 1, 4], [10, 11], [32]]
ROLES = ["softmax0.0", "softmax1.3", "softmax0.6", "softmax1.5", "loader0.0", "loader1.0", "loader0.5", "q0.0", "q1.0", "q1.2", "late0.1", "late1.2", "ready0", "ready1", "lateready1",
         "issuer0", "issuer1", "pv", "~score0", "~score1", "~pvmma", "~copy0.3", "~copy1.6", "~latecopy0.2", "~latecopy1.0", "~tma0.0", "~tma1.0", "~tmaq0", "~tmaq1"]


@pytest.mark.parametrize("items", LISTS, ids=str)
def test_no_schedule_stalls_or_mixes_tiles(items):
    for seed in range(4):
        Pair(items, OWN_BARRIERS, random.Random(seed)).run()
    for i, role in enumerate(ROLES):
        Pair(items, OWN_BARRIERS, random.Random(100 + i)).run(slow=role)


def test_the_model_sees_a_missed_phase():
    """On common barriers an issuer that is held back before the other's tile finds that tile's phase gone."""
    with pytest.raises(AssertionError, match="deadlock"):
        Pair([10, 11], False, random.Random(0)).run(slow="issuer0")
