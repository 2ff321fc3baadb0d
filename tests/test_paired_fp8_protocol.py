"""The barriers of the paired kernel for an fp8 cache (csrc/paired_fp8.cu) in the model of test_paired_protocol: every warp role and every
asynchronous unit may be held back for as long as the others can run, and what each buffer holds is checked at every use."""
import os
import random
import re

import pytest

from test_paired_protocol import Bar, Pair

SRC = open(os.path.join(os.path.dirname(__file__), "..", "opfoundry_b200", "csrc", "paired_fp8.cu")).read()


def _const(name):
    return int(re.search(r"constexpr int (?:[^;]*, )?%s = (\d+)" % name, SRC).group(1))


STAGES, V_UNITS, CONVERTERS, LOADERS, WARPS, TEAM = [_const(n) for n in ("kStages", "kVUnits", "kConvWarps", "kLoadWarps", "kSoftmaxWarps", "kTeamWarps")]


class Ring:
    def __init__(self, n, ph=0):
        self.n, self.s, self.ph = n, 0, ph

    def next(self):
        self.s += 1
        if self.s == self.n:
            self.s, self.ph = 0, self.ph ^ 1


class PairFp8(Pair):
    def __init__(self, items, rng, wait_read=True, idle=lambda c, rq, n: False, wide=0.0):
        self.items, self.rng, self.wait_read, self.idle = items, rng, wait_read, idle
        bars = lambda n, count: [[Bar(count) for _ in range(n)] for _ in range(2)]
        one = lambda count: [Bar(count) for _ in range(2)]
        self.kv_full, self.raw_empty, self.prep = bars(STAGES, LOADERS * 33), bars(STAGES, 1 + CONVERTERS + TEAM), bars(STAGES, 1)
        self.late_known = bars(STAGES, LOADERS)
        self.late = [[[None] * LOADERS for _ in range(STAGES)] for _ in range(2)]  # rows of the other CTA
        self.tile_ready = bars(STAGES, 2)   # CTA 0's, by the issuer that takes the tile
        self.v_full, self.v_empty = [Bar(CONVERTERS) for _ in range(V_UNITS)], bars(V_UNITS, 1)
        self.s_full, self.s_empty, self.p_full, self.pv_done = bars(2, 1), [Bar(2 * TEAM) for _ in range(2)], [Bar(2 * TEAM) for _ in range(2)], bars(2, 1)
        self.s3_empty, self.q_full, self.o_free = Bar(2 * TEAM), Bar(2 * WARPS), Bar(2 * WARPS)
        self.posted, self.moved = [[[[Bar(TEAM // 2) for _ in range(2)] for _ in range(2)] for _ in range(2)] for _ in range(2)]
        self.residual_here = [[Bar(WARPS // 2) for _ in range(2)] for _ in range(2)]
        self.left = [[[None] * (WARPS // 2) for _ in range(2)] for _ in range(2)]   # residuals of an item that has some, [cta][rows]
        self.wide = [[[rng.random() < wide for _ in items] for _ in range(2)] for _ in range(2)]
        self.q_here, self.q_empty, self.o_full, self.e_bar = one(WARPS), one(2), one(1), one(WARPS)
        # what the buffers hold
        self.raw = [[[None] * LOADERS for _ in range(STAGES)] for _ in range(2)]   # rows and scales, by loader warp
        self.mask = [[[None] * LOADERS for _ in range(STAGES)] for _ in range(2)]
        self.e = [[None] * STAGES for _ in range(2)]
        self.v = [[[None] * (CONVERTERS // 2) for _ in range(V_UNITS)] for _ in range(2)]
        self.q = [[None] * WARPS for _ in range(2)]                              # with the row factors
        self.score, self.score3 = [[None, None], [None, None]], [None, None]     # groups 0-2 by team | group 3 and the rope
        self.prob, self.acc = [[[None] * TEAM, [None] * TEAM] for _ in range(2)], [None, None]
        self.post = [[[[None] * 4 for _ in range(2)] for _ in range(2)] for _ in range(2)]   # [cta][team][rows][quarter]
        self.ref = [[[None] * 2 for _ in range(2)] for _ in range(2)]                        # [cta][tile mod 2][rows]
        self.v_fin = [[None] * 4 for _ in range(2)]                              # [cta][scale group]
        self.lent = [rng.random() < 0.3 for _ in range(7)]
        self.procs, self.queues = {}, []
        for c in range(2):
            for w in range(WARPS):
                self.procs["softmax%d.%d" % (c, w)] = self.softmax(c, w)
            for w in range(LOADERS):
                self.procs["loader%d.%d" % (c, w)] = self.loader(c, w, self.unit("copy%d.%d" % (c, w)))
            for w in range(CONVERTERS):
                self.procs["conv%d.%d" % (c, w)] = self.converter(c, w)
            self.procs["ready%d" % c] = self.ready(c)
        self.procs["issuer0"], self.procs["issuer1"] = self.issuer(0, self.unit("score0")), self.issuer(1, self.unit("score1"))
        self.procs["pv"] = self.pv(self.unit("pvmma"))

    def softmax(self, c, w):
        team, cs, quad = w >> 3, (w >> 2) & 1, w & 3
        h, rq = quad >> 1, quad & 1
        ring, base, end = Ring(STAGES), 0, 0
        second, n_wide = False, 0       # the form for items with residuals
        if team:
            ring.next()
        for n in range(len(self.items) + 1):
            if n < len(self.items):
                if n > 0:
                    yield self.q_empty[c], (n - 1) & 1
                self.q[c][w] = n
                self.q_full.arrive()
                yield None
                self.q_here[c].arrive()
            if n > 0:
                yield self.o_full[c], (n - 1) & 1
                for _ in range(2):
                    assert self.acc[c] == (n - 1, end - 1), "O of another item"
                    yield None
                self.o_free.arrive()
            if n == len(self.items):
                break
            base, end = end, end + self.items[n]
            yield self.q_here[c], n & 1
            assert self.q[c] == [n] * WARPS, "row factors of another item"
            wide = self.wide[c][rq][n] and not self.idle(c, rq, n)
            if wide:
                second = True
                self.left[c][rq][4 * team + 2 * cs + h] = n
                yield None
                self.residual_here[c][rq].arrive()
                yield self.residual_here[c][rq], n_wide & 1
                n_wide += 1
            for it in range(base + ((base ^ team) & 1), end, 2):
                ph2, first = (it >> 1) & 1, it == base
                if self.idle(c, rq, n):
                    yield self.s_full[c][team], ph2
                    self.s3_empty.arrive()
                    self.s_empty[team].arrive()
                    self.raw_empty[c][ring.s].arrive()
                    if it >= 2:
                        yield self.pv_done[c][team], ph2 ^ 1
                    self.posted[c][team][rq].arrive()
                    yield None
                    self.moved[c][team][rq].arrive()
                    self.ref[c][team][rq] = it
                    self.prob[c][team][w & 7] = it
                    yield None
                    self.p_full[team].arrive()
                    ring.next()
                    ring.next()
                    continue
                yield self.prep[c][ring.s], ring.ph
                yield self.s_full[c][team], ph2
                if self.wait_read:
                    yield self.moved[c][team][rq], ph2 ^ 1
                assert self.mask[c][ring.s] == [it] * LOADERS and self.e[c][ring.s] == it, "mask of another tile"
                yield None
                assert self.score3[c] == it, "scores of another tile"
                self.s3_empty.arrive()
                yield None
                assert self.score[c][team] == it, "scores of another tile"
                if not second:
                    self.s_empty[team].arrive()
                yield None
                if second:
                    assert self.score[c][team] == it and (not wide or self.left[c][rq] == [n] * (WARPS // 2)), "residuals of another item"
                    self.s_empty[team].arrive()
                assert self.raw[c][ring.s] == [it] * LOADERS, "scales of another tile"
                lent = self.lent[it % len(self.lent)]       # rows took more than 2^-e: P is multiplied with what stands beside e
                if not lent:
                    self.raw_empty[c][ring.s].arrive()
                self.post[c][team][rq][2 * h + cs] = ("max", it)
                self.posted[c][team][rq].arrive()
                yield self.posted[c][team][rq], ph2
                yield self.moved[c][team ^ 1][rq], ((it - 1) >> 1) & 1
                assert self.post[c][team][rq] == [("max", it)] * 4, "maxima of another tile"
                assert first or self.ref[c][team ^ 1][rq] == it - 1, "references of another tile"
                yield None
                if h == 0 and cs == 0:
                    self.ref[c][team][rq] = it
                self.moved[c][team][rq].arrive()
                if lent:
                    yield None
                    assert self.e[c][ring.s] == it, "powers of two of another tile"
                    self.raw_empty[c][ring.s].arrive()
                if it >= 2:
                    yield self.pv_done[c][team], ph2 ^ 1
                self.prob[c][team][w & 7] = it
                if not first and self.rng.random() < 0.3:   # the reference or e moves: O is rescaled
                    yield self.pv_done[c][team ^ 1], ((it - 1) >> 1) & 1
                    for _ in range(2):
                        assert self.acc[c] == (n, it - 1), "O is not that of the tile before"
                        yield None
                self.p_full[team].arrive()
                ring.next()
                ring.next()
            last = end - 1
            yield self.moved[c][last & 1][rq], (last >> 1) & 1
            assert self.idle(c, rq, n) or self.ref[c][last & 1][rq] == last, "references of another tile"   # (those of rows that are not live serve nobody)
            self.post[c][team][rq][2 * h + cs] = ("sum", n)
            if team == last & 1 and rq == 0:
                self.v_fin[c][2 * h + cs] = n
            self.e_bar[c].arrive()
            yield self.e_bar[c], n & 1
            for _ in range(2):
                assert all(x == ("sum", n) for t in range(2) for x in self.post[c][t][rq]) and self.v_fin[c][2 * h + team] == n, "sums of another item"
                yield None

    def issuer(self, par, mma):
        it, ring, ready = 0, Ring(STAGES), [0] * STAGES
        for n, tiles in enumerate(self.items):
            yield self.q_full, n & 1
            for _ in range(tiles):
                s = ring.s
                if (it & 1) == par:
                    yield self.tile_ready[par][s], ready[s]
                    ready[s] ^= 1
                    if it >= 2:
                        yield self.s_empty[par], ((it >> 1) & 1) ^ 1

                    def scores(it=it, n=n, s=s, last=False):
                        for c in range(2):
                            self.score3[c] = None if last else self.score3[c]
                            self.score[c][par] = self.score[c][par] if last else None
                        for _ in range(2):
                            for c in range(2):
                                assert self.raw[c][s] == [it] * LOADERS, "rows of another tile"
                                assert self.q[c] == [n] * WARPS, "Q of another item"
                            yield
                        for c in range(2):
                            if last:
                                self.score3[c] = it
                            else:
                                self.score[c][par] = it
                    mma.append(scores)
                    if it >= 1:
                        yield self.s3_empty, (it - 1) & 1
                    mma.append(lambda f=scores: f(last=True))
                    self._commit(mma, [self.s_full[c][par] for c in range(2)])
                    self._commit(mma, [self.raw_empty[c][s] for c in range(2)])
                it += 1
                ring.next()
            self._commit(mma, self.q_empty)

    def pv(self, mma):
        it, unit = 0, Ring(V_UNITS)
        for n, tiles in enumerate(self.items):
            for t in range(tiles):
                sb = it & 1
                if t == 0 and n > 0:
                    yield self.o_free, (n - 1) & 1
                yield self.p_full[sb], (it >> 1) & 1
                for u in range(2):
                    yield self.v_full[unit.s], unit.ph

                    def product(it=it, n=n, t=t, u=u, s=unit.s, sb=sb):
                        for _ in range(2):
                            for c in range(2):
                                assert self.v[c][s] == [(it, u)] * (CONVERTERS // 2), "V of another unit"
                                assert self.prob[c][sb] == [it] * TEAM, "P of another tile"
                                assert (t == 0 and u == 0) or self.acc[c] == ((n, it - 1) if u == 0 else (n, it, 0))
                            yield
                        self.acc[0] = self.acc[1] = (n, it) if u else (n, it, 0)
                    mma.append(product)
                    self._commit(mma, [self.v_empty[c][unit.s] for c in range(2)])
                    unit.next()
                self._commit(mma, [self.pv_done[c][sb] for c in range(2)])
                if t + 1 == tiles:
                    self._commit(mma, self.o_full)
                it += 1

    def ready(self, c):
        it, ring = 0, Ring(STAGES)
        for tiles in self.items:
            for _ in range(tiles):
                yield self.kv_full[c][ring.s], ring.ph
                self.tile_ready[it & 1][ring.s].arrive()
                yield None
                assert self.raw[c][ring.s] == self.late[c][ring.s] == [it] * LOADERS, "scales of another tile"
                self.e[c][ring.s] = it
                self.prep[c][ring.s].arrive()
                it += 1
                ring.next()

    def loader(self, c, w, copies):
        it, ring = 0, Ring(STAGES, 1)
        for tiles in self.items:
            for _ in range(tiles):
                s = ring.s
                yield self.raw_empty[c][s], ring.ph
                self.late[c][s][w] = it
                self.late_known[c][s].arrive()
                yield None
                self.mask[c][s][w] = it

                def copy(it=it, s=s):
                    self.raw[c][s][w] = None
                    yield
                    self.raw[c][s][w] = it
                    yield
                    self.kv_full[c][s].arrive(32)
                copies.append(copy)
                yield None
                self.kv_full[c][s].arrive(1)
                it += 1
                ring.next()

    def converter(self, c, w):
        it, u, ring, unit, known = 0, w // (CONVERTERS // 2), Ring(STAGES), Ring(V_UNITS, 1), Ring(STAGES)
        if u:
            unit.next()
        for tiles in self.items:
            for t in range(tiles):
                s = ring.s
                for ahead in ((0, 1) if t == 0 else (1,)) if u != c else ():   # the other CTA's rows are fetched a tile ahead
                    if t + ahead < tiles:
                        yield self.late_known[c][known.s], known.ph
                        assert self.late[c][known.s] == [it + ahead] * LOADERS, "rows of another tile"
                        known.next()
                yield self.prep[c][s], ring.ph
                yield self.v_empty[c][unit.s], unit.ph
                for _ in range(2):
                    assert self.raw[c][s] == [it] * LOADERS and self.e[c][s] == it, "rows of another tile"
                    yield None
                self.raw_empty[c][s].arrive()
                self.v[c][unit.s][w % (CONVERTERS // 2)] = (it, u)
                yield None
                self.v_full[unit.s].arrive()
                unit.next()
                unit.next()
                it += 1
                ring.next()


LISTS = [[1] * 9, [2] * 6, [3, 1, 2, 5, 1, 1, 4], [10, 11], [32]]
ROLES = ["softmax0.0", "softmax1.3", "softmax0.6", "softmax1.5", "softmax0.8", "softmax1.11", "softmax0.15", "loader0.0", "loader1.0", "conv0.1", "conv1.7", "ready0", "ready1",
         "issuer0", "issuer1", "pv", "~score0", "~score1", "~pvmma", "~copy0.3", "~copy1.1"]


@pytest.mark.parametrize("items", LISTS, ids=str)
def test_no_schedule_stalls_or_mixes_tiles(items):
    for seed in range(4):
        PairFp8(items, random.Random(seed)).run()
    for i, role in enumerate(ROLES):
        PairFp8(items, random.Random(100 + i)).run(slow=role)


@pytest.mark.parametrize("idle", [lambda c, rq, n: rq == 1, lambda c, rq, n: c == 1 or rq == 1, lambda c, rq, n: c == 1 and rq == 1 and n % 2 == 1,
                                  lambda c, rq, n: n % 3 == c and rq == 1], ids=["half", "one CTA", "by turns", "by CTA"])
def test_warps_without_live_rows(idle):
    for items in ([1] * 9, [3, 1, 2, 5, 1, 1, 4]):
        for i, role in enumerate([None, "softmax0.0", "softmax1.3", "softmax0.5", "softmax1.14", "softmax0.2", "pv", "issuer1", "~pvmma", "conv1.3"]):
            PairFp8(items, random.Random(i), idle=idle).run(slow=role)


def test_items_with_residuals():
    for items in ([1] * 9, [3, 1, 2, 5, 1, 1, 4]):
        for i, role in enumerate([None, "softmax0.0", "softmax1.3", "softmax0.5", "softmax1.14", "softmax0.2", "pv", "issuer1", "~score0"]):
            PairFp8(items, random.Random(i), wide=0.5, idle=(lambda c, rq, n: rq == 1) if i % 3 == 2 else lambda c, rq, n: False).run(slow=role)

def sync_points(src):
    """Every wait, arrival and commit of the kernel, in the order of the source, with its barrier and parity."""
    src, out = re.sub(r"//[^\n]*", "", src), []
    for m in re.finditer(r"\b(wait_on[23]?|warp_wait|warp_arrive(?:_lead)?|tc_commit_pair_el|cp_async_mbar_arrive_noinc)\(", src):
        depth, i = 1, m.end()
        while depth:
            depth += {"(": 1, ")": -1}.get(src[i], 0)
            i += 1
        args = re.sub(r"\s+", " ", re.sub(r"smem_u32\(&ctl->([^()]*)\)", r"&ctl->\1", src[m.end():i - 1]))
        if "ctl->" in args:     # (else a wrapper's own)
            for part in ("&ctl->", ", abort_flag", ", lane", ", el"):
                args = args.replace(part, "")
            out.append(m.group(1) + " " + args)
    return out


# What the roles above restate, role by role.  A line that differs from the source means that the model has to be looked at again.
SYNC_POINTS = """
warp_arrive_lead q_full
warp_arrive q_here
wait_on q_empty, (item_n - 1) & 1
wait_on o_full, (item_n - 1) & 1
warp_arrive_lead o_free
warp_arrive_lead o_free
warp_arrive_lead o_free
wait_on q_here, item_n & 1
warp_arrive residual_here[rq]
wait_on residual_here[rq], n_wide & 1
wait_on s_full[team], ph2
warp_arrive_lead s3_empty
warp_arrive_lead s_empty[team]
warp_arrive raw_empty[ring.s]
wait_on pv_done[team], ph2 ^ 1u
warp_arrive posted[team][rq]
warp_arrive moved[team][rq]
warp_arrive_lead p_full[team]
wait_on3 prep[ring.s], ring.ph, s_full[team], ph2, moved[team][rq], ph2 ^ 1u
warp_arrive_lead s3_empty
warp_arrive_lead s_empty[team]
warp_arrive raw_empty[ring.s]
warp_arrive_lead s_empty[team]
warp_arrive posted[team][rq]
wait_on2 posted[team][rq], ph2, moved[team ^ 1][rq], ((it - 1) >> 1) & 1u
warp_arrive moved[team][rq]
warp_arrive raw_empty[ring.s]
wait_on pv_done[team], ph2 ^ 1u
wait_on pv_done[team ^ 1], ((it - 1) >> 1) & 1u
warp_arrive_lead p_full[team]
wait_on moved[last_team][rq], (last >> 1) & 1u
warp_arrive e_bar
wait_on e_bar, item_n & 1
wait_on q_full, item_n & 1
wait_on tile_ready[par][ring.s], (ready_bits >> ring.s) & 1u
wait_on s_empty[par], ((it >> 1) & 1u) ^ 1u
wait_on s3_empty, (it - 1) & 1u
tc_commit_pair_el s_full[par]
tc_commit_pair_el raw_empty[ring.s]
tc_commit_pair_el q_empty
wait_on o_free, (item_n - 1) & 1
wait_on p_full[sb], (it >> 1) & 1u
wait_on v_full[unit.s], unit.ph
tc_commit_pair_el v_empty[unit.s]
tc_commit_pair_el pv_done[sb]
tc_commit_pair_el o_full
warp_wait kv_full[ring.s], ring.ph
warp_arrive_lead tile_ready[it & 1u][ring.s]
warp_arrive prep[ring.s]
warp_wait finished, 0
wait_on raw_empty[ring.s], ring.ph
warp_arrive late_known[ring.s]
cp_async_mbar_arrive_noinc kv_full[ring.s]
warp_arrive kv_full[ring.s]
wait_on2 prep[ring.s], ring.ph, v_empty[unit.s], unit.ph
warp_arrive raw_empty[ring.s]
warp_arrive_lead v_full[unit.s]
wait_on late_known[known.s], known.ph
wait_on late_known[known.s], known.ph
wait_on2 prep[ring.s], ring.ph, v_empty[unit.s], unit.ph
warp_arrive raw_empty[ring.s]
warp_arrive_lead v_full[unit.s]
warp_arrive finished
"""


def test_the_model_restates_the_kernels_waits_and_arrivals():
    assert sync_points(SRC) == SYNC_POINTS.strip().split("\n")


def test_the_model_counts_arrivals_as_the_kernel_does():
    names = ("kLoadWarps", "kConvWarps", "kTeamWarps", "kSoftmaxWarps", "kWarps")
    values = {n: _const(n) for n in names}
    model = PairFp8([1], random.Random(0))
    found = re.findall(r"mbar_init\(smem_u32\(&ctl->(\w+)[^)]*\), ([^;]+)\);", SRC)
    assert len({n for n, _ in found}) == 22
    for name, count in found:
        if name == "finished":      # at the end of every other warp; the model ends by itself
            continue
        bar = getattr(model, name)
        while isinstance(bar, list):
            bar = bar[0]
        assert bar.count == eval(count.replace("/", "//"), {}, values), name



def test_the_model_sees_a_missing_wait():
    """A warp that posts a tile's maxima before its team has read those of the team's last tile."""
    with pytest.raises(AssertionError, match="maxima of another tile"):
        for i in range(16):
            PairFp8([3, 1, 2, 5, 1, 1, 4], random.Random(i), wait_read=False).run(slow="softmax0.%d" % i)
