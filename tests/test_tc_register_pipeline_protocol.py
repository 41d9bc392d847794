"""A model of the mbarrier protocol of the tensor-core kernel's register
pipeline (lakde_b200/csrc/tc.cu, tc_kernel): the planner, index, copy,
converter, epilogue and MMA warps as coroutines, MMA completions landing in
issue order, mbarriers with the hardware's phase-parity wait.  Random
schedules of random row structures must finish without deadlock, and no
buffer (plan half, index slot, A tile, B stage, TMEM accumulator, M-step
accumulator copy) may be rewritten before its last reader is done.  `na` is
the number of A tiles, `ncw` / `new` the converter and epilogue warps."""

import random

import pytest

NS, NCOPY, NIDX, HALF = 8, 2, 2, 32


class Bar:
    """mbarrier: arrival count, transaction bytes, completed phases."""

    def __init__(self, count):
        self.count, self.pending, self.tx, self.completed = count, count, 0, 0

    def arrive(self, tx=0):
        self.tx += tx
        self.pending -= 1
        self._check()

    def complete_tx(self, b):
        self.tx -= b
        self._check()

    def _check(self):
        assert self.pending >= 0, "more arrivals than the phase expects"
        if self.pending == 0 and self.tx == 0:
            self.completed += 1
            self.pending = self.count

    def ready(self, parity):
        return (self.completed & 1) != parity


def simulate(rows, mode, na, seed, ncw=8, new=8, stall=False, early_release=False, mma_unplans=True,
             slow=None):
    """Runs one schedule; "ok" or "deadlock" (asserts on early reuse).

    `slow` names a warp that is scheduled far less often than the others;
    `mma_unplans=False` leaves the MMA warp out of a plan half's readers."""
    rng = random.Random(seed)
    mstep, pred = mode == "M", mode == "P"
    copies = 0 if mstep else NCOPY
    ngrp = new // 4
    pfull, pempty = [Bar(1), Bar(1)], [Bar(ncw + new + copies + mma_unplans) for _ in range(2)]
    mfull, mempty = [Bar(32) for _ in range(NS)], [Bar(ncw + new) for _ in range(NS)]
    bfull, bempty = [Bar(NCOPY), Bar(NCOPY)], [Bar(1), Bar(1)]
    mma_done, conv = [Bar(1), Bar(1)], [Bar(ncw + (0 if mstep else 4)) for _ in range(2)]
    efull, efree, afull, afree = ([Bar(n), Bar(n)] for n in (4, 4, 1, 4))
    tiles = [(r, j == 0, j == n - 1) for r, n in enumerate(rows) for j in range(n)]
    T = len(tiles)
    plan, slots = [None] * (2 * HALF), [None] * NS
    mmaq, bst, a_tile = [], [[None] * NCOPY, [None] * NCOPY], [None] * na
    done, converted, acc_read = dict(mma=-1), [0] * T, [0] * T
    copy_readers = {}  # M-step: epilogue warps still to read the group's accumulator copy
    plan_users = [set() for _ in range(T + 1)]
    slot_users = [set() for _ in range(T + 1)]
    warps = [("c", w) for w in range(ncw)] + [("e", w) for w in range(new)]

    def entry(t):
        m = plan[t % (2 * HALF)]
        assert m is not None and m["t"] == t, ("plan entry not there or overwritten", t, m)
        return m

    def planned(t):
        return ("wait", pfull[(t // HALF) & 1], (t // (2 * HALF)) & 1)

    def ready(t):
        return planned(t) if pred else ("wait", mfull[t % NS], (t // NS) & 1)

    def unplan(t, who):
        plan_users[t].discard(who)
        if t % HALF == HALF - 1:
            pempty[(t // HALF) & 1].arrive()

    def planner():
        for h in range(10**6):
            if h >= 2:
                yield ("wait", pempty[h & 1], (h // 2 - 1) & 1)
                assert not any(plan_users[t] for t in range((h - 2) * HALF, (h - 1) * HALF)), ("plan reused", h)
            stop = False
            for t in range(h * HALF, (h + 1) * HALF):
                if t == T:
                    plan[t % (2 * HALF)] = dict(t=t, n=-1)
                    stop = True
                    break
                r, first, last = tiles[t]
                plan[t % (2 * HALF)] = dict(t=t, n=r, row=r, first=first, last=last)
                plan_users[t] = set(warps) | ({"mma"} if mma_unplans else set()) | {("w", c) for c in range(copies)}
            pfull[h & 1].arrive()
            if stop:
                return
            yield ("step",)

    def indexer(iw):
        seen = 0

        def load(t):
            nonlocal seen
            while seen <= t:
                if seen % HALF == 0:
                    yield planned(seen)
                if entry(seen)["n"] < 0:
                    return False
                seen += 1
            return True

        def put(t):
            if t >= NS:
                yield ("wait", mempty[t % NS], (t // NS - 1) & 1)
                assert not slot_users[t - NS], ("index slot reused", t)
            slots[t % NS] = t
            slot_users[t] = set(warps)
            for _ in range(32):
                mfull[t % NS].arrive()
            yield ("step",)

        yield planned(iw)
        t = iw
        have = yield from load(t)
        while have:
            h1 = yield from load(t + NIDX)
            yield from put(t)
            if not h1:
                break
            have = yield from load(t + 2 * NIDX)
            yield from put(t + NIDX)
            t += 2 * NIDX
        if seen % NIDX == iw and entry(seen)["n"] < 0:
            if seen >= NS:
                yield ("wait", mempty[seen % NS], (seen // NS - 1) & 1)
            for _ in range(32):
                mfull[seen % NS].arrive()

    def copier(cw):
        first_copy = True
        for t in range(T + 1):
            yield planned(t)
            m = entry(t)
            if m["n"] < 0:
                return
            if m["first"]:
                b, row = m["row"] & 1, m["row"]
                if row >= 2:
                    yield ("wait", bempty[b], (row // 2 - 1) & 1)
                prev = [k for k, x in enumerate(tiles) if x[0] == row - 2]
                assert not prev or done["mma"] >= max(prev), ("B stage overwritten under its MMAs", t)
                bst[b][cw] = None
                yield ("step",)  # the copies land before the arrival
                bst[b][cw] = row
                bfull[b].arrive(tx=16 if stall and first_copy and cw == 0 else 0)
                first_copy = False
            unplan(t, ("w", cw))
            yield ("step",)

    def mma():
        yield planned(0)
        for t in range(T + 1):
            m, s = entry(t), t & 1
            if m["n"] < 0:
                return
            if mma_unplans:
                unplan(t, "mma")
            row = m["row"]
            if m["first"]:
                if not mstep:
                    yield ("wait", bfull[row & 1], (row >> 1) & 1)
                elif row >= 2:
                    yield ("wait", afree[row & 1], (row // 2 - 1) & 1)
            yield ("wait", conv[s], (t // 2) & 1)
            assert converted[t] == ncw
            if mstep:
                prev = [k for k, x in enumerate(tiles) if x[0] == row - 2 and x[2]]
                assert not m["first"] or not prev or acc_read[prev[0]] == 4, ("row accumulator reused", t)
            else:
                assert t < 2 or acc_read[t - 2] == 4, ("accumulator reused before its epilogue", t)

            def land(t=t, s=s, m=m, row=row):
                if not mstep:
                    assert bst[row & 1] == [row] * NCOPY, ("wrong W cores", t)
                assert a_tile[t % na] == t, ("A tile changed under its MMAs", t)
                done["mma"] = t
                mma_done[s].arrive()
                if m["last"]:
                    (afull if mstep else bempty)[row & 1].arrive()

            mmaq.append(land)
            yield ("step",)

    def converter(w):
        me = ("c", w)
        yield ready(0)
        for t in range(T + 1):
            m = entry(t)
            if m["n"] < 0:
                return
            yield ready(t + 1)
            if t >= na:
                yield ("wait", mma_done[(t - na) & 1], ((t - na) // 2) & 1)
                assert done["mma"] >= t - na
            assert pred or slots[t % NS] == t, ("slot changed under a converter", t)
            assert a_tile[t % na] in (None, t, t - na)
            a_tile[t % na] = t
            converted[t] += 1
            yield ("step",)
            conv[t & 1].arrive()
            if not pred:
                slot_users[t].discard(me)
                mempty[t % NS].arrive()
            entry(t + 1)  # the next tile's rows are loaded
            if not pred and t + 1 < T:
                assert slots[(t + 1) % NS] == t + 1
            yield ("step",)
            unplan(t, me)

    def epilogue(w):
        me, grp, use = ("e", w), w // 4, 0
        if not mstep and grp == 0:
            conv[0].arrive()
            conv[1].arrive()
        for t in range(T + 1):
            yield ready(t)
            m = entry(t)
            if m["n"] < 0:
                return
            acc = m["row"] if mstep else t
            if early_release and not pred:
                mempty[t % NS].arrive()
            if (not mstep or m["last"]) and acc % ngrp == grp:
                yield ("wait", (afull if mstep else mma_done)[acc & 1], (acc // 2) & 1)
                assert done["mma"] >= t
                if mstep:
                    if use > 0:
                        yield ("wait", efree[grp], (use - 1) & 1)
                        assert copy_readers.get(grp, 0) == 0, ("accumulator copy overwritten", t)
                    efull[grp].arrive()
                    yield ("wait", efull[grp], use & 1)
                    copy_readers[grp] = copy_readers.get(grp, 0) + 1
                    yield ("step",)
                    copy_readers[grp] -= 1
                    efree[grp].arrive()
                    use += 1
                acc_read[t] += 1
                yield ("step",)
                (afree if mstep else conv)[acc & 1].arrive()
            slot_users[t].discard(me)
            if not pred and not early_release:
                mempty[t % NS].arrive()
            unplan(t, me)
            yield ("step",)

    actors = [planner(), mma()] + [copier(c) for c in range(copies)]
    actors += [] if pred else [indexer(i) for i in range(NIDX)]
    actors += [converter(w) for w in range(ncw)] + [epilogue(w) for w in range(new)]
    waiting, alive = [None] * len(actors), [True] * len(actors)
    for _ in range(10**6):
        if not any(alive):
            return "ok"
        progressed = False
        order = list(range(len(actors)))
        rng.shuffle(order)
        for a in order:
            if not alive[a] or rng.random() < (0.97 if a == {"mma": 1}.get(slow) else 0.3):
                continue
            if waiting[a] is not None:
                if not waiting[a][1].ready(waiting[a][2]):
                    continue
                waiting[a] = None
            try:
                op = next(actors[a])
                if op[0] == "wait":
                    waiting[a] = op
            except StopIteration:
                alive[a] = False
            progressed = True
        if mmaq and rng.random() < 0.4:
            mmaq.pop(0)()
            progressed = True
        if not progressed:
            stuck = all(not alive[a] or (waiting[a] is not None and not waiting[a][1].ready(waiting[a][2]))
                        for a in range(len(actors)))
            if mmaq:
                mmaq.pop(0)()
            elif stuck:
                return "deadlock"
    raise AssertionError("schedule did not finish")


@pytest.mark.parametrize("mode,na,ncw,new", [("E", 2, 8, 8), ("E", 2, 4, 4), ("M", 2, 8, 8), ("M", 1, 4, 4),
                                             ("P", 2, 8, 8), ("P", 2, 8, 4)])
def test_random_schedules_finish_without_early_reuse(mode, na, ncw, new):
    for seed in range(60):
        rng = random.Random(seed)
        rows = [rng.randint(1, 4) for _ in range(rng.randint(0, 12))]
        if seed % 10 == 0:
            rows = [rng.choice([1, 1, 2, 40]) for _ in range(25)]  # several plan halves
        assert simulate(rows, mode, na, seed, ncw, new) == "ok", (mode, seed, rows)


# rows of several tiles, so that plan halves end inside a row, on many halves
LONG_ROWS = [[3] * 120, [2, 1] * 120, [5] * 80, [40, 1, 30, 2, 61, 3, 70, 20, 90]]


@pytest.mark.parametrize("mode,na,ncw,new", [("M", 2, 8, 8), ("M", 1, 4, 4), ("E", 2, 8, 8), ("P", 2, 8, 4)])
@pytest.mark.parametrize("rows", range(len(LONG_ROWS)))
def test_a_slow_mma_warp_reads_its_plan_entries(mode, na, ncw, new, rows):
    for seed in range(4):
        assert simulate(LONG_ROWS[rows], mode, na, seed, ncw, new, slow="mma") == "ok"


def test_the_model_sees_a_plan_half_reused_under_the_mma_warp():
    """The M-step's converters and epilogue can be done with a half whose last
    tile does not end its row before the MMA warp has read that tile's entry."""
    bad = 0
    for seed in range(4):
        for rows in LONG_ROWS:
            try:
                bad += simulate(rows, "M", 2, seed, 8, 8, slow="mma", mma_unplans=False) != "ok"
            except AssertionError:
                bad += 1
    assert bad


def test_a_copy_that_never_completes_blocks_the_mmas():
    """The time-out hook (a W copy expecting 16 bytes that never come) leaves
    the MMA warp waiting; in the kernel that wait is bounded."""
    assert simulate([1, 1], "E", 2, 1, stall=True) == "deadlock"


def test_the_model_sees_a_slot_that_is_released_too_early():
    with pytest.raises(AssertionError):
        for seed in range(20):
            simulate([2] * 10, "E", 2, seed, early_release=True)
