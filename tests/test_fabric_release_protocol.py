"""Host models of what the fabric's scheduler (monoserve_b200/csrc/fabric_sched.cuh) orders with its loads, stores and atomics when a stage
completes, on a memory in which a plain load may return any value a location has had since the last one its thread is bound to have
seen: an acquire load takes over what the release store it reads was bound to, an atomic reads the newest value, a fence makes
atomics before it acquire and atomics after it release.  Each rule of the device code is shown by leaving it out."""
import os
import random
import re

import pytest

SCHED = open(os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "monoserve_b200", "csrc", "fabric_sched.cuh")).read()


def body_of(name):
    text = SCHED[re.search(rf"\b{name}\(", SCHED).start():]
    return text[:text.index("\n}\n")]


class Memory:
    def __init__(self, **init):
        self.at = {k: [(v, {})] for k, v in init.items()}


class Thread:
    """Views are {location: index of the oldest value that may still be read}."""

    def __init__(self, mem, rnd):
        self.mem, self.rnd = mem, rnd
        self.view, self.pending, self.released = {}, {}, {}

    @staticmethod
    def _join(a, b):
        for k, i in b.items():
            a[k] = max(a.get(k, 0), i)

    def load(self, loc, acquire=False):
        past = self.mem.at[loc]
        i = self.rnd.randrange(self.view.get(loc, 0), len(past))
        self.view[loc] = i
        value, view = past[i]
        self._join(self.view if acquire else self.pending, view)
        return value

    def _write(self, loc, value, view):
        past = self.mem.at[loc]
        self.view[loc] = len(past)
        past.append((value, dict(view, **{loc: len(past)})))

    def store(self, loc, value, release=False):
        self._write(loc, value, self.view if release else self.released)

    def atomic(self, loc, f, acquire=False):
        value, view = self.mem.at[loc][-1]
        self._join(self.view if acquire else self.pending, view)
        merged = dict(self.released)
        self._join(merged, view)   # an atomic goes on what it reads
        self._write(loc, f(value), merged)
        return value

    def fence(self):
        self._join(self.view, self.pending)
        self.released = dict(self.view)


def interleave(rnd, roles, limit=2000):
    """Runs the generators at random until all are done; False: somebody is still waiting at the limit."""
    roles = list(roles)
    for _ in range(limit):
        if not roles:
            return True
        r = rnd.choice(roles)
        try:
            next(r)
        except StopIteration:
            roles.remove(r)
    return False


# ------------------------------------------------------------------------------------------ the published tail of a ring
def publish(th, entry, acquire):
    at = th.atomic("reserve", lambda v: v + 1)
    yield
    tail = th.load("tail", acquire)     # beside the reservation
    yield
    th.store(f"id{at}", entry)
    yield
    while tail != at:                   # an earlier reservation is not published yet
        tail = th.load("tail", acquire=True)
        yield
    th.store("tail", at + 1, release=True)


def two_publishers(seed, acquire):
    rnd = random.Random(seed)
    mem = Memory(reserve=0, tail=0, id0=None, id1=None)
    got = []

    def worker():
        th = Thread(mem, rnd)
        tail = 0
        while tail < 2:
            tail = th.load("tail", acquire=True)
            yield
        got.extend(th.load(f"id{i}") for i in range(2))

    assert interleave(rnd, [publish(Thread(mem, rnd), "a", acquire), publish(Thread(mem, rnd), "b", acquire), worker()])
    return sorted(map(str, got)) == ["a", "b"]


def test_a_later_publication_carries_the_earlier_one():
    assert all(two_publishers(seed, acquire=True) for seed in range(500))
    assert not all(two_publishers(seed, acquire=False) for seed in range(500))


def test_every_load_of_a_published_tail_acquires():
    assert re.search(r"ld_acq\(&R\.tail\)", body_of("release_stage"))
    assert not re.search(r"ld_volatile\(&R\.tail\)", SCHED)


# ------------------------------------------------------------------------------------------ a record written ahead of one predecessor
def joined(seed, acquire, behind):
    """A stage with two predecessors: a plan, which writes its tile count, and another stage; whoever completes last publishes it, with the
    count read beside its own decrement or behind it.  True: every tile ran, with the operands that both have left."""
    rnd = random.Random(seed)
    mem = Memory(count=0, deps=2, tail=0, id0=None, from_plan=0, from_other=0)
    ran = []

    def complete(th):
        th.fence()
        tiles = th.load("count")
        yield
        before = th.atomic("deps", lambda v: v - 1, acquire)
        yield
        if before != 1:
            return
        if behind:
            tiles = th.load("count")
            yield
        th.store("id0", tiles)
        th.store("tail", 1, release=True)

    def plan():
        th = Thread(mem, rnd)
        th.store("count", 3)
        th.store("from_plan", 1)
        yield
        yield from complete(th)

    def other():
        th = Thread(mem, rnd)
        th.store("from_other", 1)
        yield
        yield from complete(th)

    def worker():
        th = Thread(mem, rnd)
        while not th.load("tail", acquire=True):
            yield
        ran.append((th.load("id0"), th.load("count"), th.load("from_plan"), th.load("from_other")))

    assert interleave(rnd, [plan(), other(), worker()])
    return ran == [(3, 3, 1, 1)]


def test_the_last_decrement_sees_what_the_others_wrote():
    assert all(joined(seed, acquire=True, behind=True) for seed in range(500))
    assert not all(joined(seed, acquire=True, behind=False) for seed in range(500))
    assert not all(joined(seed, acquire=False, behind=True) for seed in range(500))


def test_the_release_of_a_stage_acquires_and_reads_late_records_behind():
    text = body_of("release_stage")
    assert "take_one_acq(&runtime[succ].deps)" in text and "atomicSub" not in text
    assert "atom.acquire.gpu" in body_of("take_one_acq")
    behind = text[text.index("take_one_acq"):]
    assert re.search(r"kSuccLate\) && \(entry & kSuccJoin\)\) \{\s*flags = ld_volatile\(&stages\[succ\]\.flags\);\s*tiles = ld_volatile", behind)
    assert re.search(r"if \(empty\) __threadfence\(\);", behind)   # stages that are complete at once pass on what was acquired


# ------------------------------------------------------------------------------------------ successors that are skipped
def skipped(seed, asks_first):
    """A stage releases two batches of successors, one that the iteration waits for and one that is skipped in it; the reset behind the
    first rewrites the second's count.  True: the next iteration finds the count whole."""
    rnd = random.Random(seed)
    mem = Memory(flags=1, deps=1, tail=0)

    def release():
        th = Thread(mem, rnd)
        th.store("tail", 1, release=True)       # the first batch
        yield
        if not (asks_first and th.load("flags")):
            th.atomic("deps", lambda v: v - 1)
        yield

    def rest():
        th = Thread(mem, rnd)
        while not th.load("tail", acquire=True):
            yield
        th.store("deps", 1)                     # the reset tile
        yield

    assert interleave(rnd, [release(), rest()])
    return mem.at["deps"][-1][0] == 1


def test_a_skipped_stage_keeps_its_count():
    assert all(skipped(seed, asks_first=True) for seed in range(200))
    assert not all(skipped(seed, asks_first=False) for seed in range(200))


def test_the_release_of_a_stage_asks_before_it_takes():
    text = body_of("release_stage")
    asks = re.search(r"if \(entry & kSuccLate\) skip = ld_volatile\(&stages\[succ\]\.flags\) & kStageSkip;", text)
    takes = re.search(r"skip \? 0u : take_one_acq", text)
    assert asks and takes and asks.start() < takes.start()


# ------------------------------------------------------------------------------------------ a lane that goes on to another program
def switched(seed, asks_again):
    """A worker reads the lane's words in any order while the lane goes on from program 1 to program 2 and publishes an entry of it;
    entries that are not of the program it looks at pass for exhausted and are dropped.  True: the entry is still in the ring."""
    rnd = random.Random(seed)
    mem = Memory(prog=1, gen=1, head=4, tail=4)

    def lane():
        th = Thread(mem, rnd)
        th.atomic("head", lambda v: 4)
        yield
        th.store("prog", 2, release=True)
        yield
        th.store("gen", 2, release=True)
        yield
        th.store("tail", 5, release=True)

    def worker():
        th = Thread(mem, rnd)
        for _ in range(6):
            words = ["prog", "gen", "head", "tail"]
            rnd.shuffle(words)
            seen = {}
            for w in words:
                seen[w] = th.load(w, acquire=True)
                yield
            if seen["tail"] <= seen["head"]:
                continue
            now = th.load("prog"), th.load("gen")
            yield
            if seen["prog"] != 2 and (not asks_again or now == (seen["prog"], seen["gen"])):
                th.atomic("head", lambda v: seen["tail"] if v == seen["head"] else v)

    assert interleave(rnd, [lane(), worker()])
    return mem.at["head"][-1][0] == 4


def test_entries_of_the_program_that_runs_now_are_not_dropped():
    assert all(switched(seed, asks_again=True) for seed in range(500))
    assert not all(switched(seed, asks_again=False) for seed in range(500))


def test_the_drop_of_exhausted_entries_asks_for_the_program_again():
    text = body_of("bool ring_take")
    again = text.index("ld_volatile(&L.prog)"), text.index("ld_volatile(&L.gen)")
    drop = re.search(r"if \([^;]*prog == reinterpret_cast<unsigned long long>\(V\.prog\) && gen == V\.gen\) atomicCAS\(&R\.head", text)
    assert drop and max(again) < drop.start()


# ------------------------------------------------------------------------------------------ the run-time limit
def test_the_run_time_limit_is_looked_at_whatever_lies_between_claims():
    """Every 16th round that finds nothing looks at the limit.  Counted anew behind each claim, rounds of a worker that finds work every
    time before the 16th would never get there."""
    def looks(gaps, anew):
        polls = n = 0
        for gap in gaps:
            for _ in range(gap):
                polls += 1
                n += polls % 16 == 0
            if anew:
                polls = 0
        return n
    rnd = random.Random(1)
    gaps = [rnd.randrange(16) for _ in range(1000)]
    assert looks(gaps, anew=True) == 0 and looks(gaps, anew=False) == sum(gaps) // 16
    device = open(os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "monoserve_b200", "csrc", "fabric_device.cu")).read()
    assert "(ws.polls & 15) == 0 && must_leave(false)" in device
    assert not re.search(r"ws\.polls = 0", SCHED)   # set where the worker starts, and only there


def woken(seed, watches_program):
    """The same lane; a worker that found nothing looks again once one of the words it watches has changed.  True: it finds the entry."""
    rnd = random.Random(seed)
    mem = Memory(prog=1, gen=1, head=4, tail=4)
    found = []

    def lane():
        th = Thread(mem, rnd)
        th.store("prog", 2, release=True)
        yield
        th.store("gen", 2, release=True)
        yield
        th.store("tail", 5, release=True)

    def worker():
        th, before = Thread(mem, rnd), None
        for _ in range(200):
            words = ["prog", "gen", "tail"]
            rnd.shuffle(words)
            seen = {}
            for w in words:
                seen[w] = th.load(w, acquire=True)
                yield
            watched = {w: v for w, v in seen.items() if w != "prog" or watches_program}
            if watched == before:
                continue
            before = watched
            if seen["tail"] > 4 and seen["prog"] == 2:
                found.append(1)
                return

    assert interleave(rnd, [lane(), worker()])
    return bool(found)


def test_a_worker_looks_again_when_the_program_has_changed():
    assert all(woken(seed, watches_program=True) for seed in range(2000))
    assert not all(woken(seed, watches_program=False) for seed in range(2000))
    assert "words != seen && !(of_lane && which == kWHead)" in body_of("uint32_t schedule")
