"""A host model of the operand ring's barriers as the MMA warp of the GEMM tiles sees them (gemm_mma in
monoserve_b200/csrc/gemm_core.cuh): the producer fills stages, every lane of the warp waits for a stage by the parity of its use, and one
lane frees it.  The lanes may run apart between the points where the warp meets; the model lets them, at random.  A second model has
a warp whose waits are given up: the abort flag goes up at any moment, and every lane has to get out of its loop."""
import os
import random
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "monoserve_b200", "csrc")

STAGES, LANES = 12, 4


def run(n_stages, seed, meets):
    """None, or what is still waited for when nobody can go on.  `meets`: the warp meets behind each stage's wait."""
    rnd = random.Random(seed)
    full, empty = [0] * STAGES, [0] * STAGES     # completed phases

    def waits(bar, s, parity):
        return lambda: (bar[s] & 1) != parity

    def producer():
        for i in range(n_stages):
            s, use = i % STAGES, i // STAGES
            if use:
                yield waits(empty, s, (use - 1) & 1), f"producer: stage {i}"
            full[s] += 1

    at = [0] * LANES                             # stages each lane has seen filled

    def lane(who):
        for i in range(n_stages):
            s = i % STAGES
            yield waits(full, s, (i // STAGES) & 1), f"lane {who}: stage {i}"
            at[who] = i + 1
            if meets:
                yield lambda: min(at) > i, f"lane {who}: the others at stage {i}"
            if who == 0:                         # the elected lane issues the products, whose completion frees the stage
                empty[s] += 1

    roles = [producer()] + [lane(k) for k in range(LANES)]
    want = {k: next(r) if k else None for k, r in enumerate(roles)}
    slow = rnd.randrange(1, LANES)               # one lane is scheduled rarely
    while want:
        ready = [k for k, w in want.items() if w is None or w[0]()]
        if not ready:
            return sorted(w[1] for w in want.values())
        fast = [k for k in ready if k != 1 + slow]
        k = rnd.choice(fast if fast and rnd.random() < 0.99 else ready)
        try:
            want[k] = next(roles[k])
        except StopIteration:
            del want[k]
    return None


@pytest.mark.parametrize("n_stages", [1, 12, 24, 25, 64, 200])
def test_every_lane_sees_every_stage(n_stages):
    for seed in range(20):
        assert run(n_stages, seed, meets=True) is None


def test_a_lane_that_does_not_meet_the_others_may_miss_a_phase():
    stuck = [run(64, seed, meets=False) for seed in range(20)]
    assert any(w and all("lane" in x for x in w) for w in stuck), stuck
    assert all(w is None for w in (run(12, seed, meets=False) for seed in range(20)))   # one lap cannot


def test_the_loops_of_the_mma_warp_meet_behind_each_wait():
    text = open(os.path.join(CSRC, "gemm_core.cuh")).read()
    for name in ("gemm_mma_two", "gemm_mma"):
        body = text[re.search(rf"__device__ __forceinline__ bool {name}\(", text).start():]
        body = body[:body.index("\n}\n")]
        loop = body[body.index("for (int kt = 0;"):]
        assert re.search(r"mbar_wait_bounded\(&\w+(\.full)?\[pipe\.slot\][^;]*;\s*(//[^\n]*\s*)*__syncwarp\(\);", loop), name
        assert "break" not in loop, name   # a lane that leaves alone would leave the others waiting at the meeting


def give_up(seed, combined):
    """Lanes that wait for stages, each trying the barrier and then looking at the abort flag, and meet behind each wait.  True: all have
    left the loop.  `combined`: a lane's answer counts once all lanes have one, and all take the same."""
    rnd = random.Random(seed)
    n_stages, aborted = 12, rnd.randrange(400)
    step, filled = [0], [0]
    answers = [[None] * LANES for _ in range(n_stages)]
    met, left = [0] * LANES, []

    def lane(who):
        for i in range(n_stages):
            while True:
                if filled[0] > i:
                    got = True
                    break
                yield None                       # the try and the look at the flag are two steps
                if step[0] >= aborted:
                    got = False
                    break
                yield None
            answers[i][who] = got
            if combined:
                yield lambda: None not in answers[i]
                got = all(answers[i])
            if not got:
                break
            met[who] = i + 1                     # an operation that names all 32 lanes
            yield lambda: min(met) > i
        left.append(who)

    roles = [lane(k) for k in range(LANES)]
    want = {k: None for k in range(LANES)}
    for step[0] in range(4000):
        if step[0] < aborted and rnd.random() < 0.05:
            filled[0] += 1
        ready = [k for k, w in want.items() if w is None or w()]
        if not ready:
            continue
        k = rnd.choice(ready)
        try:
            want[k] = next(roles[k])
        except StopIteration:
            del want[k]
    return len(left) == LANES


def test_a_warp_gives_up_as_one():
    assert all(give_up(seed, combined=True) for seed in range(200))
    assert not all(give_up(seed, combined=False) for seed in range(200))


def test_no_lane_leaves_a_wait_of_its_warp_alone():
    """A return or a break right behind a wait that each lane decides for itself, anywhere but in code of one lane (the schedulers) and
    in roles that only set a flag and go on (attention's MMA warps, which meet at their end)."""
    alone = re.compile(r"if \([^;{}]*!mbar_wait_bounded\([^;{}]*\)\)\s*(return false|break);")
    for name in ("gemm_core.cuh", "expert_gemm.cu", "fabric_device.cu", "attention.cu"):
        text = open(os.path.join(CSRC, name)).read()
        found = [m.group(0) for m in alone.finditer(text)]
        assert [f for f in found if "work_empty" not in f] == [], name
    attention = open(os.path.join(CSRC, "attention.cu")).read()
    assert not re.search(r"\(\*abort_flag\) break|&& \*abort_flag\) break", attention)
