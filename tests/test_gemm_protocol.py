"""A host model of the operand ring's barriers as the MMA warp of the GEMM tiles sees them (gemm_mma in
monoserve_b200/csrc/gemm_core.cuh): the producer fills stages, every lane of the warp waits for a stage by the parity of its use, and one
lane frees it.  The lanes may run apart between the points where the warp meets; the model lets them, at random."""
import random

import pytest

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
    import os
    import re
    path = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "monoserve_b200", "csrc", "gemm_core.cuh")
    text = open(path).read()
    for name in ("gemm_mma_two", "gemm_mma"):
        body = text[re.search(rf"__device__ __forceinline__ bool {name}\(", text).start():]
        body = body[:body.index("\n}\n")]
        loop = body[body.index("for (int kt = 0;"):]
        assert re.search(r"mbar_wait_bounded\(&\w+(\.full)?\[pipe\.slot\][^;]*;\s*(//[^\n]*\s*)*__syncwarp\(\);", loop), name
        assert "break" not in loop, name   # a lane that leaves alone would leave the others waiting at the meeting
