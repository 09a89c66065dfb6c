"""The tensor-core kernels' TMA ring on the CPU: a producer fills the stages, two split groups take the
stages' uses in turn, the products free them.  An mbarrier's parity wait distinguishes a phase from its
predecessor only, and loads may land in any order; the model runs random schedules of the roles with the
waits of the kernels (ring_wait in csrc/tc_blocks8.cuh) and checks that a group splits the use it is meant to."""
import random
import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "bridct_b200" / "csrc"
CHUNKS = 40


class _Barrier:
    """phase: the current, incomplete one; a parity wait passes when the phase of that parity has completed."""

    def __init__(self):
        self.phase = 0

    def passed(self, parity):
        return (self.phase & 1) != parity


def _run(stages, guard, seed):
    """One random schedule; returns the first wrong split (chunk, stage content), None if all were right."""
    rng = random.Random(seed)
    full, free, a_full = ([_Barrier() for _ in range(stages)] for _ in range(3))
    content, loading, wrong = [None] * stages, [], []

    def producer():
        for j in range(CHUNKS):
            s, u = j % stages, j // stages
            while not free[s].passed((u & 1) ^ 1):
                yield
            loading.append(j)
            yield

    def memory():
        while True:
            if loading:
                j = loading.pop(rng.randrange(len(loading)) if rng.random() < 0.5 else 0)
                content[j % stages] = j
                full[j % stages].phase += 1
            yield

    def group(g):
        for j in range(g, CHUNKS, 2):
            s, u = j % stages, j // stages
            while guard and not free[s].passed((u & 1) ^ 1):
                yield
            while not full[s].passed(u & 1):
                yield
            if content[s] != j:
                wrong.append((j, content[s]))
                return
            yield
            a_full[s].phase += 1

    def products():
        for j in range(CHUNKS):
            s, u = j % stages, j // stages
            while not a_full[s].passed(u & 1):
                yield
            yield
            free[s].phase += 1

    roles = {"p": producer(), "m": memory(), "g0": group(0), "g1": group(1), "x": products()}
    for _ in range(200000):
        name = rng.choice(sorted(roles))
        if next(roles[name], "end") == "end":
            del roles[name]
            if wrong:
                return wrong[0]
            if set(roles) == {"m"}:
                return None
    raise AssertionError(f"{stages} stages: no progress")


@pytest.mark.parametrize("stages", [2, 3, 4, 5, 6])
def test_groups_split_the_use_they_wait_for(stages):
    for seed in range(200):
        assert _run(stages, stages % 2 == 1, seed) is None


def test_the_model_sees_what_the_guard_is_for():
    assert any(_run(3, False, seed) for seed in range(200))


def test_both_kernels_with_two_split_groups_wait_this_way():
    blocks, passes = ((CSRC / n).read_text() for n in ("tc_blocks8.cuh", "tc_pass.cuh"))
    body = blocks[blocks.index("bool ring_wait("):]
    body = body[:body.index("}\n")]
    assert re.search(r"STAGES % 2 && !mbar_wait\(stage_free, \(u & 1u\) \^ 1u\)\) return false", body)
    assert "return mbar_wait(stage_full, u & 1u);" in body
    for code in (blocks, passes):
        groups = code[code.index("} else if (warp >= 4 && warp < 12) {"):]
        groups = groups[:groups.index("} else if (warp >= 12)")]
        assert "ring_wait<kStages>(bars.stage_full + 8 * s, bars.stage_free + 8 * s" in groups
        assert not re.search(r"[^_]mbar_wait\(bars\.stage_full", groups)
