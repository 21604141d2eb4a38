"""Rings of packed weights that two groups of consumers take in turn (csrc/grouped_gemm.cu): no wait may be over before the data it is for has arrived,
in whatever order copies end."""
import os
import random
import re

import pytest

SOURCE = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "krasis_b200", "csrc", "grouped_gemm.cu")
DEPTHS = {m.group(1): int(m.group(2)) for m in re.finditer(r"struct Fmt<(\w+)> \{[^}]*kStagesW = (\d+);", open(SOURCE).read())}


def _wrong_reads(blocks, stages, per_stage, seed):
    """K blocks pass through a ring of `stages` stages of per_stage blocks each; group kb % 2 consumes block kb.  Barriers as the hardware has them: a
    wait for a parity is over when the barrier's current phase has the other one.  Returns how often a group read a stage that did not hold its block."""
    rng = random.Random(seed)
    full, empty = [0] * stages, [0] * stages                  # completed phases
    left = [per_stage] * stages                               # consumers of the stage that have not freed it in this phase
    holds, inflight = [None] * stages, []                     # (stage, load)
    made, at, wrong = 0, [0, 1], 0                            # next load; next block of each group
    loads = blocks // per_stage
    for _ in range(100000):
        if made == loads and not inflight and all(a >= blocks for a in at):
            return wrong
        who = rng.randrange(4)
        if who == 0 and made < loads:
            st, n = made % stages, made // stages
            if empty[st] % 2 != ((n & 1) ^ 1):                # waits for parity (n & 1) ^ 1
                inflight.append((st, made))
                made += 1
        elif who == 1 and inflight:                           # any copy may end next
            st, load = inflight.pop(rng.randrange(len(inflight)))
            holds[st] = load
            full[st] += 1
        elif who >= 2 and at[who - 2] < blocks:
            kb = at[who - 2]
            load = kb // per_stage
            st, n = load % stages, load // stages
            if full[st] % 2 != (n & 1):                       # waits for parity n & 1
                if holds[st] != load or full[st] != n + 1:
                    return wrong + 1                          # the counts no longer mean anything from here on
                at[who - 2] += 2
                left[st] -= 1
                if left[st] == 0:
                    left[st] = per_stage
                    empty[st] += 1
    return wrong + 1                                          # nobody gets on


@pytest.mark.parametrize("fmt", sorted(DEPTHS))
def test_two_groups_take_blocks_in_turn(fmt):
    depth = DEPTHS[fmt]
    per_stage = 2 if depth >= 4 else 1
    for seed in range(200):
        assert _wrong_reads(24, depth // per_stage, per_stage, seed) == 0, (fmt, depth, seed)


def test_an_odd_ring_is_found():
    """What the check above is about: three stages of single blocks."""
    assert len(DEPTHS) == 5 and any(_wrong_reads(24, 3, 1, seed) for seed in range(200))
