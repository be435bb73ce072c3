"""The weight ring of the dequant-GEMM as a state machine: loads land in any order, groups of warps run at any pace, an mbarrier's parity wait passes iff the phase in progress has the
other parity.  With two full barriers a stage no group can take a unit that has not landed, and nothing stops; with one it can (units of a stage are taken by different groups, which do
not follow one another's phases), unless the stages are a multiple of the groups."""
import random

import pytest


def _run(stages, groups, units, barriers, rng):
    phase, emptied = [0] * barriers, [0] * stages
    issued, flying, landed, at = 0, [], set(), list(range(groups))
    while any(u < units for u in at):
        moves = [("land", u) for u in flying]
        if issued < units and (issued < stages or emptied[issued % stages] >= issued // stages):
            moves.append(("issue", issued))
        moves += [("take", g) for g in range(groups) if at[g] < units and (phase[at[g] % barriers] & 1) != (at[g] // barriers & 1)]
        if not moves:
            return "stuck"
        what, i = rng.choice(moves)
        if what == "issue":
            flying.append(i)
            issued += 1
        elif what == "land":
            flying.remove(i)
            phase[i % barriers] += 1
            landed.add(i)
        else:
            if at[i] not in landed:
                return "early"
            emptied[at[i] % stages] += 1
            at[i] += groups
    return "ok"


@pytest.mark.parametrize("stages,groups", [(3, 2), (4, 2), (5, 2), (3, 3), (4, 3), (5, 3), (6, 3), (7, 3), (8, 3)])
def test_two_full_barriers_a_stage(stages, groups):
    rng = random.Random(stages * 10 + groups)
    assert {_run(stages, groups, 50, 2 * stages, rng) for _ in range(200)} == {"ok"}
    one = {_run(stages, groups, 50, stages, rng) for _ in range(400)}
    assert ("early" in one) == (stages % groups != 0)
