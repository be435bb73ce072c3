"""The weight ring of the dequant-GEMM as a state machine, over the stages and groups of every instance that is built: loads land in any order, each of a group's four warps runs at its own
pace, a stage is refilled when all four have handed it back, an A buffer is taken again when its products have been issued, an mbarrier's parity wait passes iff the phase in progress has
the other parity.  With two full barriers for a stage no warp takes a unit that has not landed or that has been overwritten, and nothing stops.  (A model of the waits in qmatmul_tc_kernel,
in the kernel's order: with one full barrier for a stage it finds a unit that is not there for 3 stages of 2 groups, and 4 or 5 of 3.)"""
import ctypes as C
import random

import pytest

import candle_vllm_b200 as pkg


class _Barrier:
    def __init__(self, count):
        self.count, self.left, self.phase = count, count, 0

    def arrive(self):
        self.left -= 1
        if self.left == 0:
            self.left, self.phase = self.count, self.phase + 1

    def passes(self, parity):
        return (self.phase & 1) != parity


def _run(stages, groups, units, rng):
    full = [_Barrier(1) for _ in range(2 * stages)]
    empty, ready, free = [_Barrier(4) for _ in range(stages)], [_Barrier(4) for _ in range(groups)], [_Barrier(1) for _ in range(groups)]
    held = [None] * stages                                  # unit whose bytes a stage has
    issued, issuing, flying = 0, 0, []                      # units loaded; products issued; loads on their way
    at = {(g, w): [g, "take"] for g in range(groups) for w in range(4)}
    while any(u < units for u, _ in at.values()) or issuing < units:
        moves = [("land", u) for u in flying]
        if issued < units and empty[issued % stages].passes((issued // stages & 1) ^ 1):
            moves.append(("load", issued))
        if issuing < units and ready[issuing % groups].passes(issuing // groups & 1):
            moves.append(("products", issuing))
        for who, (u, what) in at.items():
            if u < units and (full[u % (2 * stages)].passes(u // (2 * stages) & 1) if what == "take" else free[who[0]].passes((u // groups & 1) ^ 1)):
                moves.append((what, who))
        if not moves:
            return "stuck"
        what, i = rng.choice(moves)
        if what == "load":
            held[i % stages] = None
            flying.append(i)
            issued += 1
        elif what == "land":
            flying.remove(i)
            held[i % stages] = i
            full[i % (2 * stages)].arrive()
        elif what == "products":
            free[i % groups].arrive()
            issuing += 1
        else:
            u = at[i][0]
            if held[u % stages] != u:
                return "not there"
            if what == "take":
                at[i][1] = "store"
            else:                                           # (the second half of a row is read before the stage goes back)
                empty[u % stages].arrive()
                ready[i[0]].arrive()
                at[i] = [u + groups, "take"]
    return "ok"


def _rings():
    L = pkg.lib()
    n = L.qmatmul_weight_rings(None, C.c_int32(0))
    pairs = (C.c_int32 * (2 * n))()
    assert L.qmatmul_weight_rings(pairs, C.c_int32(n)) == n
    return sorted({(pairs[2 * i], pairs[2 * i + 1]) for i in range(n)})


def test_rings_of_the_kernel():
    rings = _rings()
    assert len(rings) >= 4 and all(3 <= stages <= 8 and groups in (2, 3) for stages, groups in rings)
    for stages, groups in rings:
        rng = random.Random(stages * 10 + groups)
        assert {_run(stages, groups, 40, rng) for _ in range(60)} == {"ok"}, (stages, groups)
