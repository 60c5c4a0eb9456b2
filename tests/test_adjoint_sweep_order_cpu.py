"""The exchange of the cooperative adjoint sweep (k_adj_sweep_umma) as a model on the host: four CTAs that each send every CTA
of the cluster one arrival a step, delivered in any order, to barriers that only count them.  A CTA may leave a step's wait
only when all four CTAs' arrivals of that step have reached it, whichever message is late."""
import itertools
import os
import re

from neuronbridge_gb300 import build

CTAS = 4


def _barriers_of_the_kernel():
    src = open(os.path.join(build.CSRC, "nbg_adjoint_tc.cu")).read()
    return int(re.search(r"constexpr int kExchangeBarriers = (\d+);", src).group(1))


def _sound(barriers, late, steps=6):
    """Everything runs as far as it can with the message `late` = (from, to, step) held back; then it is delivered.  False as
    soon as a CTA has left the wait of a step without all of its arrivals."""
    step = [0] * CTAS  # the step that each CTA waits in; its arrivals are sent on entry
    count = [[0] * barriers for _ in range(CTAS)]
    phase = [[0] * barriers for _ in range(CTAS)]
    got = [[set() for _ in range(steps + 1)] for _ in range(CTAS)]
    held, flying = [], [(c, d, 0) for c in range(CTAS) for d in range(CTAS)]

    def deliver(m):
        src, dst, j = m
        b = j % barriers
        got[dst][j].add(src)
        count[dst][b] += 1
        if count[dst][b] == CTAS:
            count[dst][b], phase[dst][b] = 0, phase[dst][b] + 1

    while True:
        moved = False
        while flying:
            m = flying.pop()
            (held.append if m == late else deliver)(m)
            moved = True
        for c in range(CTAS):
            j = step[c]
            # a parity wait: passes while the barrier is not in the phase waited for
            if j < steps and phase[c][j % barriers] % 2 != (j // barriers) % 2:
                if len(got[c][j]) != CTAS:
                    return False
                step[c] = j + 1
                flying += [(c, d, j + 1) for d in range(CTAS)] if j + 1 < steps else []
                moved = True
        if not moved:
            if not held:
                return all(j == steps for j in step)
            deliver(held.pop())


LATE = list(itertools.product(range(CTAS), range(CTAS), range(4)))


def test_no_arrival_stands_in_for_another():
    assert all(_sound(_barriers_of_the_kernel(), late) for late in LATE)


def test_the_model_tells_one_barrier_from_two():
    assert _sound(1, None) and not all(_sound(1, late) for late in LATE)
