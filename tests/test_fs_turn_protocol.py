"""CPU model of the full-space tile passes' stage (csrc/bk_lanczos.cuh, fs_turn_kernel):
one shared-memory tile, one mbarrier, task `it` waits for phase `it`. A run that gives up
must not leave while a copy is still on its way into the CTA's shared memory. The phases
that the kernel waits for are read from its source. No GPU is used."""
import os
import re

import pytest

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "bernasconi-krylov_b200", "csrc",
                   "bk_lanczos.cuh")


def _phases():
    """(the phase expressions of the task's own waits, that of the wait before leaving)"""
    with open(SRC) as f:
        body = f.read().split("fs_turn_kernel(const __grid_constant__ FtParams P) {")[1].split("\n}\n")[0]
    found = re.findall(r"mbar_wait_bounded\(fb, (.+?), P\.err\)", body)
    assert len(found) == 3
    return found[:2], found[2]


def _value(expr, it):
    return int(eval(expr.replace("1u", "1"), {"it": it}))


class Barrier:
    """An mbarrier for one copy a phase: `landed` of `issued` phases are complete."""

    def __init__(self):
        self.issued = self.landed = 0

    def complete(self, parity):
        """try_wait: the phase of this parity that precedes the incomplete one has completed."""
        return (self.landed & 1) != parity

    def wait(self, parity):
        """A bounded wait: the copies on their way land while it polls."""
        while not self.complete(parity):
            if self.landed == self.issued:
                return False
            self.landed += 1
        return True


@pytest.mark.parametrize("tasks", [1, 2, 3, 6])
def test_no_copy_is_in_flight_when_a_failed_run_leaves(tasks):
    own, leave = _phases()
    for failing in range(tasks):
        bar, left = Barrier(), False
        bar.issued = 1  # the first task's copy
        for it in range(tasks):
            if it == failing:
                # a counter's wait gave up before the load's (which is then skipped), or the
                # load's own did: the copy has not landed in either case
                left = True
            else:
                for expr in own:
                    assert bar.wait(_value(expr, it))
            if left:
                bar.wait(_value(leave, it))
                break
            bar.issued += 1
        assert left and bar.landed == bar.issued, (tasks, failing)
