"""acfd_autotune times what a step runs: on small FP64 grids whose brick stages
write their ghost copies themselves, the other variants with the fill that follows
them; with bodies, or a fill of formulas, every variant has the same fill and the
stages alone are timed.  The tuned step is no slower than the untuned one."""
import time

import pytest
import torch

from artracfd_b200 import abi, configs
from artracfd_b200.case import Boundary
from artracfd_b200.solver import Solver

pytestmark = pytest.mark.gpu
STAGES = 1 + 3 * abi.STAGE_VARIANTS * 5  # dt, and five stages a variant and axis


@pytest.mark.parametrize("walls", [False, True], ids=["copies", "formulas"])
def test_launches_of_the_tuner(walls):
    spec = configs.tgv(n=20)
    if walls:
        spec.boundaries = [Boundary(abi.NOSLIPWALL, (-1.0,))] * 2 + spec.boundaries[2:]
    part, model = spec.descriptors()
    with Solver(part, model, abi.FP64) as s:
        s.upload(spec.initial_nodes(part, model))
        s.treat_boundary(abi.TO)
        n = s.launches()
        s.autotune()
        fills = 0 if walls else 3 * (abi.STAGE_VARIANTS - abi.BRICK_VARIANTS) * 5
        assert s.launches() - n == STAGES + fills


def test_tuned_step_is_no_slower():
    spec = configs.tgv(n=32)
    part, model = spec.descriptors()
    node = spec.initial_nodes(part, model)

    def seconds(tune):
        with Solver(part, model, abi.FP64) as s:
            s.upload(node)
            s.treat_boundary(abi.TO)
            if tune:
                s.autotune()
            dt = 0.1 * s.time_step(0.5)
            s.evolve(dt, graph=True)
            best = 1.0
            for _ in range(6):
                torch.cuda.synchronize()
                t = time.perf_counter()
                for _ in range(20):
                    s.evolve(dt, graph=True)
                torch.cuda.synchronize()
                best = min(best, (time.perf_counter() - t) / 20)
        return best

    assert seconds(True) <= 1.1 * seconds(False)
