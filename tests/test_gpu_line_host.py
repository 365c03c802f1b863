"""Queueing a step of line-march launches costs the host no more on long lines
than on short ones: the tile and the cuts of a launch are found once per case."""
import time

import pytest
import torch

from artracfd_b200 import abi, configs
from artracfd_b200.case import Boundary
from artracfd_b200.solver import Solver

pytestmark = pytest.mark.gpu


def _queue_seconds(cells):
    spec = configs.sod(m=cells)
    spec.regions = []
    spec.boundaries = [Boundary(abi.OUTFLOW)] * 6
    part, model = spec.descriptors()
    with Solver(part, model, abi.FP64) as s:
        s.upload(spec.initial_nodes(part, model))
        s.treat_boundary(abi.TO)
        s.set_tiles([abi.PLANE_VARIANT] * 3)
        dt = 0.1 * s.time_step(0.5)
        best = 1.0
        for _ in range(20):
            torch.cuda.synchronize()
            t = time.perf_counter()
            s.evolve(dt, graph=False)
            best = min(best, time.perf_counter() - t)
        torch.cuda.synchronize()
    return best


@pytest.mark.parametrize("axis", [0, 1, 2])
def test_queueing_a_step_does_not_grow_with_the_lines(axis):
    """Six stages, six fills and the set of dt either way: the host's time is that
    of 13 launches.  Three times allows for a busy host; the searches for tiles of
    300,000 cells took more than ten times as long."""
    short, long_ = [1, 1, 1], [1, 1, 1]
    short[axis], long_[axis] = 300, 300_000
    assert _queue_seconds(tuple(long_)) <= 3.0 * _queue_seconds(tuple(short))
