"""The stage variants that the FP64 form starts on: a step on them takes no longer
than the step on the first brick (which every grid ran on before the line march),
on grids that leave the line march's lanes empty -- planes, lines, thin rods and
unsplit sweeps -- as on those that fill them.  A quarter is allowed for noise; with
the line march on every axis from 131,072 nodes, five of these grids took 1.3 to 15
times as long."""
import time

import pytest
import torch

from artracfd_b200 import abi, configs
from artracfd_b200.case import Boundary
from artracfd_b200.solver import Solver

pytestmark = pytest.mark.gpu
GRIDS = [((512, 512, 1), 0, False), ((400, 1, 400), 0, False), ((1, 200000, 1), 0, False), ((1, 1, 200000), 0, False),
         ((12, 20000, 1), 0, False), ((128, 4096, 1), 0, False), ((4, 9000, 5), 0, False), ((128, 128, 128), 1, True),
         ((64, 64, 64), 1, False), ((200000, 1, 1), 0, False), ((1, 600, 600), 0, False), ((96, 96, 96), 0, True),
         ((700, 300, 2), 0, False), ((700, 300, 2), 1, True)]


def _step_seconds(part, model, node, tiles):
    with Solver(part, model, abi.FP64) as s:
        s.upload(node)
        s.treat_boundary(abi.TO)
        if tiles is not None:
            s.set_tiles(tiles)
        dt = 0.1 * s.time_step(0.5)
        s.evolve(dt, graph=True)
        best = 1.0
        for _ in range(4):
            torch.cuda.synchronize()
            t = time.perf_counter()
            for _ in range(6):
                s.evolve(dt, graph=True)
            torch.cuda.synchronize()
            best = min(best, (time.perf_counter() - t) / 6)
    return best


@pytest.mark.parametrize("cells,multidim,viscous", GRIDS, ids=[f"{g[0]}-{g[1]}" for g in GRIDS])
def test_defaults_are_no_slower_than_the_brick(cells, multidim, viscous):
    spec = configs.tgv(n=8) if viscous else configs.sod()
    spec.m = cells
    spec.domain_lo, spec.domain_hi = (0.0, 0.0, 0.0), tuple(c / 64.0 for c in cells)
    spec.regions = []
    spec.multidim = multidim
    spec.boundaries = [Boundary(abi.PERIODIC if viscous else abi.OUTFLOW)] * 6
    part, model = spec.descriptors()
    node = spec.initial_nodes(part, model)
    assert _step_seconds(part, model, node, None) <= 1.25 * _step_seconds(part, model, node, [0, 0, 0])
