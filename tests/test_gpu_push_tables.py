"""The tables of ghost copies that the FP64 brick stages write are built for the
first step that uses them: a case on other kernels never holds them, one that is
given the brick kernels later does from its next step on, with the same bits."""
import numpy as np
import pytest
import torch

from artracfd_b200 import abi, configs
from artracfd_b200.solver import Solver

pytestmark = pytest.mark.gpu


def test_tables_come_with_the_first_step_that_uses_them():
    spec = configs.tgv(n=48)  # four tables of 166,000 nodes: 2.7 MB, more than one 2 MB page
    part, model = spec.descriptors()
    node = spec.initial_nodes(part, model)

    def held(tiles):
        with Solver(part, model, abi.FP64) as s:
            s.upload(node)
            s.treat_boundary(abi.TO)
            s.set_tiles([abi.PLANE_VARIANT] * 3)
            dt = 0.1 * s.time_step(0.5)
            s.evolve(dt)
            torch.cuda.synchronize()
            before = torch.cuda.mem_get_info()[0]
            s.set_tiles(tiles)
            n = s.launches()
            s.evolve(dt)
            torch.cuda.synchronize()
            return before - torch.cuda.mem_get_info()[0], s.launches() - n, s.download()["U"].copy()

    line, n_line, u_line = held([abi.PLANE_VARIANT] * 3)
    brick, n_brick, u_brick = held([0, 0, 0])
    assert line == 0 and n_line == 37
    assert brick >= 1 << 21 and n_brick == 19
    assert np.allclose(u_line, u_brick, rtol=0, atol=1e-9 * np.abs(u_line).max())
