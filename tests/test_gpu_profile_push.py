"""acfd_profile_step runs the step that acfd_evolve_fluid runs, also on small FP64
grids whose stages write their ghost copies themselves: the same launches and bits,
a piece per stage and no fill pieces; where one axis is on a march, that axis alone
has fills."""
import numpy as np
import pytest

from artracfd_b200 import abi, configs
from artracfd_b200.solver import Solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tiles", [[0, 0, 0], [1, 0, abi.PLANE_VARIANT], [abi.PLANE_VARIANT] * 3], ids=str)
def test_profiled_step_is_the_step(tiles):
    spec = configs.sod(m=(40, 9, 7))
    part, model = spec.descriptors()
    node = spec.initial_nodes(part, model)
    got = []
    for profiled in (False, True):
        with Solver(part, model, abi.FP64) as s:
            s.upload(node)
            s.treat_boundary(abi.TO)
            s.set_tiles(tiles)
            dt = s.time_step(spec.cfl)
            n = s.launches()
            pieces = s.profile_step(dt) if profiled else s.evolve(dt)
            got.append((s.launches() - n, s.download()["U"].copy()))
    want = []
    for ax in (2, 1, 0, 0, 1, 2):
        for q in range(3):
            want.append((abi.PIECE_STAGE, ax, q))
            if tiles[ax] >= abi.BRICK_VARIANTS:
                want.append((abi.PIECE_FILL, ax, q))
    assert [p[:3] for p in pieces] == want
    assert got[0][0] == got[1][0]
    assert np.array_equal(got[0][1], got[1][1])
