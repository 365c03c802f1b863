"""FP64 steps whose stages write their ghost copies themselves: the copies are
exact, so a step equals, bit for bit on every node and level, the step of the
ordered fill launches (ACFD_BC_PHASES), eager and captured, on the brick kernels
(which do so) and beside line-march sweeps (which do not), for grids whose copies
overlap at edges and corners, also where nodes inside the domain are not fluid."""
import numpy as np
import pytest

from artracfd_b200 import abi, configs
from artracfd_b200.case import Boundary
from artracfd_b200.solver import Solver

pytestmark = pytest.mark.gpu
P, O = Boundary(abi.PERIODIC), Boundary(abi.OUTFLOW)
FACES = {"periodic": [P] * 6, "outflow": [O] * 6, "mixed": [O, O, P, P, O, O]}


@pytest.mark.parametrize("tiles", [[0] * 3, [1] * 3, [5] * 3, [0, 5, 8], [8, 1, 0]], ids=str)
@pytest.mark.parametrize("faces", FACES)
@pytest.mark.parametrize("viscous", [True, False], ids=["viscous", "inviscid"])
def test_step_equals_the_step_of_the_ordered_fill(viscous, faces, tiles, monkeypatch):
    spec = configs.tgv(n=8) if viscous else configs.sod()
    spec.m = (23, 9, 6)
    spec.regions = []
    spec.boundaries = FACES[faces]
    part, model = spec.descriptors()
    node = spec.initial_nodes(part, model)
    rng = np.random.default_rng(5)
    inner = node["did"] == 0
    lev = node["U"][:, 0, :].copy()
    lev[inner, 0] *= rng.uniform(0.9, 1.1, int(inner.sum()))
    node["U"][:, 0, :] = lev
    node["did"][np.flatnonzero(inner)[::37]] = 1  # nodes that no stage updates
    out = []
    for env in ("", "ACFD_BC_PHASES"):
        if env:
            monkeypatch.setenv(env, "1")
        for graph in (False, True):
            with Solver(part, model, abi.FP64) as s:
                s.upload(node)
                s.treat_boundary(abi.TO)
                s.set_tiles(tiles)
                before = s.launches()
                for _ in range(2):
                    s.evolve(0.3 * s.time_step(1.0), graph=graph)
                launches = s.launches() - before
                out.append(s.download()["U"].copy())
        if not env and max(tiles) < 2:
            assert launches < 2 * 25
    for u in out[1:]:
        assert np.array_equal(u, out[0])
