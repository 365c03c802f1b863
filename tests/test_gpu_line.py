"""FP64 line-march stage kernels (variants from PLANE_VARIANT on) at the edges
of their tiles: extents just above and below a tile's width and rows, lines of
a few nodes, lines longer than a tile, segments of one plane, several items per
block.  One time step from the same state on the oracle (the reference's
operations in the reference's order), within the FP64 form's bound per step
(1e-12 of the magnitude of each conservative variable)."""
import numpy as np
import pytest

from artracfd_b200 import abi, configs
from artracfd_b200.case import Boundary
from artracfd_b200.solver import Solver
from oracle.oracle import Oracle

from test_gpu_parity import TOL_STEP, rel_err

pytestmark = pytest.mark.gpu

P, O = Boundary(abi.PERIODIC), Boundary(abi.OUTFLOW)
# cells along x, y, z
SIZES = [(4, 4, 4), (18, 12, 13), (22, 33, 5), (127, 3, 9), (260, 5, 4), (33, 70, 37), (5, 64, 65)]


@pytest.fixture(scope="module")
def orc():
    return Oracle()


def _case(m, viscous, weno5, rng):
    spec = configs.tgv(n=8) if viscous else configs.sod()
    spec.m = m
    spec.domain_lo, spec.domain_hi = (0.0, 0.0, 0.0), (1.0, 0.9, 1.1)
    spec.sScheme = int(weno5)
    spec.regions = []
    spec.boundaries = [O, O, P, P, P, P] if m[0] % 2 else [P, P, O, O, P, P]
    part, model = spec.descriptors()
    node = spec.initial_nodes(part, model)
    inner = node["did"] == 0
    k = int(inner.sum())
    rho = rng.uniform(0.6, 1.6, k)
    v = rng.uniform(-0.4, 0.4, (k, 3))
    p = rng.uniform(0.7, 1.4, k) * (70.0 if viscous else 1.0)
    U = np.empty((k, 5))
    U[:, 0] = rho
    U[:, 1:4] = rho[:, None] * v
    U[:, 4] = 0.5 * rho * (v * v).sum(axis=1) + p / (model.gamma - 1.0)
    lev = node["U"][:, 0, :].copy()
    lev[inner] = U
    node["U"][:, 0, :] = lev
    return part, model, node


@pytest.mark.parametrize("scheme", ["weno5", "weno3"])
@pytest.mark.parametrize("viscous", [True, False], ids=["viscous", "inviscid"])
@pytest.mark.parametrize("m", SIZES, ids=["x".join(map(str, m)) for m in SIZES])
def test_line_kernels_at_tile_edges(m, viscous, scheme, orc):
    part, model, node = _case(m, viscous, scheme == "weno5", np.random.default_rng(sum(m)))
    want = node.copy()
    orc.treat_boundary(want, part, model, abi.TO)
    got = []
    for v in (abi.PLANE_VARIANT, abi.PLANE_VARIANT + 2, abi.PLANE_SHARE_VARIANT, abi.PLANE_SHARE_VARIANT + 2):
        with Solver(part, model, abi.FP64) as s:
            s.upload(node)
            s.treat_boundary(abi.TO)
            s.set_tiles([v] * 3)
            dt = 0.2 * s.time_step(1.0)
            s.evolve(dt)
            got.append(s.download()["U"][:, 0, :].copy())
    orc.evolve_fluid(want, part, model, dt)
    for u in got:
        assert rel_err(u, want["U"][:, 0, :]) <= TOL_STEP
        assert np.array_equal(u, got[0])
