"""Refill of newly uncovered fluid nodes, bit for bit the oracle's on every node,
where they come in whole rows (a nearly flat face that moves along each axis),
where they lie deep (a body taken away, whose nodes search wide boxes) and where
they outnumber the room of the list (the bodies that stay are small).  And in about
the same time along every axis."""
import time

import numpy as np
import pytest
import torch

from artracfd_b200 import abi, configs
from artracfd_b200.solver import Solver
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu


def _sphere(centre, radius):
    P = abi.Polyhedron()
    P.faceN = P.edgeN = P.vertN = 0
    P.state, P.r = 0, radius
    P.T, P.cf, P.area = -1.0, 1.0, 4.0 * np.pi * radius * radius
    for s in range(3):
        P.O[s], P.V[s] = centre[s], 0.0
        P.box[s][0], P.box[s][1] = centre[s] - radius, centre[s] + radius
    return P


def _case(n, rng=None):
    """Crossflow in a box of n cells of size 1 a side, no bodies yet."""
    spec = configs.ib_spheres(n=n, level=1)
    spec.bodies = []
    spec.domain_lo, spec.domain_hi = (0.0, 0.0, 0.0), (float(n),) * 3
    part, model = spec.descriptors()
    node = spec.initial_nodes(part, model)
    if rng is not None:
        inner = node["did"] == 0
        lev = node["U"][:, 0, :].copy()
        lev[inner] *= rng.uniform(0.95, 1.05, (int(inner.sum()), 1))
        node["U"][:, 0, :] = lev
    return part, model, node


def _flat(n, axis, at):
    c = [0.5 * n] * 3
    c[axis] = at - 400.0
    return _sphere(c, 400.0)


MOVES = {
    "flat x": lambda n: ([_flat(n, 0, 9.4)], [_flat(n, 0, 8.3)]),
    "flat y": lambda n: ([_flat(n, 1, 9.4)], [_flat(n, 1, 8.3)]),
    "flat z": lambda n: ([_flat(n, 2, 9.4)], [_flat(n, 2, 8.3)]),
    "taken away": lambda n: ([_sphere((12.0, 12.0, 12.0), 6.2)], [_sphere((19.0, 19.0, 19.0), 2.5)]),
    "two small ones left": lambda n: ([_sphere((11.0, 12.0, 13.0), 9.1)],
                                      [_sphere((4.0, 4.0, 4.0), 1.6), _sphere((19.5, 4.0, 19.5), 1.6)]),
}


@pytest.mark.parametrize("move", MOVES)
def test_refill_is_the_oracles(move):
    n = 24
    part, model, node = _case(n, np.random.default_rng(7))
    before, after = MOVES[move](n)
    orc = Oracle()
    want = node.copy()
    orc.compute_geometric_field(want, part, model, before)
    covered = want["did"] > 0
    orc.compute_geometric_field(want, part, model, after)
    assert (covered & (want["did"] == 0)).sum() > 300
    with Solver(part, model, abi.FP64_EXACT) as s:
        s.upload(node)
        s.geo_upload(before)
        s.compute_geometric_field()
        s.geo_upload(after)
        s.compute_geometric_field()
        got = s.download()
    for f in ("did", "fid", "lid", "gst"):
        assert np.array_equal(got[f], want[f]), f
    assert np.array_equal(got["U"][:, 0, :], want["U"][:, 0, :])


def test_direction_of_the_motion_costs_nothing():
    """A face that uncovers a plane of 128 x 128 nodes, back and forth along x (one
    node a row) and along z (whole rows): a warp that takes its own rows' nodes one
    after the other took three times as long along z."""
    n = 128
    part, model, node = _case(n)
    best = {}
    for axis in (0, 2):
        with Solver(part, model, abi.FP64) as s:
            s.upload(node)
            took = []
            for k in range(14):
                s.geo_upload([_flat(n, axis, 40.2 if k % 2 == 0 else 39.3)])
                torch.cuda.synchronize()
                t = time.perf_counter()
                s.compute_geometric_field()
                torch.cuda.synchronize()
                if k % 2 and k > 2:
                    took.append(time.perf_counter() - t)
            best[axis] = min(took)
    assert best[2] <= 1.6 * best[0]
