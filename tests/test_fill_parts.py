"""The part of a ghost fill that a stage reads (GhostReads in
csrc/ghost_tasks.h, compiled here for the host): one stage of the oracle on a
state whose other ghost nodes are NaN gives the bits of the stage on the whole
fill, and every ghost node of the part is read (without it the stage's result
holds a NaN)."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from artracfd_b200 import abi, configs
from artracfd_b200.case import Boundary
from oracle.oracle import Oracle

_HARNESS = r"""
#include <cstdio>
#include <cstdlib>
#include "ghost_tasks.h"
int main(int argc, char **argv)
{
    int a[14];
    for (int q = 0; q < 14; ++q) a[q] = std::atoi(argv[q + 1]);  // n[3] lo[3] hi[3] s half viscous pitch (unused)
    const long long total = (long long)a[0] * a[1] * a[2];
    GhostReads reads(a[0], a[1], a + 3, a + 6, a[10], a[11]);
    for (int q = 0; q < total; ++q) std::putchar(reads(q) >> a[9] & 1);
    return 0;
}
"""
P, O, W = Boundary(abi.PERIODIC), Boundary(abi.OUTFLOW), Boundary(abi.NOSLIPWALL, (-1.0,))


@pytest.fixture(scope="module")
def harness(tmp_path_factory):
    gxx = shutil.which("g++")
    if gxx is None:
        pytest.skip("no host C++ compiler")
    d = tmp_path_factory.mktemp("parts")
    (d / "parts.cpp").write_text(_HARNESS)
    csrc = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "artracfd_b200", "csrc")
    subprocess.run([gxx, "-O2", "-std=c++17", "-I" + csrc, str(d / "parts.cpp"), "-o", str(d / "parts")], check=True)
    return str(d / "parts")


@pytest.mark.parametrize("s", [0, 1, 2])
@pytest.mark.parametrize("weno5", [True, False], ids=["weno5", "weno3"])
@pytest.mark.parametrize("viscous", [True, False], ids=["viscous", "inviscid"])
def test_part_of_the_fill_is_what_the_stage_reads(harness, viscous, weno5, s):
    spec = configs.tgv(n=8) if viscous else configs.sod()
    spec.m = (9, 7, 6)
    spec.sScheme = int(weno5)
    spec.regions = []
    spec.boundaries = [O, O, P, P, W, W]
    part, model = spec.descriptors()
    node = spec.initial_nodes(part, model)
    rng = np.random.default_rng(s)
    n = [int(v) for v in part.n]
    lo, hi = ([int(part.ns[0][t][q]) for t in range(3)] for q in range(2))
    U = np.empty((node.size, 5))
    U[:, 0] = rng.uniform(0.8, 1.2, node.size)
    U[:, 1:4] = rng.uniform(-0.2, 0.2, (node.size, 3))
    U[:, 4] = rng.uniform(200.0, 210.0, node.size)
    shape = (n[2], n[1], n[0])
    inner = np.zeros(shape, dtype=bool)
    inner[lo[2]:hi[2], lo[1]:hi[1], lo[0]:hi[0]] = True
    out = subprocess.run([harness] + [str(v) for v in (*n, *lo, *hi, s, 3 if weno5 else 2, int(viscous), n[0], 0)],
                         check=True, capture_output=True).stdout
    read = np.frombuffer(out, dtype=np.uint8).astype(bool).reshape(shape)
    assert read[inner].all()
    orc = Oracle()

    def stage(keep):
        nd = node.copy()
        lev = U.copy()
        lev[~keep.ravel()] = np.nan
        nd["U"][:, 0, :] = lev
        orc.lllu(nd, part, model, 1e-4, 0.0, 1.0, abi.TO, abi.TO, abi.TN, s)
        return nd["U"][inner.ravel(), 1, :]

    whole = stage(np.ones(shape, dtype=bool))
    assert np.isfinite(whole).all()
    assert np.array_equal(stage(read), whole)
    ghosts = np.argwhere(read & ~inner)
    for g in ghosts[rng.choice(len(ghosts), 12, replace=False)]:
        less = read.copy()
        less[tuple(g)] = False
        assert not np.isfinite(stage(less)).all(), g
