"""The X half steps of a batch as Y sweeps of the transposed states.

A batch of all-viscous (or all-inviscid) cases whose ghost fills are copies sweeps
x with the Y plane-march launch on transposed levels of every case.  The
discretisation is that of the X launch in another compiled kernel, so the two agree
to FP32 round-off, on grids whose extents all differ and are no multiple of a
32-node tile; ACFD_X_TRANSPOSE=0 at the batch's creation keeps the X launch.  The
cases' own handles keep the X sweep.
"""
import dataclasses

import numpy as np
import pytest

from artracfd_b200 import abi, configs
from artracfd_b200.batch import Batch

from test_gpu_march import TOL_FP32_ORDER, _const_sensor
from test_gpu_parity import rel_err

pytestmark = pytest.mark.gpu


def _specs(tScheme, viscous):
    rng = np.random.default_rng(3)
    if not viscous:
        out = [configs.sod(m=(33, 6, 4)), configs.sod(m=(20, 9, 5))]
    else:
        out = [dataclasses.replace(configs.tgv(n=16, Re=800.0, Ma=0.2, stepN=0), m=(40, 28, 20)),
               dataclasses.replace(configs.riemann_viscous(n=16, Re=1000.0, Ma=0.3, rng=rng), m=(9, 37, 12)),
               dataclasses.replace(configs.tgv(n=16, Re=1200.0, Ma=0.3, stepN=0), m=(25, 16, 33))]
    return [dataclasses.replace(s, tScheme=tScheme) for s in out]


def _run(specs, params, steps, calls=1):
    descs = [s.descriptors() for s in specs]
    with Batch(descs) as b:
        for c, spec in enumerate(specs):
            b.upload(c, spec.initial_nodes(*descs[c]))
            b.treat_boundary(c)
        if params is not None:
            b.sensor_load(params, 0.5)
        b.set_precision(abi.FP32_BULK if params is None else abi.FP32_HYBRID)
        n0 = b.launches()
        dts = np.concatenate([b.advance([s.cfl for s in specs], steps) for _ in range(calls)])
        n = b.launches() - n0
        return dts, [b.download(c)["U"].copy() for c in range(len(specs))], n


@pytest.mark.parametrize("form", ["all", "none", "fp32"])
@pytest.mark.parametrize("tScheme,viscous", [(1, True), (0, True), (1, False)])
def test_batch_transposed_x_matches_x_launch(form, tScheme, viscous, monkeypatch):
    specs = _specs(tScheme, viscous)
    params = None if form == "fp32" else _const_sensor(50.0 if form == "all" else -50.0)
    monkeypatch.setenv("ACFD_X_TRANSPOSE", "0")
    rdts, ref, rn = _run(specs, params, 3)
    monkeypatch.setenv("ACFD_X_TRANSPOSE", "1")
    dts, got, n = _run(specs, params, 3)
    one, again, _ = _run(specs, params, 1, calls=3)
    assert n == rn + 3 * (2 if form == "fp32" else 3)
    assert np.array_equal(dts[0], rdts[0])
    assert np.array_equal(dts, one)
    for c in range(len(specs)):
        for lev in range(3):  # ghosts included, on all three levels
            err = rel_err(got[c][:, lev], ref[c][:, lev])
            assert err <= TOL_FP32_ORDER, (c, lev, err)
        assert np.array_equal(got[c], again[c])
