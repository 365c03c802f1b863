"""The transposed levels that a batch holds to be faster are the library's to give
back: a case that fits only without them is created all the same, and the batch goes
on with the X sweep, also while another thread advances it.  The sizes leave 50 MB
and more on either side of what is asserted; nothing but allocations is near the
device's limit."""
import threading

import pytest
import torch

from artracfd_b200 import abi, configs
from artracfd_b200.batch import Batch
from artracfd_b200.solver import Solver

from test_gpu_march import TOL_FP32_ORDER
from test_gpu_parity import rel_err

pytestmark = pytest.mark.gpu
MB = 1 << 20


def _batch(spec):
    desc = spec.descriptors()
    b = Batch([desc])
    b.upload(0, spec.initial_nodes(*desc))
    b.treat_boundary(0)
    return b


@pytest.mark.parametrize("threaded", [False, True], ids=["between steps", "during steps"])
def test_levels_go_back_when_a_case_needs_the_memory(threaded):
    spec, large = configs.tgv(n=96, Re=800.0, Ma=0.2, stepN=0), configs.tgv(n=120)
    with _batch(spec) as b:  # loads the kernels, and what a batch with the levels holds
        b.advance([spec.cfl], 8)
        whole = b.download(0)["U"][:, 0, :].copy()
    with Solver(*large.descriptors()):
        pass
    hog = torch.empty(torch.cuda.mem_get_info()[0] - 660 * MB, dtype=torch.uint8, device="cuda")
    try:
        with _batch(spec) as b:  # 150 MB of state, 142 of records, 139 transposed
            n = b.launches()
            b.advance([spec.cfl], 1)
            assert b.launches() - n == 40  # CFL, dt, 18 stages and fills, two transposes
            left = torch.cuda.mem_get_info()[0]
            assert left < 260 * MB  # a case of 120^3 takes 281
            t = threading.Thread(target=b.advance, args=([spec.cfl], 7))
            if threaded:
                t.start()
            try:
                with Solver(*large.descriptors()) as s:
                    assert s.node_count > 0
                    if not threaded:
                        n = b.launches()
                        b.advance([spec.cfl], 7)
                        assert b.launches() - n == 7 * 38
            finally:
                if threaded:
                    t.join()
            b.advance([spec.cfl], 0)
            got = b.download(0)["U"][:, 0, :].copy()
            assert not b.transposed()
    finally:
        del hog
        torch.cuda.empty_cache()
    assert rel_err(got, whole) <= 8 * TOL_FP32_ORDER
