"""Batches whose instances run different parts of the schedule, in one group of
launches: photometric instances of three levels beside ICP instances that have
fewer levels, or no iteration at one of them.  A kernel is launched only where an
instance runs it (a launch that no CTA waits in would break the order of the
launches around it), and every replay gives the oracle's poses."""
import numpy as np
import pytest

import recon_gb300 as rg
from scenes import frame_pair
from test_gpu_parity import assert_bitexact, run_pair

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

CASES = [
    # size; levels and iterations (coarse to fine) of the ICP instances; ICP preparation
    # launches and Gauss-Newton iterations of a group of one photometric and one ICP instance
    (160, 120, 1, (4, 0, 0, 0), 1, 3 + 3 + 4),
    (320, 240, 1, (2, 0, 0, 0), 4, 3 + 3 + 2),
    (320, 240, 3, (2, 0, 2, 0), 5, 3 + 3 + 2),
    (160, 120, 3, (0, 4, 0, 0), 1, 3 + 4 + 2),
]


@pytest.mark.parametrize("W,H,L,icp_iters,prepare,iterations", CASES)
@pytest.mark.parametrize("mode", [rg.GEOMETRIC, rg.BIOBJECTIVE])
def test_levels_that_only_some_instances_run(W, H, L, icp_iters, prepare, iterations, mode):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    n = 8  # four groups of two instances
    pair = frame_pair(W, H, 3, seed=W + L, deg=1.5, mm=15.0)
    kinds = [(rg.PHOTOMETRIC, 3, (3, 3, 2, 0)), (mode, L, icp_iters)]
    cfgs = [rg.make_config(W, H, kinds[i % 2][1], mode=kinds[i % 2][0], iters=kinds[i % 2][2], n_select=2048)
            for i in range(n)]
    b = rg.Batch(cfgs, [pair.cal.calib] * n)
    b.set_reference([pair.g0] * n, [pair.d0] * n)
    b.set_current([pair.g1] * n, [pair.d1] * n)
    start = np.tile(np.eye(4, dtype=np.float32), (n, 1, 1))
    want = []
    for m, levels, iters in kinds:
        p = frame_pair(W, H, levels, seed=W + L, deg=1.5, mm=15.0)
        want.append(run_pair(p, m, iters=iters, n_select=2048)[4])
    first = rg.launch_count()
    for r in range(20):
        T, st = b.track(start)
        for i in range(n):
            assert_bitexact(T[i], want[i % 2], f"pose of instance {i}, replay {r}")
            assert st[i].status == rg.OK and st[i].solves == sum(kinds[i % 2][2]), (i, r)
        if r == 0:
            launched = rg.launch_count() - first
    for i in range(n):
        b.set_iterations(i, (0, 0, 0, 0))
    first = rg.launch_count()
    b.track(start)
    launched -= rg.launch_count() - first  # those around the schedule
    assert launched == 4 * (prepare + 2 * iterations)
    b.close()
