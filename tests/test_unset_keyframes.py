"""Instances of a batch that have not been given a keyframe: they take part in
the launches, have no point to match, and keep their pose, wherever it lies."""
import numpy as np
import pytest

import recon_gb300 as rg
from scenes import frame_pair
from test_gpu_parity import assert_bitexact, run_pair

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("W,H,L", [(90, 70, 2), (320, 240, 2)])
@pytest.mark.parametrize("mode", [rg.GEOMETRIC, rg.BIOBJECTIVE])
@pytest.mark.parametrize("solver", [rg.SOLVER_CHOLESKY, rg.SOLVER_CG])
def test_instance_without_keyframe_keeps_its_pose(W, H, L, mode, solver):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    pair = frame_pair(W, H, L, seed=17, deg=1.0, mm=10.0)
    iters = (2, 2)
    cfg = rg.make_config(W, H, L, mode=mode, iters=iters, n_select=1024, solver=solver)
    b = rg.Batch([cfg] * 3, [pair.cal.calib] * 3)
    b.set_reference([None, pair.g0, None], [None, pair.d0, None])
    b.set_current([pair.g1] * 3, [pair.d1] * 3)
    # a keyframe of zeros would project its one point to the middle of the image
    far = np.eye(4, dtype=np.float32)
    far[:3, 3] = (3.0, -2.0, -700.0)
    start = np.stack([far, np.eye(4, dtype=np.float32), np.eye(4, dtype=np.float32)])
    T, st = b.track(start)
    for i in (0, 2):
        assert_bitexact(T[i], start[i], f"pose of instance {i}")
        assert (st[i].iterations, st[i].solves, st[i].non_spd) == (4, 0, 0), i
        assert list(st[i].icp_selected) == [0, 0, 0, 0] and st[i].status == rg.ERR_NOT_ENOUGH_POINTS, i
    _, _, _, _, To, _ = run_pair(pair, mode, solver=solver, iters=iters, n_select=1024)
    assert_bitexact(T[1], To, "pose of the instance with a keyframe")
