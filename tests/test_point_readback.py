"""The current frame's level-0 points as they are read back (formed on the host from
the stored depths): the bits that the GPU gives them, infinite depths on the
principal point's column and row among them (0 times infinity)."""
import numpy as np
import pytest

import recon_gb300 as rg
from recon_gb300 import synth

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def test_level0_points_have_the_gpus_bits():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    W, H = 64, 48
    c = np.array(synth.make_calibration(W, H).calib, np.float32)
    KL = c[43:52]
    KL[2], KL[5] = 20.0, 17.0  # the principal point lies on a pixel
    near, far = float(c[62]), float(c[63])
    frame = np.full((H, W, 4), 0.5, np.float32)
    rng = np.random.default_rng(3)
    frame[..., 3] = rng.random((H, W))
    frame[rng.random((H, W)) < 0.05, 3] = np.inf
    frame[:, 20, 3] = np.inf
    frame[H - 1 - 17, ::3, 3] = np.inf  # rows are stored bottom-up
    frame[rng.random((H, W)) < 0.05, 3] = np.nan
    trk = rg.Tracker(rg.make_config(W, H, 1, iters=(1,), n_select=1024), c)
    trk.set_current_rgbd_float4(0, frame)
    got = trk.get_array(0, "cur_pts", 0, np.float32, 4 * W * H).reshape(H, W, 4)
    with np.errstate(invalid="ignore"):
        z = -(frame[::-1, :, 3] * (np.float32(far) - np.float32(near)) + np.float32(near))
        x, y = np.arange(W, dtype=np.float32)[None, :], np.arange(H, dtype=np.float32)[:, None]
        want = np.stack([(x - KL[2]) * z / KL[0], (y - KL[5]) * z / KL[4], z, np.ones_like(z)], -1).astype(np.float32)
        want[~(z < 0)] = 0.0
    bits = want.view(np.uint32)
    bits[np.isnan(want)] = 0x7FFFFFFF  # the NaN of a GPU operation
    assert np.isnan(want).sum() > 60
    assert np.array_equal(got.view(np.uint32), bits)
    trk.close()
