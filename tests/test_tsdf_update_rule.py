"""Which grids list the blocks that an update visits: those on which the two
launches more are paid back on a single grid.  Counted on both sides of the line,
and the listed update against the CPU oracle at the first size that takes it: a
last tile that is cut off, image edges inside a tile, a camera in the grid, and
missing, infinite and NaN distances."""
import numpy as np
import pytest

import oracle_lib as O
import recon_gb300 as rg

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

K = np.array([0.9, 0, 0.5, 0, -1.2, 0.5, 0, 0, 1], np.float32)
LISTED = 328  # 11 x 41 x 41 blocks; the last of 11 tiles along x has 8 of 32 voxels


def distances(W, H, dim, rng, view):
    y, x = np.mgrid[0:H, 0:W]
    dist = (dim * (1.1 + 0.08 * np.sin(x / 40.0) * np.cos(y / 30.0) + 0.25 * (x > W // 2))).astype(np.float32)
    dist[rng.random((H, W)) < 0.02] = 0.0
    if view == "nan":
        dist[H // 3: H // 3 + 9, W // 4: W // 4 + 9] = np.nan
        dist[H // 2, W // 2] = np.inf
    return dist


@pytest.mark.parametrize("R,launches", [(64, 1), (256, 1), (320, 1), (LISTED, 3)])
def test_launches_of_an_update(R, launches):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    v = rg.TSDF(rg.tsdf_params(R, 83, 61))
    v.set_dist_map(distances(83, 61, 1750.0, np.random.default_rng(R), "room"))
    before = rg.launch_count()
    v.update(np.eye(4, dtype=np.float32), K)
    assert rg.launch_count() - before == launches
    v.close()


@pytest.mark.parametrize("view,W,H", [("room", 160, 120), ("inside", 83, 61), ("nan", 83, 61)])
def test_listed_update_matches_oracle(view, W, H):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    rng = np.random.default_rng(W)
    dim = 600.0 if view == "inside" else 1750.0
    origin, size = (0.0, 150.0, -300.0 if view == "inside" else -2350.0), (dim, dim, dim)
    o = O.OracleTSDF(O.tsdf_params(LISTED, W, H, origin=origin, dim=size))
    v = rg.TSDF(rg.tsdf_params(LISTED, W, H, cube_origin=origin, cube_dim=size))
    dist = distances(W, H, dim, rng, view)
    T = np.eye(4, dtype=np.float32)
    T[:3, 3] = (20.0, -35.0, 10.0)
    for _ in range(2):
        v.set_dist_map(dist)
        v.update(T, K)
        o.update(dist, T, K)
        assert np.array_equal(v.get("tsdf").view(np.uint32), o.grid.view(np.uint32))
    assert (o.grid.reshape(-1, 2)[:, 1] > 0).mean() > 0.01  # voxels were fused
    v.close()
