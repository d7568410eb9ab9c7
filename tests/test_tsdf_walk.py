"""The ray cast's crossing of empty blocks against the CPU oracle's voxel by
voxel walk, bit for bit: rays through several empty bricks and super bricks,
boundaries of two or three axes at the same time, rays along a grid axis, a
camera in and outside the grid, grids that are no multiple of a super brick, and
voxel sizes whose corner coordinates are exact sums and are not."""
import numpy as np
import pytest

import oracle_lib as O

pytestmark = pytest.mark.gpu

K = np.array([0.9, 0, 0.5, 0, -1.2, 0.5, 0, 0, 1], np.float32)


def _pose(rng, kind, dim):
    T = np.eye(4)
    if kind == "diagonal":  # equal direction components: plane crossings at equal times
        z = -np.array([1.0, 1.0, 1.0]) / np.sqrt(3.0)
        x = np.array([1.0, -1.0, 0.0]) / np.sqrt(2.0)
        T[:3, :3] = np.stack([x, np.cross(-z, x), -z], 1)
    elif kind == "random":
        q, _ = np.linalg.qr(rng.normal(size=(3, 3)))
        T[:3, :3] = q * np.sign(np.linalg.det(q))
        T[:3, 3] = rng.uniform(-0.6, 0.6, 3) * dim
    elif kind == "outside":
        T[:3, 3] = (0.11 * dim, -0.07 * dim, 2.3 * dim)
    return T.astype(np.float32)


@pytest.mark.parametrize("R,dim", [(8, 64.0), (40, 500.0), (64, 1750.0), (104, 1234.567), (128, 1500.0)])
@pytest.mark.parametrize("fill", [0.0, 2e-5, 2e-2])
def test_ray_cast_matches_voxel_walk(R, dim, fill):
    import recon_gb300 as rg
    rng = np.random.default_rng(R * 7 + int(fill * 1e6))
    W, H = 72, 52
    origin, size = (3.0, -7.5, 11.25), (dim, dim, dim)
    o = O.OracleTSDF(O.tsdf_params(R, W, H, origin=origin, dim=size))
    v = rg.TSDF(rg.tsdf_params(R, W, H, cube_origin=origin, cube_dim=size))
    grid = np.stack([rng.uniform(0.05, 1.0, R ** 3), np.ones(R ** 3)], 1).astype(np.float32)
    # negative values alone, and 5 x 5 x 5 together, so that the fine search hits as well
    g = grid.reshape(R, R, R, 2)
    for z, y, x in rng.integers(0, R, (int(fill * R ** 3) + (fill > 0), 3)):
        n = int(rng.choice([1, 5]))
        g[z:z + n, y:y + n, x:x + n, 0] = -rng.uniform(0.2, 1.0)
    o.grid[:] = grid.reshape(-1)
    v.set_grid(grid)
    hits = 0
    for kind in ("axis", "diagonal", "random", "random", "outside"):
        T = _pose(rng, kind, dim)
        for cubic in (False, True):
            v.raycast(T, K, cubic_filter=cubic)
            xyz = o.raycast(T, K, filtering=cubic)
            assert np.array_equal(v.get("xyz").view(np.uint32), xyz.view(np.uint32)), (kind, cubic)
            hits += int((xyz.reshape(-1, 4)[:, :3] != 0).any(1).sum())
    # a single negative voxel need not be met by a ray; none is met in an empty grid
    assert hits == 0 if fill == 0.0 else (hits > 0 or fill < 1e-3)
    v.close()


@pytest.mark.parametrize("R,W,H", [(232, 160, 120), (256, 83, 61)])
@pytest.mark.parametrize("view", ["room", "inside", "nan"])
def test_update_of_picked_blocks_matches_oracle(R, W, H, view):
    """A grid large enough for the update to list its blocks: blocks behind the
    surface, a camera in the grid, missing, infinite and NaN distances, image
    edges inside a tile."""
    import recon_gb300 as rg
    rng = np.random.default_rng(R + W)
    dim = 1750.0 if view != "inside" else 600.0
    origin, size = (0.0, 150.0, -2350.0 if view != "inside" else -300.0), (dim, dim, dim)
    o = O.OracleTSDF(O.tsdf_params(R, W, H, origin=origin, dim=size))
    v = rg.TSDF(rg.tsdf_params(R, W, H, cube_origin=origin, cube_dim=size))
    y, x = np.mgrid[0:H, 0:W]
    dist = (dim * (1.1 + 0.08 * np.sin(x / 40.0) * np.cos(y / 30.0) + 0.25 * (x > W // 2))).astype(np.float32)
    dist[rng.random((H, W)) < 0.02] = 0.0
    if view == "nan":
        dist[H // 3: H // 3 + 9, W // 4: W // 4 + 9] = np.nan
        dist[H // 2, W // 2] = np.inf
    T = np.eye(4, dtype=np.float32)
    T[:3, 3] = (20.0, -35.0, 10.0)
    Kn = np.array([0.9, 0, 0.5, 0, -1.2, 0.5, 0, 0, 1], np.float32)
    for _ in range(2):
        v.set_dist_map(dist)
        v.update(T, Kn)
        o.update(dist, T, Kn)
        assert np.array_equal(v.get("tsdf").view(np.uint32), o.grid.view(np.uint32))
    changed = (o.grid.reshape(-1, 2)[:, 1] > 0).mean()
    assert changed > 0.01  # voxels were fused
    v.close()
