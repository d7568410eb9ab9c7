"""The work that is timed when this framework is made faster, through its public
entry points: tracking of single frame pairs, of keyframe segments and of bulk
frame pairs, the reconstruction stream, the learned start pose's network, and
the Kinect pre-processing.

Sizes come from bench.py's workloads, the tests and the synthetic generator:
images of 80x60 to 640x480 (odd-sized pyramids among them), 1 to 256 tracker
instances, grids of 64^3 to 512^3 voxels, network batches of 8 to 256 samples.
Inputs are seeded procedural scenes rendered on the GPU.
"""
import os

import numpy as np
import torch

import recon_gb300 as rg
from recon_gb300 import initnet, synth

MODES = {"photo": rg.PHOTOMETRIC, "geometric": rg.GEOMETRIC, "biobj": rg.BIOBJECTIVE}
# bi-objective weight, keyframe-fusion gate (mm) and depth noise of bench.py
LAMBDA, GATE_MM, NOISE = 0.5, 30.0, 0.01
SEGMENT, FUSED = 10, 5  # frames tracked against a keyframe, and how many of them are fused into it
BULK_SIZES = [(80, 60), (160, 120), (320, 240), (640, 480)]
CUBE = ((0.0, 150.0, -2350.0), (1750.0, 1750.0, 1750.0))  # grid around the synthetic room
TSDF_NOISE = 0.001
WEIGHTS = os.path.join(os.path.dirname(os.path.abspath(rg.__file__)), "weights", "initnet_200k.npz")


def _pair(name, **kw):
    c = {"name": name, "kind": "pair", "W": 640, "H": 480, "levels": 4, "mode": "biobj", "iters": "1,3,10,5",
         "hist_bins": 64, "solver": "cholesky", "precision": "fp32", "settle": False, "host": True,
         "new_keyframe": False}
    c.update(kw)
    return c


def _segments(name, **kw):
    c = {"name": name, "kind": "segments", "W": 640, "H": 480, "levels": 4, "n": 30, "iters": "1,3,10,5",
         "learned": False, "settle": False, "host": False}
    c.update(kw)
    return c


def listed():
    return [
        # a small camera image tracked live by its intensities: the smallest call
        _pair("photo_160x120", W=160, H=120, levels=3, mode="photo", iters="3,4,4,0"),
        # one frame pair registered photometrically with fixed 10/10/10 iterations
        _pair("photo_320x240", W=320, H=240, levels=3, mode="photo", iters="10,10,10,0", hist_bins=256, host=False),
        # a live RGB-D camera: each frame arrives in host memory and is tracked against the keyframe
        _pair("live_640x480"),
        # a keyframe change on an odd-sized camera: new reference, then its first frame, by geometry alone
        _pair("keyframe_482x362", W=482, H=362, levels=2, mode="geometric", iters="4,4,0,0", solver="cg",
              host=False, new_keyframe=True),
        # a recorded 300-frame trajectory in 30 keyframe segments, keyframes fused on the way
        _segments("segments_640x480_30"),
        # the same streamed from pinned host memory with the learned start pose and its short schedule
        _segments("learned_640x480_30", iters="1,2,2,1", learned=True, host=True),
        # bulk registration of unrelated frame pairs of mixed resolution
        {"name": "bulk_256", "kind": "bulk", "n": 256},
        # the reconstruction stream on a coarse preview grid, on the usual grid, and on the finest
        {"name": "tsdf_64", "kind": "tsdf", "R": 64, "W": 320, "H": 240, "frames": 2},
        {"name": "tsdf_256", "kind": "tsdf", "R": 256, "W": 640, "H": 480, "frames": 6},
        {"name": "tsdf_512", "kind": "tsdf", "R": 512, "W": 640, "H": 480, "frames": 2},
        # a training batch of the start-pose network: forward and backward
        {"name": "net_gradient_256", "kind": "net", "n": 256, "gradient": True},
        # one captured Kinect frame made ready for the tracker
        {"name": "kinect_640x480", "kind": "kinect", "W": 640, "H": 480, "hdr": False},
    ]


def _size(rng, levels):
    """A camera size of 80x60 to 640x480 whose pyramid has `levels` levels."""
    m = 1 << (levels - 1)
    w = 80.0 * 8.0 ** rng.random()
    h = w * rng.uniform(0.6, 0.8)
    W, H = min(640, int(w)) // m * m, min(480, int(h)) // m * m
    return max(W, 80 // m * m), max(H, 56 // m * m)


def _net_size(rng):
    k = rng.randint(2, 8)  # the network takes multiples of 80x60
    return 80 * k, 60 * k


def _iters(rng, levels):
    v = [rng.randint(1, 10) for _ in range(levels)]
    return ",".join(str(x) for x in v + [0] * (4 - levels))


def draw(rng):
    kind = rng.choice(["pair", "pair", "pair", "segments", "segments", "bulk", "tsdf", "tsdf", "net", "kinect"])
    if kind == "pair":
        levels = rng.randint(2, 4)
        W, H = _size(rng, levels)
        settle = rng.random() < 0.2
        c = _pair("", W=W, H=H, levels=levels, mode=rng.choice(["photo", "geometric", "biobj", "biobj"]),
                  iters=_iters(rng, levels), hist_bins=rng.choice([64, 256]),
                  solver=rng.choice(["cholesky", "cholesky", "cg"]), precision=rng.choice(["fp32", "mixed"]),
                  settle=settle, host=rng.random() < 0.5, new_keyframe=rng.random() < 0.3)
    elif kind == "segments":
        learned = rng.random() < 0.5
        n = max(1, min(30, int(round(30.0 ** rng.random()))))
        W, H = _net_size(rng) if learned else _size(rng, 3)
        c = _segments("", W=W, H=H, levels=4 if W % 8 == 0 and H % 8 == 0 and W >= 320 else 3, n=n, learned=learned,
                      settle=rng.random() < 0.25, host=rng.random() < 0.5)
        short = [1, 2, 2, 1] if learned else [rng.randint(1, 3), rng.randint(1, 3), rng.randint(1, 8), rng.randint(1, 5)]
        if W % 4 or H % 4:
            c["levels"] = 2
        short = short[:c["levels"]] + [0] * (4 - c["levels"])
        c["iters"] = ",".join(str(x) for x in short)
    elif kind == "bulk":
        c = {"kind": "bulk", "n": int(round(4 * 64.0 ** rng.random()))}
    elif kind == "tsdf":
        W = rng.randint(160, 640)
        c = {"kind": "tsdf", "R": 8 * int(round(8 * 8.0 ** rng.random())), "W": W, "H": int(W * rng.uniform(0.6, 0.75)),
             "frames": rng.randint(1, 2)}
    elif kind == "net":
        c = {"kind": "net", "n": int(round(8 * 32.0 ** rng.random())), "gradient": rng.random() < 0.6}
    else:
        W, H = _size(rng, 2)
        c = {"kind": "kinect", "W": W, "H": H, "hdr": rng.random() < 0.5}
    c.pop("name", None)
    return c


# ---------------------------------------------------------------- inputs

def _render(cal, scene, poses, seed, noise=NOISE, gray=True):
    """Gray (uint8) and depth (mm, 16 bits) of every pose, on the GPU."""
    n = len(poses)
    g = torch.empty((n, cal.height, cal.width), dtype=torch.uint8, device="cuda") if gray else None
    d = torch.empty((n, cal.height, cal.width), dtype=torch.int16, device="cuda")
    for f in range(n):
        rg.render_depth(scene, synth.camera_struct(cal, "L", poses[f]), noise, seed + 1, f, d[f])
        if gray:
            rg.render_gray(scene, synth.camera_struct(cal, "R", poses[f]), g[f])
    torch.cuda.synchronize()
    return g, d


def _points(W, H):
    return int(min(8192, (W * H // 2 // 1024) * 1024))


def _config(case, W, H, levels, iters, mode, **kw):
    return rg.make_config(W, H, levels, mode=mode, iters=iters, n_select=_points(W, H), lam=LAMBDA, **kw)


def _schedule(case):
    return tuple(int(v) for v in case["iters"].split(","))


def _settle(case):
    return (0.1, 1e-4) if case["settle"] else (0.0, 0.0)


def _prepare_pair(case, seed):
    W, H = case["W"], case["H"]
    rng = np.random.default_rng(seed)
    cal = synth.make_calibration(W, H, distortion=True)
    scene = synth.make_scene(int(rng.integers(1 << 30)))
    moved = synth.offset_pose(int(rng.integers(1 << 30)), float(rng.uniform(0.3, 1.5)), float(rng.uniform(3.0, 20.0)))
    g, d = _render(cal, scene, [np.eye(4), moved], int(rng.integers(1 << 30)))
    if case["host"]:
        g, d = g.cpu().numpy(), d.cpu().numpy().view(np.uint16)
    cfg = _config(case, W, H, case["levels"], _schedule(case), MODES[case["mode"]], hist_bins=case["hist_bins"],
                  solver=rg.SOLVER_CG if case["solver"] == "cg" else rg.SOLVER_CHOLESKY,
                  precision=rg.PRECISION_MIXED if case["precision"] == "mixed" else rg.PRECISION_FP32,
                  settle=_settle(case))
    trk = rg.Tracker(cfg, cal.calib)
    trk.set_reference(g[0], d[0])
    return {"kind": "pair", "tracker": trk, "gray": g, "depth": d, "new_keyframe": case["new_keyframe"]}


def _prepare_segments(case, seed):
    W, H, n = case["W"], case["H"], case["n"]
    rng = np.random.default_rng(seed)
    cal = synth.make_calibration(W, H)
    scene = synth.make_scene(int(rng.integers(1 << 30)))
    poses = synth.smooth_trajectory(SEGMENT * n + 1, int(rng.integers(1 << 30)))
    g, d = _render(cal, scene, poses, int(rng.integers(1 << 30)))
    if case["host"]:
        g, d = g.cpu().pin_memory(), d.cpu().pin_memory()
    cfg = _config(case, W, H, case["levels"], _schedule(case), rg.BIOBJECTIVE, settle=_settle(case))
    batch = rg.Batch([cfg] * n, [cal.calib] * n)
    net = None
    if case["learned"]:
        net = initnet.InitNet(max_batch=n)
        net.set_params(np.load(WEIGHTS)["params"])
        batch.set_init_net(net, _schedule(case))
    ref = SEGMENT * np.arange(n)
    return {"kind": "segments", "batch": batch, "net": net, "gray": g, "depth": d, "ref": ref,
            "frames": ref[None, :] + np.arange(1, SEGMENT + 1)[:, None]}


def _prepare_bulk(case, seed):
    rng = np.random.default_rng(seed)
    cals = {s: synth.make_calibration(*s) for s in BULK_SIZES}
    # the resolutions in equal shares, in an order of their own for each seed
    sizes = [BULK_SIZES[i % len(BULK_SIZES)] for i in rng.permutation(case["n"])]
    configs, calibs, g, d = [], [], [], []
    for W, H in sizes:
        levels = 4 if W == 640 else 3
        iters = tuple(int(v) for v in rng.integers(4, 13, size=levels))
        scene = synth.make_scene(int(rng.integers(1 << 30)))
        moved = synth.offset_pose(int(rng.integers(1 << 30)), float(rng.uniform(0.5, 4.0)),
                                  float(rng.uniform(0.5, 50.0)))
        a, b = _render(cals[(W, H)], scene, [np.eye(4), moved], int(rng.integers(1 << 30)))
        configs.append(_config(case, W, H, levels, iters, rg.BIOBJECTIVE))
        calibs.append(cals[(W, H)].calib)
        g.append(a)
        d.append(b)
    batch = rg.Batch(configs, calibs)
    start = np.tile(np.eye(4, dtype=np.float32), (case["n"], 1, 1))
    return {"kind": "bulk", "batch": batch, "start": start, "frames": [[[x[f] for x in v] for v in (g, d)] for f in (0, 1)]}


def _tsdf_inputs(case, seed):
    W, H = case["W"], case["H"]
    rng = np.random.default_rng(seed)
    cal = synth.make_calibration(W, H)
    scene = synth.make_scene(int(rng.integers(1 << 30)))
    poses = synth.smooth_trajectory(case["frames"], int(rng.integers(1 << 30))).astype(np.float32)
    _, depth = _render(cal, scene, poses, int(rng.integers(1 << 30)), TSDF_NOISE, gray=False)
    return cal, poses, depth, rg.normalized_K(cal.camera_K("L"), W, H)


def _prepare_tsdf(case, seed):
    cal, poses, depth, K = _tsdf_inputs(case, seed)
    grid = rg.TSDF(rg.tsdf_params(case["R"], case["W"], case["H"], cal.min_dist, cal.max_dist, cube_origin=CUBE[0],
                                  cube_dim=CUBE[1]))
    views = {k: torch.as_tensor(grid.view(k), device="cuda") for k in ("xyz", "normal", "shaded", "tsdf")}
    return {"kind": "tsdf", "grid": grid, "poses": poses, "depth": depth, "K": K, "views": views}


def _net_inputs(case, seed):
    """Coarse image pairs (gray in [0, 1], depth in metres / 4) and target outputs."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    n = case["n"]

    def smooth(channels):
        z = torch.randn((n, channels, 15, 20), generator=gen, device="cuda")
        return torch.nn.functional.interpolate(z, size=(60, 80), mode="bilinear", align_corners=False)

    base, change = smooth(2), 0.1 * smooth(2)
    gray = lambda v: torch.sigmoid(v)  # noqa: E731
    depth = lambda v: 0.5 + 0.2 * torch.tanh(v)  # noqa: E731
    x = torch.stack([gray(base[:, 0]), depth(base[:, 1]), gray((base + change)[:, 0]), depth((base + change)[:, 1])], -1)
    return x.to(torch.bfloat16).contiguous(), torch.randn((n, 6), generator=gen, device="cuda")


def _prepare_net(case, seed):
    x, target = _net_inputs(case, seed)
    net = initnet.InitNet(max_batch=case["n"])
    net.set_params(np.load(WEIGHTS)["params"])
    return {"kind": "net", "net": net, "x": x, "target": target, "gradient": case["gradient"]}


def _prepare_kinect(case, seed):
    W, H = case["W"], case["H"]
    rng = np.random.default_rng(seed)
    cal = synth.make_calibration(W, H, distortion=True)
    c0, c1 = float(cal.calib[61]), float(cal.calib[42])
    scene = synth.make_scene(int(rng.integers(1 << 30)))
    g, d = _render(cal, scene, [np.eye(4)], int(rng.integers(1 << 30)))
    # 11-bit disparity of the depth image (2047: none) and a coloured image of its gray values
    z = d[0].to(torch.float64)
    disp = torch.where(z > 0, ((1.0 / z.clamp(min=1.0) - c0) / c1).round().clamp(0, 2046), torch.full_like(z, 2047.0))
    tint = torch.from_numpy(rng.uniform(0.7, 1.0, size=(H, W, 3))).cuda()
    rgb = (g[0].double()[..., None] * tint).to(torch.uint8).contiguous()
    # the camera matrix of the gray image and its inverse, in pixels
    return {"kind": "kinect", "disp": disp.to(torch.int16).contiguous(), "rgb": rgb, "c": (c0, c1),
            "range": (cal.min_dist, cal.max_dist), "K": cal.calib[0:9].copy(), "iK": cal.calib[9:18].copy(),
            "kc": cal.calib[18:23].copy(), "hdr": case["hdr"]}


def prepare(case, seed):
    return {"pair": _prepare_pair, "segments": _prepare_segments, "bulk": _prepare_bulk, "tsdf": _prepare_tsdf,
            "net": _prepare_net, "kinect": _prepare_kinect}[case["kind"]](case, seed)


# ---------------------------------------------------------------- one pass

def _run_pair(s):
    trk, g, d = s["tracker"], s["gray"], s["depth"]
    if s["new_keyframe"]:
        trk.set_reference(g[0], d[0])
    trk.set_current(g[1], d[1])
    T, st = trk.track()
    return {"pose": T, "iterations": st.iterations, "solves": st.solves, "points": list(st.icp_selected)}


def _run_segments(s):
    b, g, d, f = s["batch"], s["gray"], s["depth"], s["frames"]
    b.set_reference_frames(g, d, s["ref"])
    first, _ = b.track_sequence_frames(g, d, f[:FUSED])
    b.fuse_sequence(FUSED, GATE_MM)
    rest, st = b.track_sequence_frames(g, d, f[FUSED:])
    return {"poses": np.concatenate([first, rest]), "points": np.array([list(x.icp_selected) for x in st])}


def _run_bulk(s):
    b = s["batch"]
    b.set_reference(*s["frames"][0])
    b.set_current(*s["frames"][1])
    T, st = b.track(s["start"])
    return {"poses": T, "points": np.array([list(x.icp_selected) for x in st])}


def _run_tsdf(s):
    grid, K = s["grid"], s["K"]
    grid.reset()
    for T, depth in zip(s["poses"], s["depth"]):
        grid.set_dist_depth16(depth)
        grid.update(T, K)
        grid.raycast(T, K)
    return s["views"]


def _run_net(s):
    if not s["gradient"]:
        return {"out": s["net"].forward(s["x"])}
    g, loss = s["net"].gradient(s["x"], s["target"])
    return {"gradient": g, "loss": loss}


def _run_kinect(s):
    (c0, c1), (near, far) = s["c"], s["range"]
    if s["hdr"]:
        disp = rg.kinect_disparity_to_float(s["disp"])
        z = rg.kinect_depth_normalized(disp, c0, c1, near, far, -4.0, -3.0)
        rgb = rg.kinect_undistort_rgb_hdr(s["rgb"], s["K"], s["iK"], s["kc"])
        return {"disp": disp, "z": z, "rgb": rgb, "gray": rg.kinect_rgb_to_gray_hdr(rgb)}
    z = rg.kinect_disparity_to_depth(s["disp"], c0, c1, near, far, -4.0, -3.0)
    gray = rg.kinect_rgb_to_gray(s["rgb"])
    return {"z": z, "gray": gray, "undistorted": rg.kinect_undistort_gray(gray, s["K"], s["iK"], s["kc"])}


_RUN = {"pair": _run_pair, "segments": _run_segments, "bulk": _run_bulk, "tsdf": _run_tsdf, "net": _run_net,
        "kinect": _run_kinect}


def run(state):
    return _RUN[state["kind"]](state)


# ---------------------------------------------------------------- what a pass cannot do without

# FP32 operations of one point in one Gauss-Newton iteration (projection, taps,
# residual, Jacobian, the 27 sums), and bytes of the prepared keyframe
ICP_FLOPS, PHOTO_FLOPS, ICP_BYTES = 230, 180, 24


def _track_work(W, H, levels, iters, mode, frames=1, keyframes=0, fused=0):
    """Frames read once; the prepared keyframe read once for each tracked frame."""
    px = [(W >> l) * (H >> l) for l in range(levels)]
    P = _points(W, H)
    run_levels = [l for l in range(levels) if iters[levels - 1 - l] > 0]
    photo, icp = mode != "geometric", mode != "photo"
    flops = sum(iters[levels - 1 - l] * (photo * PHOTO_FLOPS * P + icp * ICP_FLOPS * px[l]) for l in run_levels)
    state = sum(photo * 28 * P + icp * ICP_BYTES * px[l] for l in run_levels) + photo * 12 * P
    return {"bytes": frames * (3 * px[0] + state + 64) + keyframes * (3 * px[0] + state) + fused * 3 * px[0],
            "flops": frames * flops + (keyframes + fused) * 60 * px[0]}


def work(case):
    kind = case["kind"]
    if kind == "pair":
        return _track_work(case["W"], case["H"], case["levels"], _schedule(case), case["mode"],
                           keyframes=int(case["new_keyframe"]))
    if kind == "segments":
        w = _track_work(case["W"], case["H"], case["levels"], _schedule(case), "biobj", SEGMENT, 2, FUSED)
        return {k: case["n"] * v for k, v in w.items()}
    if kind == "bulk":
        total = {"bytes": 0, "flops": 0}
        for i in range(case["n"]):
            W, H = BULK_SIZES[i % len(BULK_SIZES)]
            levels = 4 if W == 640 else 3
            w = _track_work(W, H, levels, [8] * levels, "biobj", keyframes=1)
            total = {k: total[k] + w[k] for k in total}
        return total
    if kind == "tsdf":
        # the grid written once; per frame the depth read, about a third of the
        # voxels read and written, and the three float4 images written
        vox, px, n = case["R"] ** 3, case["W"] * case["H"], case["frames"]
        return {"bytes": 8 * vox + n * (2 * px + 16 * vox // 3 + 48 * px), "flops": n * (30 * vox + 300 * px)}
    if kind == "net":
        n = case["n"]
        macs = sum(h * w * co * 9 * ci for (ci, co), (h, w) in zip(initnet.LAYERS, _net_sizes()[1:]))
        passes = 3 if case["gradient"] else 1
        return {"bytes": n * 60 * 80 * 4 * 2 + 4 * initnet.param_count() * (2 if case["gradient"] else 1),
                "flops": 2 * macs * n * passes}
    px = case["W"] * case["H"]
    return {"bytes": (2 + 4 + 1 + 3 + 12 + 12 + 4) * px if case["hdr"] else (2 + 4 + 3 + 1 + 1 + 1) * px,
            "flops": 60 * px}


def _net_sizes():
    s = [(60, 80)]
    for _ in initnet.LAYERS:
        s.append(((s[-1][0] + 1) // 2, (s[-1][1] + 1) // 2))
    return s


# ---------------------------------------------------------------- 64 bits

def _exact_tsdf(case, seed):
    """The grid after all frames; the ray cast's images are decided by the
    signs of grid samples along each ray and have no value of their own."""
    cal, poses, depth, K = _tsdf_inputs(case, seed)
    R, W, H = case["R"], case["W"], case["H"]
    half = np.asarray(CUBE[1], np.float64)
    origin = np.asarray(CUBE[0], np.float64)
    step = 2 * half / R
    start = origin - half + step / 2
    lim, tol, slope = step[0], half[0] / 200.0, half[0] * 0.03
    K = np.asarray(K, np.float64)
    axis = [torch.from_numpy(start[k] + step[k] * np.arange(R)).cuda() for k in range(3)]
    value = torch.ones((R, R, R), dtype=torch.float64, device="cuda")
    weight = torch.zeros_like(value)
    for f in range(case["frames"]):
        T = synth.inv_se3(poses[f].astype(np.float64))
        img = depth[f].to(torch.float64)
        for z0 in range(0, R, 64):
            z, y, x = torch.meshgrid(axis[2][z0:z0 + 64], axis[1], axis[0], indexing="ij")
            p = [T[r, 0] * x + T[r, 1] * y + T[r, 2] * z + T[r, 3] for r in range(3)]
            u, v = (p[0] / p[2] * K[0] + K[2]) * W, (p[1] / p[2] * K[4] + K[5]) * H
            ok = (u >= 1) & (u < W - 2) & (v >= 1) & (v < H - 2)
            at = torch.nonzero(ok, as_tuple=True)
            u, v, dist = u[at], v[at], -p[2][at]
            ui, vi = u.long(), v.long()
            fu, fv = u - ui, v - vi
            taps = [img[vi + j, ui + i] for j in (0, 1) for i in (0, 1)]
            m = (1 - fu) * (1 - fv) * taps[0] + fu * (1 - fv) * taps[1] + (1 - fu) * fv * taps[2] + fu * fv * taps[3]
            keep = torch.ones_like(u, dtype=torch.bool)
            for t in taps:
                keep &= (t >= lim) & ((m - t).abs() <= tol)
            sdf = (m - dist) / slope
            keep &= sdf >= -1.25
            at = tuple(i[keep] for i in at)
            old, w = value[z0:z0 + 64][at], weight[z0:z0 + 64][at]
            value[z0:z0 + 64][at] = (w * old + sdf[keep].clamp(-1, 1)) / (w + 1)
            weight[z0:z0 + 64][at] = (w + 1).clamp(max=16)
    return {"xyz": None, "normal": None, "shaded": None, "tsdf": torch.stack([value, weight], -1)}


class _RoundGradient(torch.autograd.Function):
    """The identity; its gradient is rounded to 16 bits, as the tensor cores take it."""

    @staticmethod
    def forward(ctx, x):
        return x.view_as(x)

    @staticmethod
    def backward(ctx, g):
        return g.to(torch.bfloat16).to(torch.float64)


def _exact_net(case, seed):
    """The network as it is defined, with 16-bit weights, activations and
    convolution gradients; everything between them in 64 bits."""
    x, target = _net_inputs(case, seed)
    p = torch.from_numpy(np.load(WEIGHTS)["params"].astype(np.float64)).cuda().requires_grad_(True)
    off, wfc, bfc, _, _ = initnet.layout()

    def round16(v):  # the gradient passes through
        return v + (v.to(torch.bfloat16).to(torch.float64) - v).detach()

    a = x.to(torch.float64).permute(0, 3, 1, 2)
    for (cin, cout), (w, b) in zip(initnet.LAYERS, off):
        kp = (9 * cin + 15) // 16 * 16
        k = round16(p[w:w + cout * kp]).view(cout, kp)[:, :9 * cin].view(cout, 3, 3, cin).permute(0, 3, 1, 2)
        # the 3x3 / stride 2 / pad 1 patches as one matrix product
        h, v = (a.shape[2] + 1) // 2, (a.shape[3] + 1) // 2
        cols = torch.nn.functional.unfold(a, 3, padding=1, stride=2)
        z = _RoundGradient.apply(k.reshape(cout, -1) @ cols) + p[b:b + cout, None]
        a = round16(torch.relu(z)).view(case["n"], cout, h, v)
    y = a.mean((2, 3)) @ p[wfc:wfc + 6 * initnet.FEAT].view(6, -1).T + p[bfc:bfc + 6]
    if not case["gradient"]:
        return {"out": y.detach()}
    loss = ((y - target.to(torch.float64)) ** 2).mean()
    loss.backward()
    return {"gradient": p.grad, "loss": loss.detach().reshape(1)}


def _exact_kinect(case, seed):
    """The depth and colour maps; 8-bit images are whole numbers."""
    s = _prepare_kinect(case, seed)
    W, H = case["W"], case["H"]
    (c0, c1), (near, far) = [[float(np.float32(v)) for v in s[k]] for k in ("c", "range")]
    disp = s["disp"].cpu().numpy().astype(np.float64)

    def depth(d):
        z = np.abs(1.0 / (c0 + c1 * d))
        return np.where((z > far) | (z < near), 0.0, z)

    if not case["hdr"]:
        z = np.zeros((H, W))
        rows = 4 * (H // 4)
        block = disp[0:rows - 3, 0:W - 4]  # the IR image is shifted by (-4, -3)
        z[3:rows, 4:] = np.where(block < 2047, depth(block), 0.0)
        return {"z": z, "gray": None, "undistorted": None}
    full = np.where(disp < 2047, disp, 65535.0)
    xs, ys = np.maximum(2 * np.arange(W // 2) - 4, 0), np.maximum(2 * np.arange(H // 2) - 3, 0)
    taps = [full[np.ix_(ys + j, xs + i)] for j in (0, 1) for i in (0, 1)]
    least = np.minimum.reduce(taps)
    ok = np.all([t < 2047 for t in taps], axis=0)
    z = np.where(ok, (depth(least) - near) / (far - near), 0.0)
    K, iK = s["K"].astype(np.float64).reshape(3, 3), s["iK"].astype(np.float64).reshape(3, 3)
    kc = s["kc"].astype(np.float64)
    y, x = np.mgrid[0:H, 0:W].astype(np.float64)
    a, b = iK[0, 0] * x + iK[0, 1] * y + iK[0, 2], iK[1, 0] * x + iK[1, 1] * y + iK[1, 2]
    r2 = a * a + b * b
    r = 1 + kc[0] * r2 + kc[1] * r2 ** 2 + kc[4] * r2 ** 3
    a, b = a * r, b * r
    u, v = K[0, 0] * a + K[0, 1] * b + K[0, 2], K[1, 0] * a + K[1, 1] * b + K[1, 2]
    ui, vi = np.trunc(u).astype(int), np.trunc(v).astype(int)
    ok = (ui >= 0) & (vi >= 0) & (ui < W - 2) & (vi < H - 2)
    fu, fv = (u - ui)[..., None], (v - vi)[..., None]
    ui, vi = np.where(ok, ui, 0), np.where(ok, vi, 0)
    img = s["rgb"].cpu().numpy().astype(np.float64) / 255.0
    rgb = ((1 - fu) * (1 - fv) * img[vi, ui] + fu * (1 - fv) * img[vi, ui + 1] + (1 - fu) * fv * img[vi + 1, ui]
           + fu * fv * img[vi + 1, ui + 1]) * ok[..., None]
    return {"disp": full, "z": z, "rgb": rgb, "gray": rgb @ np.array([0.3, 0.59, 0.11])}


def exact(case, seed):
    """None for the tracked poses: they are the end of a chain of whole-number
    decisions (selected points, histogram medians, truncated sums)."""
    f = {"tsdf": _exact_tsdf, "net": _exact_net, "kinect": _exact_kinect}.get(case["kind"])
    return f(case, seed) if f else None
