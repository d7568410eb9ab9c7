"""The linearisation kernel at the sizes where its parts begin and end, against
the oracle bit for bit and iteration by iteration: fewer and more photometric
chunks than the cluster has CTAs, histograms of both sizes, levels that are
smaller than one block of 1024 pixels, end inside a block, or have odd widths
(level 0 reads depths, the others points), and steps large enough for pixels to
leave the image."""
import pytest

import recon_gb300 as rg
from scenes import frame_pair
from test_gpu_parity import assert_bitexact, compare_traces, run_pair

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

CASES = [
    # W, H, levels, points, histogram bins, mode, rotation (deg), translation (mm)
    (64, 48, 2, 1024, 64, rg.BIOBJECTIVE, 1.0, 10.0),
    (90, 70, 2, 3072, 256, rg.BIOBJECTIVE, 1.5, 15.0),
    (322, 246, 2, 8192, 64, rg.GEOMETRIC, 2.0, 20.0),
    (320, 240, 3, 9216, 256, rg.PHOTOMETRIC, 2.0, 20.0),
    (320, 240, 3, 16384, 64, rg.BIOBJECTIVE, 8.0, 150.0),
    (640, 480, 4, 1024, 256, rg.BIOBJECTIVE, 3.0, 40.0),
]


@pytest.mark.parametrize("W,H,L,P,bins,mode,deg,mm", CASES)
def test_linearisation_matches_oracle(W, H, L, P, bins, mode, deg, mm):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    pair = frame_pair(W, H, L, seed=W + P, deg=deg, mm=mm, distortion=W == 320)
    trk, _, T, _, To, trace = run_pair(pair, mode, iters=(2, 3, 3, 2), n_select=P, hist_bins=bins)
    compare_traces(trk.trace(0), trace)
    assert_bitexact(T, To, "final pose")


def test_blocks_per_cta_of_a_full_device():
    """So many instances that a CTA of the correspondence kernel takes several
    blocks, with numbers of blocks that it does not divide."""
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    pairs = [frame_pair(640, 480, 2, seed=91, deg=2.0, mm=20.0), frame_pair(322, 246, 2, seed=92, deg=2.0, mm=20.0),
             frame_pair(90, 70, 2, seed=93, deg=1.5, mm=15.0)]
    order = [0] + [1, 2] * 6
    iters = (2, 2)
    cfgs = [rg.make_config(pairs[k].W, pairs[k].H, 2, mode=rg.GEOMETRIC, iters=iters, n_select=1024) for k in order]
    b = rg.Batch(cfgs, [pairs[k].cal.calib for k in order])
    b.set_reference([pairs[k].g0 for k in order], [pairs[k].d0 for k in order])
    b.set_current([pairs[k].g1 for k in order], [pairs[k].d1 for k in order])
    T, _ = b.track()
    for k, p in enumerate(pairs):
        _, _, _, _, To, _ = run_pair(p, rg.GEOMETRIC, iters=iters, n_select=1024)
        for i, o in enumerate(order):
            if o == k:
                assert_bitexact(T[i], To, f"instance {i}")


@pytest.mark.parametrize("W,H,L", [(75, 53, 1), (90, 70, 2), (128, 96, 2)])
def test_frame_preparation_at_odd_sizes_and_alignments(W, H, L):
    """Odd widths take pixels one by one, even ones in pairs unless the caller's
    images lie at odd addresses."""
    import numpy as np
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    pair = frame_pair(W, H, L, seed=W, deg=1.0, mm=8.0)
    iters = (2, 3)[:L]
    trk, _, T, _, To, trace = run_pair(pair, rg.BIOBJECTIVE, iters=iters, n_select=1024)
    compare_traces(trk.trace(0), trace)
    assert_bitexact(T, To, "final pose")
    g, d = (torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (pair.g1, pair.d1.view(np.int16)))
    for shift in (1, 2, 3):
        gs, ds = torch.zeros(g.numel() + shift, dtype=g.dtype, device="cuda"), torch.zeros(d.numel() + shift, dtype=d.dtype, device="cuda")
        gs[shift:] = g.reshape(-1)
        ds[shift:] = d.reshape(-1)
        trk.set_current(gs[shift:].view(H, W), ds[shift:].view(H, W))
        Ts, _ = trk.track(np.eye(4, dtype=np.float32))
        assert_bitexact(Ts, To, f"pose from images {shift} elements further")
