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
