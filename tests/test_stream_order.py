"""What the Python layer does around a launch: rows that a kernel does not
write are 0 in a new image, and the library's stream waits for torch's current
one, whichever that is."""
import numpy as np
import pytest

import recon_gb300 as rg

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("H", [48, 49, 50, 51, 53])
def test_rows_that_no_kernel_writes_are_zero(H):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    W = 40
    for _ in range(3):  # memory that held something else before
        junk = torch.full((H, W), 255, dtype=torch.uint8, device="cuda")
        del junk
        rgb = torch.full((H, W, 3), 200, dtype=torch.uint8, device="cuda")
        gray = rg.kinect_rgb_to_gray(rgb)
        white = (200 * (19588 + 38469 + 7471)) >> 16  # the conversion's 16-bit weights
        assert int(gray[H // 4 * 4:].sum()) == 0 and int((gray[:H // 4 * 4] != white).sum()) == 0
        K = np.array([30, 0, 20, 0, 30, 24, 0, 0, 1], np.float32)
        iK = np.linalg.inv(K.reshape(3, 3).astype(np.float64)).astype(np.float32)
        out = rg.kinect_undistort_gray(gray, K, iK, np.zeros(5, np.float32))
        assert int(out[H // 6 * 6:].sum()) == 0


@pytest.mark.parametrize("side", [False, True])
def test_inputs_still_being_written_are_waited_for(side):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    W, H = 640, 480
    grid = rg.TSDF(rg.tsdf_params(32, W, H))
    src = torch.randint(500, 4000, (H, W), dtype=torch.int16, device="cuda")
    stream = torch.cuda.Stream() if side else torch.cuda.current_stream()
    torch.cuda.synchronize()
    for k in range(4):
        with torch.cuda.stream(stream):
            big = torch.zeros(64 << 20, device="cuda")
            for _ in range(8):  # work in front of the input's own
                big += 1.0
            depth = src + k
            grid.set_dist_depth16(depth)
        assert np.array_equal(grid.get("dist").reshape(H, W), (src + k).cpu().numpy().astype(np.float32))
    grid.close()
