"""The kernels' fixed-point sums (recon_gb300/csrc/fx.cuh) against 128-bit integers
on the GPU: single values of every exponent, sums with cancellation, values out of
range, and the rounding to FP64 at ties and where it carries into the exponent."""
import pytest

import recon_gb300 as rg


@pytest.mark.gpu
def test_fixed_point_sums_are_exact():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    assert rg.selftest_fixed_point() == 0
