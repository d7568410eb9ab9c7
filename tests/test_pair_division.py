"""The division that the packed kernels use (recon_gb300/csrc/pair_math.cuh)
against IEEE division on the GPU: every mantissa of the reciprocal, and
pseudo-random quotients over the range of operands that it is used for.  What
lies outside the range goes through the compiler's division; the poses of the
parity tests cover both."""
import pytest

import recon_gb300 as rg


@pytest.mark.gpu
def test_division_is_correctly_rounded():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    assert rg.selftest_division() == 0
