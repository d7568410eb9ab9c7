"""The solve and the pose update on one warp (csrc/solve.cuh) against the oracle,
bit for bit: twists on both sides of the small-twist rule (2^-100 <= |x_k| <
2^-4), zero entries, large angles, and conjugate-gradient systems that use one
step, all steps, or stop early.  The Cholesky solve runs in every tracking
parity test.  A system with the identity matrix has x = b after one step."""
import ctypes

import numpy as np
import pytest

import oracle_lib as O
import recon_gb300 as rg
from recon_gb300 import synth

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
EDGE = 2.0 ** -4


def spd(seed, scale):
    M = np.random.default_rng(seed).normal(size=(6, 6))
    return (M @ M.T + 0.3 * np.eye(6)) * scale


TWISTS = {
    "small": [0.011, -0.007, 0.003, 0.004, -0.012, 0.02],
    "just_below": [np.nextafter(np.float32(EDGE), np.float32(0))] * 6,
    "at_edge": [0.01, -EDGE, 0.02, 0.01, 0.003, -0.004],
    "least": [2.0 ** -100, 0.01, -0.02, 0.03, -2.0 ** -100, 0.01],
    "below_least": [2.0 ** -101, 0.01, -0.02, 0.03, 0.02, 0.01],
    "zero_entry": [0.01, 0.0, -0.02, 0.0, 0.001, 0.0],
    "large": [0.9, -1.4, 2.1, 0.5, -3.0, 40.0],
    "nothing": [0.0] * 6,
}
CASES = [(k, np.eye(6), v) for k, v in TWISTS.items()]
CASES += [(f"spd_{s}", spd(s, 10.0 ** (s - 2)), np.random.default_rng(50 + s).normal(size=6) * 0.02 * 10.0 ** (s - 2))
          for s in range(5)]


@pytest.mark.parametrize("name,A,b", CASES, ids=[c[0] for c in CASES])
def test_solve_and_update_match_oracle(name, A, b):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    L = rg.lib()
    A, b = np.ascontiguousarray(A, np.float32), np.ascontiguousarray(b, np.float32)
    for T in (np.eye(4), synth.offset_pose(3, 7.0, 40.0), 1.02 * synth.offset_pose(4, 30.0, 900.0)):
        T = np.ascontiguousarray(T, np.float32)
        d = [torch.from_numpy(v.copy()).cuda() for v in (A, b, T)]
        L.solveMotionCuda(*[ctypes.c_void_p(v.data_ptr()) for v in d], ctypes.c_float(1000.0), None)
        torch.cuda.synchronize()
        x, To = np.zeros(6), T.copy()
        O.lib().orc_solve_cg(O.ptr(A.astype(np.float64)), O.ptr(b.astype(np.float64)), 1e-8, 6, O.ptr(x))
        O.lib().orc_expm_update(O.ptr(x), O.ptr(To), 1000.0)
        got = d[2].cpu().numpy()
        assert np.array_equal(got.view(np.uint32), To.view(np.uint32)), (name, got, To)
