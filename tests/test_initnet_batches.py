"""The start network at the batch sizes where its launches change: one sample,
the first sizes at which a CTA of a layer takes several tiles of output pixels,
sizes that end inside a tile, numbers of splits on both sides of the three ways
to add them, and an input at an address that is a multiple of 4 bytes only.
Against the oracle, with the tolerances of test_initnet_gpu (the order of
accumulation differs)."""
import numpy as np
import pytest

import oracle_lib as O
from oracle_lib import ptr as p
from test_initnet_gpu import FWD_RTOL, GRAD_RTOL, _blocks, _need_gpu, _problem

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

import recon_gb300.initnet as IN  # noqa: E402


@pytest.mark.parametrize("n", [1, 33, 122, 245, 815])
def test_forward_at_launch_boundaries(n):
    _need_gpu()
    params, inp, inp_np, _ = _problem(20 + n, n)
    net = IN.InitNet(max_batch=n)
    net.set_params(params)
    y = net.forward(inp).cpu().numpy().astype(np.float64)
    want = np.zeros((n, 6))
    O.lib().orc_net_forward(p(params), p(inp_np), n, 0, p(want))
    assert np.linalg.norm(y - want) <= FWD_RTOL * np.linalg.norm(want)


@pytest.mark.parametrize("n,shift", [(1, 0), (7, 2), (130, 6), (245, 0)])
def test_gradient_at_launch_boundaries(n, shift):
    _need_gpu()
    params, inp, inp_np, target = _problem(40 + n, n)
    net = IN.InitNet(max_batch=n)
    net.set_params(params)
    room = torch.zeros(inp.numel() + shift, dtype=inp.dtype, device="cuda")
    room[shift:] = inp.reshape(-1)
    g, loss = net.gradient(room[shift:].view(inp.shape), torch.from_numpy(target).cuda())
    g = g.cpu().numpy().astype(np.float64)
    want = np.zeros(params.size)
    lw = O.lib().orc_net_loss_grad(p(params), p(inp_np), p(target), n, 0, p(want))
    assert abs(float(loss.item()) - lw) <= 1e-3 * lw
    for name, a, b in _blocks():
        err = np.linalg.norm(g[a:b] - want[a:b])
        ref = np.linalg.norm(want[a:b])
        assert err <= GRAD_RTOL * ref + 1e-9, (name, err, ref)
