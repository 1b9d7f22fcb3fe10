"""The warm-start network's 3 x 3 x 3 convolutions at grids whose tiles have remainders (levels of
1 to 40 voxels a side; each number of blocks per cluster) against torch float64 autograd."""
import numpy as np
import pytest
import torch

from mdft_b200 import warmstart
from oracle import warmnet_ref as W

pytestmark = pytest.mark.gpu


# grid n: levels n, n/2, n/4, n/8 around the 8 x 4 x 4 tile
@pytest.mark.parametrize("n", [8, 24, 40])
def test_forward_and_gradients(n):
    net = warmstart.WarmNet(n, seed=n)
    rng = np.random.default_rng(n)
    x = rng.standard_normal((3, n, n, n)).astype(np.float32)
    t = rng.standard_normal((4, n, n, n)).astype(np.float32)
    m = (rng.random((n, n, n)) > 0.25).astype(np.float32)
    dx, dt, dm = (torch.tensor(v, device="cuda") for v in (x, t, m))
    out = torch.empty((4, n, n, n), device="cuda")
    torch.cuda.synchronize()
    net.forward(dx.data_ptr(), out.data_ptr())
    g, loss = net.gradients(dx.data_ptr(), dt.data_ptr(), dm.data_ptr())
    torch.cuda.synchronize()
    p = torch.tensor(W.bf16_weights(net.get_params()).astype(np.float64), requires_grad=True)
    net.close()
    y = W.forward(p, torch.tensor(x, dtype=torch.float64), torch)
    L = W.loss(y, torch.tensor(t, dtype=torch.float64), torch.tensor(m, dtype=torch.float64))
    L.backward()
    ref = y.detach().numpy()
    assert np.abs(out.cpu().numpy() - ref).max() < 1e-5 * np.abs(ref).max()
    assert abs(loss - L.item()) <= 1e-5 * abs(L.item())
    # per layer the bound of the 16^3 comparison; a layer's gradient is a sum over voxels
    off, gr = 0, p.grad.numpy()
    for li, (k, _, _, ci, co, _, _) in enumerate(W.LAYERS):
        nw = int(np.prod(W.weight_shape(k, ci, co)))
        for a, b in ((off, off + nw), (off + nw, off + nw + co)):
            assert np.abs(g[a:b] - gr[a:b]).max() < 2e-4 * np.abs(gr[a:b]).max(), li
        off += nw + co
