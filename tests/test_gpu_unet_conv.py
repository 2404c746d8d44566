"""The network's convolutions at the edges of their 8 x 16 voxel tiles: one
8 x 8 x 8 volume (a single voxel at the lowest level), rows and columns that end
inside a tile, and z-planes that end inside a block's slab."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
from aphid_git_b200 import unet
from oracle import unet_ref as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(3, 2, 1), (9, 33, 8), (70, 17, 9), (20, 64, 41)])
def test_convolutions_at_tile_edges(dims):
    """Tolerances: the outputs' is the BF16 rounding of a stored activation
    (2^-8) through 15 layers that mostly average it, 1e-2; the gradient may
    differ from the restatement's by twice the latter's own BF16 noise (its
    distance from FP64), since both carry noise of that size."""
    X, Y, Z = dims
    rng = np.random.default_rng(X)
    Xp, Yp, Zp = pd = R.padded(dims)
    p = (R.init_params(X) * 0.7).astype(np.float32)
    x, t = (rng.standard_normal((X * Y * Z, c)).astype(np.float32) for c in (3, 8))

    def pad(a):
        out = np.zeros((Zp, Yp, Xp, a.shape[1]))
        out[:Z, :Y, :X] = a.reshape(Z, Y, X, -1)
        return out.reshape(Zp * Yp * Xp, -1)

    wp = pad(np.ones((X * Y * Z, 1)))[:, 0]
    g, y = {}, {}
    for bf in (True, False):
        y[bf], st = R.forward(p.astype(np.float64), pad(x), pd, bf=bf)
        g[bf] = R.backward(R.loss_grad(y[bf], pad(t), wp)[1], st, bf=bf)
    y_ref = y[True].reshape(Zp, Yp, Xp, 8)[:Z, :Y, :X].reshape(-1, 8)
    with unet.UNet(*dims, train=True) as net:
        net.set_params(p)
        xd, yd = torch.from_numpy(x).cuda(), torch.empty(X * Y * Z, 8, device="cuda")
        net.forward(xd, yd)
        net.train_step(xd, torch.from_numpy(t).cuda(), update=False)
        gd = net.grads()
    assert np.linalg.norm(yd.cpu().numpy() - y_ref) <= 1e-2 * np.linalg.norm(y_ref)
    noise = np.linalg.norm(g[True] - g[False])
    assert np.linalg.norm(gd - g[True]) <= 2 * noise + 1e-3 * np.linalg.norm(g[True])
