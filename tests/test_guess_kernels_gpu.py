"""Feature extraction, pooling and composing of the warm-start guess at the edges
of their tiles, vectors and channel groups.

Features agree with the oracle bit for bit. The guess is guidance + bilinear(c)
for the network's prediction c on the pooled problem (pooled here in the same
order, so c is the same); interpolating takes a weight good to the coordinate's
rounding, a coordinate of at most n coarse cells two roundings, and five
operations on values of |g| + 4 |c| at most: with e = 2^-24,
|difference| <= e (4 n 2 max|c| + 8 (max|g| + 4 max|c|))."""
import numpy as np
import pytest

from oracle import unet_ref as R

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def torch():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    return torch


@pytest.fixture(scope="module")
def net(ctx, torch):
    from paintop_b200 import warmstart
    return warmstart.UNet(ctx, seed=5)


# tiles of 32 x 32: one, its edges, several and a remainder; runs longer than 32
@pytest.mark.parametrize("holes", [0.0, 0.02, 0.5])
@pytest.mark.parametrize("B,H,W", [(1, 8, 8), (2, 32, 32), (1, 24, 40), (3, 40, 104), (1, 128, 96), (1, 8, 264)])
def test_features_at_tile_edges(net, torch, B, H, W, holes):
    from paintop_b200 import _lib
    rng = np.random.default_rng(B + H + W)
    g, a = (rng.random((B, H, W), dtype=np.float32) for _ in range(2))
    m = (rng.random((B, H, W)) >= holes).astype(np.float32)
    want = R.features(g, a, m)
    d = [torch.as_tensor(x, device="cuda") for x in (g, a, m)]
    assert np.array_equal(net.features(*d).cpu().numpy().view(np.uint32), want.view(np.uint32))
    out = torch.empty(B * H * W * 4 + 1, device="cuda")  # features that are not 16-byte aligned
    torch.cuda.synchronize()
    net._check(_lib.lib().pt_unet_features(net.h, d[0].data_ptr(), d[1].data_ptr(), d[2].data_ptr(), B, H, W,
                                           out.data_ptr() + 4), "features")
    assert np.array_equal(out[1:].cpu().numpy().view(np.uint32), want.reshape(-1).view(np.uint32))


# channel groups of four, three and one; widths and scales that leave remainders;
# images that start off a 16-byte boundary
@pytest.mark.parametrize("H,W,C,s", [(9, 7, 1, 1), (33, 50, 2, 3), (64, 61, 3, 4), (41, 75, 4, 5), (30, 31, 5, 2), (95, 96, 7, 7), (40, 37, 8, 64)])
@pytest.mark.parametrize("skew", [0, 1])
def test_guess_at_remainders(net, torch, H, W, C, s, skew):
    from paintop_b200 import _lib
    rng = np.random.default_rng(H * W + C)
    g, a = (rng.random((H, W, C), dtype=np.float32) for _ in range(2))
    m = (rng.random((H, W)) > 0.2).astype(np.float32)
    hv, wv = -(-H // s), -(-W // s)
    Hc, Wc = -(-max(hv, 8) // 8) * 8, -(-max(wv, 8) // 8) * 8

    def pool(img):
        out = np.zeros((Hc, Wc), np.float32)
        for y in range(hv):
            for x in range(wv):
                block, acc = img[y * s:y * s + s, x * s:x * s + s], np.float32(0)
                for v in block.reshape(-1):
                    acc = np.float32(acc + v)
                out[y, x] = acc * (np.float32(1.0) / np.float32(block.size))
        return out

    def put(x):
        t = torch.empty(x.size + 4, device="cuda")
        t[skew:skew + x.size] = torch.as_tensor(x.reshape(-1), device="cuda")
        return t

    dg, da, dm, out = put(g), put(a), put(m), torch.zeros(g.size + 4, device="cuda")
    torch.cuda.synchronize()
    net._check(_lib.lib().pt_unet_guess(net.h, dg.data_ptr() + 4 * skew, da.data_ptr() + 4 * skew,
                                        dm.data_ptr() + 4 * skew, W, H, C, s, out.data_ptr() + 4 * skew), "guess")
    got = out[skew:skew + g.size].cpu().numpy().reshape(H, W, C)
    assert not out[:skew].any() and not out[skew + g.size:].any()
    pooled = [np.stack([pool(x[..., c]) for c in range(C)]) for x in (g, a)] + [np.stack([pool(m)] * C)]
    corr = net.forward(net.features(*(torch.as_tensor(x, device="cuda") for x in pooled))).cpu().numpy().astype(np.float64)
    ys, xs = (np.clip((np.arange(n) + 0.5) / s - 0.5, 0, k - 1) for n, k in ((H, hv), (W, wv)))
    iy, ix = np.floor(ys).astype(int), np.floor(xs).astype(int)
    jy, jx = np.minimum(iy + 1, hv - 1), np.minimum(ix + 1, wv - 1)
    wy, wx = (ys - iy)[:, None], (xs - ix)[None, :]
    top = corr[:, iy][:, :, ix] * (1 - wx) + corr[:, iy][:, :, jx] * wx
    bot = corr[:, jy][:, :, ix] * (1 - wx) + corr[:, jy][:, :, jx] * wx
    want = g + np.moveaxis(top * (1 - wy) + bot * wy, 0, 2)
    peak = np.abs(corr).max()
    tol = 2.0 ** -24 * (8 * max(hv, wv) * peak + 8 * (np.abs(g).max() + 4 * peak))
    assert np.abs(got - want).max() <= tol
