"""The in-cluster SOR solve (rbsor_cluster.cu) against the tile kernel.

A call of few values takes the cluster kernel; the same image beside a large
one takes the tile kernel. Both run the same iteration with the same arithmetic
a cell, so outputs and iteration counts agree bit for bit; the histories' sums of squares are taken in
another order (n terms in FP64: a relative difference of at most n 2^-53, 1e-10
for the largest region here)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from paintop_b200 import _lib
    with _lib.Context(0) as c:
        c.set_config(2)
        yield c


def _problem(seed, w, h, c, box):
    rng = np.random.default_rng(seed)
    src, tgt = rng.random((h, w, c), dtype=np.float32), rng.random((h, w, c), dtype=np.float32)
    mask = np.zeros((h, w), np.float32)
    x0, y0, x1, y1 = box
    mask[y0:y1 + 1, x0:x1 + 1] = rng.random((y1 + 1 - y0, x1 + 1 - x0)) > 0.1
    mask[y0, x0] = mask[y1, x1] = 1.0  # the region's bounding box is the box
    return src.reshape(-1), tgt.reshape(-1), mask.reshape(-1)


# (width, height, box): one cell; one row; a patch's edges in x and y; odd first
# rows; blocks of 224 patches exactly full and one row more (two- and four-row
# patches); 16 blocks; blocks of 480; an image too wide for any cluster
CASES = [
    (3, 3, (1, 1, 1, 1)), (40, 5, (1, 2, 38, 2)), (33, 17, (1, 1, 31, 15)), (34, 20, (8, 3, 15, 10)),
    (64, 64, (7, 1, 16, 62)), (70, 66, (9, 5, 60, 64)), (250, 30, (1, 1, 248, 14)), (250, 30, (1, 1, 248, 15)),
    (1800, 36, (1, 1, 1790, 33)), (1800, 36, (3, 2, 1780, 9)), (512, 300, (20, 11, 490, 285)), (700, 420, (1, 1, 698, 418)),
    (4100, 60, (1, 1, 4098, 40)), (96, 1100, (3, 1, 90, 1090)),
]


@pytest.mark.parametrize("w,h,box", CASES)
def test_cluster_matches_tiles(ctx, w, h, box):
    c, cap = (3 if w * h < 40000 else 1), 60
    src, tgt, mask = _problem(w + h, w, h, c, box)
    p = dict(source=src, target=tgt, mask=mask, width=w, height=h, channels=c, lam=0.003 * (w % 3), tolerance=1e-7,
             omega=1.7, max_iterations=cap if w % 2 else 400)
    big = np.zeros(2048 * 2048, np.float32)
    other = dict(source=big, target=big, mask=big, width=2048, height=2048, channels=1)
    small = ctx.solve_batch([p], want_history=True)[0]
    tiles = ctx.solve_batch([p, other], want_history=True)[0]
    assert np.array_equal(small[0].view(np.uint32), tiles[0].view(np.uint32))
    for a, b in zip(small[1], tiles[1]):
        assert (a["iterations"], a["stop_reason"], a["refinements"]) == (b["iterations"], b["stop_reason"], b["refinements"])
        np.testing.assert_allclose(a["residual_history"], b["residual_history"], rtol=1e-10)


def _alike(a, b):
    """Images and counts bit for bit, histories to the order of their sums."""
    assert np.array_equal(a[0].view(np.uint32), b[0].view(np.uint32))
    for x, y in zip(a[1], b[1]):
        assert (x["iterations"], x["stop_reason"], x["refinements"]) == (y["iterations"], y["stop_reason"], y["refinements"])
        np.testing.assert_allclose(x["residual_history"], y["residual_history"], rtol=1e-10)


def _batch(shapes, cap):
    probs = []
    for k, (w, h, box) in enumerate(shapes):
        src, tgt, mask = _problem(k, w, h, 1, box)
        probs.append(dict(source=src, target=tgt, mask=mask, width=w, height=h, channels=1, lam=0.01 * (k % 2),
                          tolerance=1e-6, omega=1.8, max_iterations=cap))
    return probs


# images that ask for one cluster size, their regions of many: every split of it
SAME = [[(250, 250, (1 + k, 2 * k, 248 - 20 * k, 240 - 9 * k)) for k in range(1, 10)],
        [(64, 64, (1 + k, 1 + k % 3, 62 - 3 * k, 62 - k)) for k in range(12)]]


@pytest.mark.parametrize("shapes", SAME)
def test_cluster_batch_and_reruns(ctx, shapes):
    """Regions of one call, each as if solved alone, twice the same."""
    probs = _batch(shapes, 300)
    first, again = (ctx.solve_batch(probs, want_history=True) for _ in range(2))
    for p, a, b in zip(probs, first, again):
        alone = ctx.solve_batch([p], want_history=True)[0]
        for x in (b, alone):
            assert np.array_equal(a[0].view(np.uint32), x[0].view(np.uint32))
            assert [r["residual_history"] for r in a[1]] == [r["residual_history"] for r in x[1]]


def test_batch_of_every_class(ctx):
    """Images that ask for different clusters, or for too many large ones, are the
    tile kernel's; each ends as if solved alone."""
    for probs in (_batch(CASES[:11], 300), _batch([(512, 300, (20, 11, 490, 285))] * 8, 60)):
        for p, a in zip(probs, ctx.solve_batch(probs, want_history=True)):
            _alike(a, ctx.solve_batch([p], want_history=True)[0])


# (count x width x height is 4e6 and more)
@pytest.mark.parametrize("count,w,h,box", [(44, 250, 382, (1, 1, 248, 380)), (53, 257, 300, (3, 2, 255, 297)),
                                           (90, 64, 700, (1, 1, 62, 698)), (62, 256, 256, (5, 7, 250, 248))])
def test_cluster_of_many_values(ctx, count, w, h, box):
    """4e6 values and more in images that the least blocks hold: patches of four rows
    first. Each region as if solved alone, where patches of two rows come first."""
    x0, y0, x1, y1 = box
    probs = _batch([(w, h, (x0 + k % 3, y0 + k % 5, x1 - k % 4, y1 - k % 7)) for k in range(count)], 120)
    many = ctx.solve_batch(probs, want_history=True)
    for p, a in list(zip(probs, many))[::9]:
        _alike(a, ctx.solve_batch([p], want_history=True)[0])


@pytest.mark.parametrize("config", range(5))
@pytest.mark.parametrize("w,h,box", [(5, 4, (1, 1, 3, 2)), (114, 86, (1, 1, 112, 84)), (113, 85, (1, 2, 111, 82)), (241, 175, (2, 1, 239, 171))])
def test_tiles_of_every_config(w, h, box, config):
    """The tile kernel's row and column remainders in each tile size, against the cluster kernel."""
    from paintop_b200 import _lib
    with _lib.Context(0) as c:
        c.set_config(config)
        test_cluster_matches_tiles(c, w, h, box)


@pytest.mark.parametrize("count", [1, 30, 31, 32, 63, 100])
def test_tiles_of_many_systems(ctx, count):
    """Systems beside a large image take the tile kernel, whose blocks look for work
    32 systems at a time; each ends as if solved alone."""
    big = np.zeros(2048 * 2048, np.float32)
    probs = [dict(source=big, target=big, mask=big, width=2048, height=2048, channels=1)]
    for k in range(count):
        w, h = 20 + 7 * (k % 9), 12 + 5 * (k % 11)
        src, tgt, mask = _problem(k, w, h, 1, (1, 1, w - 2, h - 2))
        probs.append(dict(source=src, target=tgt, mask=mask, width=w, height=h, channels=1, lam=0.0, tolerance=1e-6,
                          omega=1.7, max_iterations=20 + 13 * (k % 7)))
    for p, a in list(zip(probs, ctx.solve_batch(probs)))[1::7]:
        alone = ctx.solve_batch([p])[0]
        assert np.array_equal(a[0].view(np.uint32), alone[0].view(np.uint32))
        assert [r["iterations"] for r in a[1]] == [r["iterations"] for r in alone[1]]
