"""Batches of images that ask for different cluster sizes: launched side by side, a
stream a size, forked and joined inside the graph that device-buffer calls capture; and
which kernel a call takes, so that a comparison of the two compares two."""
import numpy as np
import pytest

from tests import device_solve
from tests.test_cluster_solve_gpu import CASES, _alike, _batch, _problem

pytestmark = pytest.mark.gpu

TILES = 6  # launches of a device-buffer call without clusters: count, compaction, assembly, init, k_solve, emit


@pytest.fixture(scope="module")
def ctx():
    from paintop_b200 import _lib
    with _lib.Context(0) as c:
        c.set_config(2)
        yield c


@pytest.mark.parametrize("w,h,box", CASES)
def test_which_kernel_a_call_takes(ctx, w, h, box):
    """The two calls that test_cluster_matches_tiles compares."""
    p = _batch([(w, h, box)], 20)[0]
    big = np.zeros(2048 * 2048, np.float32)
    other = dict(source=big, target=big, mask=big, width=2048, height=2048, channels=1, tolerance=1e-6, max_iterations=20)
    device_solve.solve_batch(ctx, [p])
    assert ctx.last_timing()[2] > TILES
    device_solve.solve_batch(ctx, [p, other])
    assert ctx.last_timing()[2] == TILES


def _other_images(probs, seed):
    """The same shapes with other images and smaller regions, whose splits differ."""
    out = []
    for k, p in enumerate(probs):
        w, h = p["width"], p["height"]
        box = (1 + (w > 20), 1 + (h > 20), max(1 + (w > 20), (w - 2) // 2), max(1 + (h > 20), 2 * (h - 2) // 3))
        src, tgt, mask = _problem(seed + k, w, h, 1, box)
        out.append(dict(p, source=src, target=tgt, mask=mask))
    return out


@pytest.mark.parametrize("take", [slice(0, 11), slice(3, 8)])
def test_mixed_batch_on_device_buffers_captured_and_replayed(ctx, take):
    first = _batch(CASES[take], 300)
    second = _other_images(first, 50)
    got = []
    for probs in (first, second, first):  # captured, then replayed with other buffers
        got.append(device_solve.solve_batch(ctx, probs, want_history=True))
        assert ctx.last_timing()[2] >= TILES + 2  # clusters of several sizes
    for a, b in zip(got[0], got[2]):
        assert np.array_equal(a[0].view(np.uint32), b[0].view(np.uint32))
        assert [r["residual_history"] for r in a[1]] == [r["residual_history"] for r in b[1]]
    for probs, res in ((first, got[0]), (second, got[1])):
        for p, a in zip(probs, res):
            _alike(a, device_solve.solve_batch(ctx, [p], want_history=True)[0])
            _alike(a, ctx.solve_batch([p], want_history=True)[0])


def test_mixed_batches_of_two_contexts_at_once(ctx):
    """Two threads, a context each: their side streams are their own."""
    import threading
    from paintop_b200 import _lib
    probs = _batch(CASES[3:8], 300)
    want = device_solve.solve_batch(ctx, probs)
    with _lib.Context(0) as other:
        other.set_config(2)
        res = {}

        def work(name, c):
            res[name] = [device_solve.solve_batch(c, probs) for _ in range(5)]

        threads = [threading.Thread(target=work, args=a) for a in (("a", ctx), ("b", other))]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
    for runs in res.values():
        for run in runs:
            for a, b in zip(run, want):
                assert np.array_equal(a[0].view(np.uint32), b[0].view(np.uint32))
