"""The multigrid bands' flags: a single interior cell at the edges of the strips and
bands, solved by hand, and the launches of a call without iterations."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

W, H = 400, 40
COLUMNS = [1, 7, 8, 119, 120, 121, 231, 232, 343, 344, 398]
ROWS = [1, 7, 8, 15, 16, 38]


def _images():
    rng = np.random.default_rng(3)
    return rng.random((H, W), dtype=np.float32), rng.random((H, W), dtype=np.float32)


def test_single_cells_at_strip_and_band_edges(ctx):
    from paintop_b200 import _lib
    g, a = _images()
    at = [(x, y) for x in COLUMNS for y in ROWS]
    probs = []
    for x, y in at:
        mask = np.zeros((H, W), np.float32)
        mask[y, x] = 1.0
        probs.append(dict(source=g, target=a, mask=mask, width=W, height=H, channels=1, tolerance=1e-12, max_iterations=20,
                          flags=_lib.PT_FLAG_MULTIGRID))
    g, a = g.astype(np.float64), a.astype(np.float64)
    for alone in (False, True):
        res = [ctx.solve_batch([p])[0] for p in probs] if alone else ctx.solve_batch(probs)
        for (x, y), (out, per, _) in zip(at, res):
            assert per[0]["converged"]
            ring = lambda v: v[y, x - 1] + v[y, x + 1] + v[y - 1, x] + v[y + 1, x]
            want = a.copy()
            want[y, x] = (ring(a) - (ring(g) - 4.0 * g[y, x])) / 4.0
            # |u| < 2.5: half a unit in the last place of FP32, and the bar's 1e-12
            assert np.abs(out.reshape(H, W).astype(np.float64) - want).max() <= 2.0 ** -23 + 1e-11


def test_a_call_without_iterations_launches_one_kernel_a_level(ctx):
    """300 x 200 has seven levels: assembly, six coarsenings, residual, output."""
    from paintop_b200 import _lib
    rng = np.random.default_rng(1)
    img = rng.random((200, 300), dtype=np.float32)
    mask = np.ones((200, 300), np.float32)
    ctx.solve_batch([dict(source=img, target=img[::-1].copy(), mask=mask, width=300, height=200, channels=1, tolerance=1e-6,
                          max_iterations=0, flags=_lib.PT_FLAG_MULTIGRID)])
    assert ctx.last_timing()[2] <= 9
