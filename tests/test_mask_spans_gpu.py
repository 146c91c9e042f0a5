"""The polygon rasteriser at the edges of its spans, runs and crossing counts,
bit for bit against the oracle; the ellipse's saturated pixels against the
oracle's formula at every pixel."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _comb(w, h, teeth):
    """Thin teeth within four pixels: many crossings among one lane's columns."""
    pts = []
    for k in range(teeth):
        x = w / 2 + 3.5 * k / teeth
        pts += [(x, 1.1), (x + 1.5 / teeth, h - 1.3)]
    return pts + [(w / 2 + 5.0, h - 1.0), (w / 2 - 1.0, h - 0.5)]


def _fan(w, h, n):
    """n edges whose rows wind up to n / 2 times around."""
    return [(w / 2 + 0.49 * w * math.cos(2 * math.pi * k * 5 / n + 0.1), h / 2 + 0.49 * h * math.sin(2 * math.pi * k * 5 / n + 0.1))
            for k in range(n)]


CASES = [(127, 9, _fan(127, 9, 7)), (128, 9, _fan(128, 9, 7)), (129, 9, _fan(129, 9, 7)), (2047, 5, _fan(2047, 5, 11)),
         (2048, 5, _fan(2048, 5, 11)), (2052, 5, _fan(2052, 5, 11)), (4100, 3, _fan(4100, 3, 9)), (64, 40, _comb(64, 40, 7)),
         (64, 40, _comb(64, 40, 9)), (300, 60, _comb(300, 60, 60)), (500, 40, _fan(500, 40, 255)), (500, 40, _fan(500, 40, 256)),
         (500, 40, _fan(500, 40, 257)), (1, 1, _fan(1, 1, 3))]


@pytest.mark.parametrize("rule", ["nonzero", "even-odd"])
@pytest.mark.parametrize("k", range(len(CASES)))
def test_polygon_spans(ctx, oracle, k, rule):
    from paintop_b200 import masks
    w, h, pts = CASES[k]
    got = masks.polygon(ctx, w, h, pts, rule).cpu().numpy()
    want = oracle.mask_polygon(w, h, pts, rule)
    assert np.array_equal(got.view(np.uint32), np.ascontiguousarray(want, np.float32).view(np.uint32))


@pytest.mark.parametrize("radii,half", [((30.0, 11.0), 0.0), ((30.0, 11.0), 2.5), ((5.0, 40.0), 7.0), ((1e-3, 20.0), 1.0),
                                        ((1e160, 1e160), 1.0), ((1e-160, 3.0), 0.0), ((1e101, 2.0), 0.5)])
def test_ellipse_saturated_pixels(ctx, oracle, radii, half):
    from paintop_b200 import masks
    got = masks.ellipse(ctx, 90, 70, (44.3, 35.9), radii, 0.6, half).cpu().numpy().astype(np.float64)
    want = oracle.mask_ellipse(90, 70, (44.3, 35.9), radii, 0.6, half)
    # hypot's last bit may differ (a few ulps of the coverage); saturated values are exact
    assert np.allclose(got, want, rtol=0, atol=1e-6, equal_nan=True)
    flat = (want == 0) | (want == 1)
    assert np.array_equal(got[flat], np.asarray(want, np.float64)[flat])
