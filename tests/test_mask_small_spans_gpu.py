"""The polygon rasteriser where spans get shorter and where runs have many crossings,
bit for bit against the oracle: images on either side of each span length, one to
sixteen runs; runs of seven, eight and up to 256 crossings a subsample row; runs
that end at the image's edge."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _star(seed, w, h, n, far=1.3):
    rng = np.random.default_rng(seed)
    a, r = np.sort(rng.uniform(0, 2 * math.pi, n)), rng.uniform(.1, .5 * far, n)
    return list(zip(w * (.5 + r * np.cos(a)), h * (.5 + r * np.sin(a))))


def _zigzag(w, h, teeth):
    """2 teeth + 1 crossings a row, spread over the width."""
    pts = []
    for k in range(teeth):
        pts += [(w * (k + .25) / teeth, -1.0), (w * (k + .75) / teeth, h + 1.0)]
    return pts + [(w + 2.0, h + 2.0), (-2.0, h + 2.0)]


SIZES = [(1, 1), (3, 40), (16, 5), (127, 30), (128, 30), (129, 30), (257, 700), (513, 300), (700, 1200), (1025, 640), (2049, 1185)]
SHAPES = [lambda w, h: _star(1, w, h, 3), lambda w, h: _star(2, w, h, 32), lambda w, h: _star(3, w, h, 33),
          lambda w, h: _star(4, w, h, 256), lambda w, h: _zigzag(w, h, 3), lambda w, h: _zigzag(w, h, 4),
          lambda w, h: _zigzag(w, h, 60), lambda w, h: _zigzag(w, h, 127)]


@pytest.mark.parametrize("rule", ["nonzero", "even-odd"])
@pytest.mark.parametrize("w,h", SIZES)
def test_polygon_on_small_images(ctx, oracle, w, h, rule):
    from paintop_b200 import masks
    for shape in SHAPES if w * h < 400000 else SHAPES[:1] + SHAPES[4:5]:
        pts = shape(w, h)
        got = masks.polygon(ctx, w, h, pts, rule).cpu().numpy()
        want = oracle.mask_polygon(w, h, pts, rule)
        assert np.array_equal(got.view(np.uint32), np.ascontiguousarray(want, np.float32).view(np.uint32))
