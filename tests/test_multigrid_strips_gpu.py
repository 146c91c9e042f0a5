"""One iteration of the multigrid-CG solve against the numpy model of its
preconditioner, at the edges of the strips, bands and the one-block tail.

The residual after one iteration is ||r - alpha A z|| with z the V-cycle of r
and alpha = r.z / z.Az. The device evaluates z in FP32: about 60 roundings of
2^-24 a cell and level, so its residual, relative to ||r||, is within 1e-5 of
the model's in FP64."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# one strip exactly full, one column more, two and three strips, a band and one
# row more, a single coarse level, all levels in the tail but the first, the
# tail's largest level, thin images
SHAPES = [(128, 40), (129, 41), (240, 17), (241, 64), (400, 65), (9, 9), (20, 8), (65, 64), (129, 128), (131, 127),
          (9, 300), (700, 9), (1030, 515)]


@pytest.fixture(scope="module")
def ctx():
    from paintop_b200 import _lib
    with _lib.Context(0) as c:
        yield c


@pytest.mark.parametrize("w,h", SHAPES)
@pytest.mark.parametrize("lam", [0.0, 0.01])
def test_first_iteration_matches_the_model(ctx, w, h, lam):
    from oracle import mg_model as M
    from paintop_b200 import _lib
    rng = np.random.default_rng(w * 1000 + h)
    src, tgt = rng.random((h, w), dtype=np.float32), rng.random((h, w), dtype=np.float32)
    mask = (rng.random((h, w)) > 0.05).astype(np.float32)
    mask[:, w // 2:w // 2 + 2] = 0.0       # two regions; and rows without any active cell
    mask[h // 3:h // 3 + h // 5] = 0.0
    act = mask > 0.5
    act[0] = act[-1] = act[:, 0] = act[:, -1] = False
    g, a = src.astype(np.float64), tgt.astype(np.float64)
    r = np.where(act, (M.nsum(a) - (4 + lam) * a) - ((M.nsum(g) - 4 * g) - lam * a), 0.0)
    r /= np.linalg.norm(r)
    lv = M.levels(act, lam)
    z = M.vcycle(lv, r)
    az = M.apply_a(act, z, 1.0, 4.0 + lam)
    want = np.linalg.norm(r - (r * z).sum() / (z * az).sum() * az)
    _, per, _ = ctx.solve(src, tgt, mask, w, h, 1, lam=lam, tolerance=1e-12, max_iterations=1, flags=_lib.PT_FLAG_MULTIGRID)
    assert per[0]["iterations"] == 1
    assert abs(per[0]["final_residual"] - want) <= 1e-5, (per[0]["final_residual"], want)


@pytest.mark.parametrize("w,h", [(241, 64), (20, 8)])
@pytest.mark.parametrize("lam", [1e-7, 0.3, 7.0, 1e4])
def test_first_iteration_of_screened_systems(ctx, w, h, lam):
    """Divisions by a diagonal that is no power of two, far and near 4."""
    test_first_iteration_matches_the_model(ctx, w, h, lam)
