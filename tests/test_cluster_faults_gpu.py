"""A cluster solve whose wait runs out, made without a GPU fault: with
PAINTOP_CUDA_FAULT=cluster-silent the last block of every cluster sends no sums of
squares, the blocks' waits for them end after 20 ms, all blocks leave together, the
call returns PT_TIMEOUT and the context stays usable."""
import numpy as np
import pytest

from tests import device_solve
from tests.test_fault_injection_gpu import injected

pytestmark = pytest.mark.gpu


def _problem(w, h, c):
    rng = np.random.default_rng(w * 7 + h)
    src, tgt = rng.random(h * w * c, dtype=np.float32), rng.random(h * w * c, dtype=np.float32)
    mask = np.zeros((h, w), np.float32)
    mask[1:h - 1, 1:w - 1] = 1.0
    return src, tgt, mask.reshape(-1)


# one block; several; sixteen of four-row patches
@pytest.mark.parametrize("w,h,c", [(30, 20, 1), (97, 71, 3), (300, 200, 2), (400, 400, 1)])
@pytest.mark.parametrize("device", [False, True])
def test_silent_block_ends_in_a_timeout_and_the_context_survives(ctx, w, h, c, device):
    from paintop_b200 import _lib
    src, tgt, mask = _problem(w, h, c)
    p = dict(source=src, target=tgt, mask=mask, width=w, height=h, channels=c, tolerance=1e-7, max_iterations=200)

    def solve():
        out, per = (device_solve.solve_batch(ctx, [p]) if device else ctx.solve_batch([p]))[0][:2]
        return out, [(r["iterations"], r["stop_reason"]) for r in per]

    want, reports = solve()
    for _ in range(2):
        with injected("cluster-silent"):
            with pytest.raises(_lib.CudaError) as e:
                solve()
        assert e.value.status == _lib.PT_TIMEOUT and "gave up" in ctx.last_error()
        got, again = solve()
        assert np.array_equal(got.view(np.uint32), want.view(np.uint32)) and again == reports


def test_budget_bounds_a_call_of_more_clusters_than_run_at_a_time(cuda_lib):
    """All systems sweep to their cap, so that a call's time is that of its waves of
    clusters; a budget of half of it ends the call, and twice it does not."""
    from paintop_b200 import _lib
    c = _lib.Context(0)
    try:
        src, tgt, mask = _problem(256, 256, 1)
        probs = [dict(source=src, target=tgt, mask=mask, width=256, height=256, channels=1, tolerance=1e-30,
                      omega=1.0, max_iterations=3000)] * 256
        c.solve_batch(probs[:1])
        one = c.last_timing()[0]
        want = c.solve_batch(probs)[-1]
        assert want[1][0]["iterations"] == 3000
        whole = c.last_timing()[0]
        assert whole > 4 * one  # waves
        c.set_budget(whole / 2e3)
        for solve in (c.solve_batch, lambda p: device_solve.solve_batch(c, p)):
            with pytest.raises(_lib.CudaError) as e:
                solve(probs)
            assert e.value.status == _lib.PT_TIMEOUT and "wall budget" in c.last_error()
        c.set_budget(whole * 2e-3)
        again = c.solve_batch(probs)[-1]
        assert np.array_equal(again[0].view(np.uint32), want[0].view(np.uint32))
    finally:
        c.close()


def test_budget_ends_one_cluster(cuda_lib):
    from paintop_b200 import _lib
    c = _lib.Context(0)
    try:
        src, tgt, mask = _problem(97, 71, 3)
        c.set_budget(1e-4)
        with pytest.raises(_lib.CudaError) as e:
            c.solve(src, tgt, mask, 97, 71, 3, max_iterations=100000, tolerance=1e-30, omega=1.0)
        assert e.value.status == _lib.PT_TIMEOUT and "wall budget" in c.last_error()
        c.set_budget(600)
        assert c.solve(src, tgt, mask, 97, 71, 3, max_iterations=10)[1][0]["iterations"] == 10
    finally:
        c.close()


@pytest.mark.parametrize("device", [False, True])
def test_without_room_for_clusters_the_tiles_solve(ctx, device):
    """PAINTOP_CUDA_FAULT=cluster-room: as where the device can place no cluster of
    sixteen blocks. The call takes k_solve alone (fewer launches) and gives the same image."""
    src, tgt, mask = _problem(97, 71, 3)
    p = dict(source=src, target=tgt, mask=mask, width=97, height=71, channels=3, tolerance=1e-7, max_iterations=200)

    def solve():
        got = (device_solve.solve_batch(ctx, [p]) if device else ctx.solve_batch([p]))[0][0]
        return got, ctx.last_timing()[2]

    want, launches = solve()
    with injected("cluster-room"):
        got, fewer = solve()
    again, same = solve()
    assert fewer < launches == same
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32)) and np.array_equal(again.view(np.uint32), want.view(np.uint32))
