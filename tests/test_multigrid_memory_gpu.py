"""Device memory of a multigrid call: what fits the card once has to fit it always."""
import pytest

pytestmark = pytest.mark.gpu


def test_a_call_takes_48_bytes_a_cell_at_most(cuda_lib):
    """One channel, lambda 0: u, b' and r in FP64 (24 bytes a cell), x, r, z, q in FP32
    (16), the lower levels' three FP32 arrays (4) and the flags (4/3) make 45.3; the
    arena holds a quarter more than a call asks for. The bound is what the separate
    half-sweeps took: five FP32 vectors and two arrays a lower level, 48 bytes."""
    import numpy as np
    import torch
    from paintop_b200 import _lib
    from tests import device_solve
    c = _lib.Context(0)
    try:
        def problem(n):
            rng = np.random.default_rng(n)
            mask = np.zeros((n, n), np.float32)
            mask[n // 4:n // 2, n // 4:n // 2] = 1.0
            return dict(source=rng.random((n, n), dtype=np.float32), target=rng.random((n, n), dtype=np.float32), mask=mask,
                        width=n, height=n, channels=1, tolerance=1e-6, max_iterations=50, flags=_lib.PT_FLAG_MULTIGRID)
        device_solve.solve_batch(c, [problem(64)])  # the kernels are loaded
        big = problem(4096)
        torch.empty(6 * 4096 * 4096, device="cuda")  # the test's own images come from torch's cache
        before = torch.cuda.mem_get_info()[0]
        assert device_solve.solve_batch(c, [big])[0][1][0]["converged"]
        assert before - torch.cuda.mem_get_info()[0] <= 1.25 * 48 * 4096 * 4096
    finally:
        c.close()
