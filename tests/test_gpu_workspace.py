"""Calls near the end of the device's memory."""
import gc

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
MB = 1 << 20


class Full:
    """All of the device's memory but `left` bytes, held while inside."""

    def __init__(self, left):
        self.left = left

    def __enter__(self):
        import torch
        gc.collect()
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        free, _ = torch.cuda.mem_get_info()
        self.held = [torch.empty(free - self.left, dtype=torch.uint8, device="cuda")]
        left, _ = torch.cuda.mem_get_info()
        assert abs(left - self.left) < 64 * MB
        return self

    def __exit__(self, *exc):
        import torch
        self.held = []
        torch.cuda.empty_cache()


def test_linear_gives_its_operand_image_back(oracle):
    """A call leaves its image (200 MB) with the context; a larger one that fits only without it still runs, by the form that needs none."""
    import torch

    import kronos_2t_b200 as k2
    from test_gpu_kernels import _wide_matrix, upload
    torch.zeros(1, device="cuda")
    rows, cols, n0, n1 = 64, 1024, 100_000, 150_000
    m = _wide_matrix(oracle, "b4", rows, cols)
    x = np.random.Generator(np.random.PCG64(2)).standard_normal((n1, cols), np.float32)
    ctx = k2.Context(0)
    dm = upload(ctx, m)
    try:
        want = ctx.linear(dm, x[:n0])
        # the second call wants 200 MB more for x and 60 MB for the rest; its own image would be 300 MB
        with Full(160 * MB):
            got = ctx.linear(dm, x)
        assert np.array_equal(got[:n0], want)
        assert np.array_equal(got[n0:], ctx.linear(dm, x[n0:]))
    finally:
        dm.free()
        ctx.close()
