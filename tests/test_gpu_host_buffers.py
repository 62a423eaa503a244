"""kronos_cuda_linear on page-locked host buffers (read by the kernel where they lie, small results stored by one) against pageable ones (copied):
the same bits, at sizes on both sides of the limit for stored results, at addresses the kernels cannot take, for calls queued one behind another."""
import numpy as np
import pytest

from k2t_rng import normal
from test_gpu_kernels import _wide_matrix, upload

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import kronos_2t_b200 as k2
    c = k2.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("rows,cols,n_tok", [(5, 64, 1), (71, 576, 3), (16384, 64, 1), (16385, 64, 1), (300, 2048, 40), (64, 8192, 16), (64, 8192, 17)])
@pytest.mark.parametrize("shift_x,shift_out", [(0, 0), (1, 0), (2, 4), (0, 3)])
def test_pinned_and_pageable(ctx, oracle, rows, cols, n_tok, shift_x, shift_out):
    import torch
    x = normal(rows + cols, (n_tok, cols))
    dm = upload(ctx, _wide_matrix(oracle, "b4", rows, cols))
    try:
        want = ctx.linear(dm, x)
        px, po = torch.zeros(x.size + 8).pin_memory(), torch.full((n_tok * rows + 8,), -7.0).pin_memory()
        px[shift_x:shift_x + x.size] = torch.from_numpy(x.reshape(-1))
        ctx.linear_ptr(dm, px.data_ptr() + 4 * shift_x, n_tok, po.data_ptr() + 4 * shift_out)
    finally:
        dm.free()
    got = po.numpy()
    assert np.array_equal(got[shift_out:shift_out + want.size].reshape(want.shape), want)
    assert (got[:shift_out] == -7).all() and (got[shift_out + want.size:] == -7).all()


def test_queued_calls_follow_one_another(ctx, oracle):
    """A queued call may take the result of the one before it from host memory."""
    import torch
    a, b = upload(ctx, _wide_matrix(oracle, "b4", 640, 128)), upload(ctx, _wide_matrix(oracle, "b5", 96, 640))
    try:
        x = normal(5, (1, 128))
        want = ctx.linear(b, ctx.linear(a, x))
        for _ in range(20):
            p = [torch.zeros(n).pin_memory() for n in (128, 640, 96)]
            p[0][:] = torch.from_numpy(x[0])
            ctx.linear_async_ptr(a, p[0].data_ptr(), 1, p[1].data_ptr())
            ctx.linear_async_ptr(b, p[1].data_ptr(), 1, p[2].data_ptr())
            ctx.synchronize()
            assert np.array_equal(p[2].numpy(), want[0])
    finally:
        a.free()
        b.free()
