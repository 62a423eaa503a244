"""The prompt GEMM over half-precision operand images (kronos_cuda_linear with sixteen tokens and more, prompt batches of the engine)
against the oracle's batch forms, bit for bit."""
import ctypes as C

import numpy as np
import pytest

from k2t_rng import normal
from test_gpu_kernels import _wide_matrix, upload

pytestmark = pytest.mark.gpu

FORMATS = ["b4", "b5", "b6", "nf3", "nf4", "nf4g128", "nf5g128", "e8q2"]


@pytest.fixture(scope="module")
def ctx():
    import kronos_2t_b200 as k2
    c = k2.Context(0)
    yield c
    c.close()


def _check(ctx, oracle, m, x):
    dm = upload(ctx, m)
    try:
        got = ctx.linear(dm, x)
    finally:
        dm.free()
    act = oracle.act_populate_fwht(x)
    want = oracle.nibble4_gemv(oracle.nibble4_from_bipolar(m, False), act) if m.kind == 0 else oracle.nf_gemv(m, act)
    assert np.array_equal(got, want)


@pytest.mark.parametrize("fmt", FORMATS)
@pytest.mark.parametrize("rows,cols,n_tok", [(54, 64, 16), (71, 1536, 17), (300, 2112, 33), (129, 576, 128), (260, 4160, 100), (18944, 128, 64), (18944, 192, 131)])
def test_linear_of_many_tokens(ctx, oracle, fmt, rows, cols, n_tok):
    """Odd row counts, partial tiles of 32, 64 and 128 tokens, one chunk to more than two passes of 32, zero chunks of single tokens and of all."""
    x = normal(n_tok * 7 + rows, (n_tok, cols))
    x[n_tok - 1, cols - 64:] = 0.0
    x[n_tok // 2, :] = 0.0
    if cols > 1024:
        x[:, 960:1024] = 0.0
    _check(ctx, oracle, _wide_matrix(oracle, fmt, rows, cols), x)


@pytest.mark.parametrize("fmt", ["b4", "b6", "nf3", "nf4"])
def test_largest_dots(ctx, oracle, fmt):
    """Every code and every activation of a chunk at the end of its range: the sum of the 64 products is the largest there is
    (64 x 127 x 127 for a codebook), and single products of one and of either sign decide its last digit."""
    rows, cols, n_tok = 128, 256, 48
    rng = np.random.Generator(np.random.PCG64(3))
    q = np.where(rng.random((n_tok, cols)) < 0.02, -1.0, 1.0).astype(np.float32)
    q[:, 5::64] = 1.0 / 127.0
    x = np.ascontiguousarray(q)
    for t in range(n_tok):
        oracle.lib().k2o_ifwht64(x[t].ctypes.data, cols, 0)
    if fmt.startswith("b"):
        planes = int(fmt[1])
        u = np.full((rows, cols), (1 << planes) - 1, np.uint8)
        u[1::2] = 0
        u[rng.random((rows, cols)) < 0.02] = 1
        m = oracle.bipolar_from_codes(u, np.full((rows, cols // 64), 0x3F80, np.uint16), planes)
    else:
        bits = int(fmt[2])
        idx = np.full((rows, cols), (1 << bits) - 1, np.uint8)
        idx[1::2] = 0
        idx[rng.random((rows, cols)) < 0.02] = 3
        book = np.zeros(16, np.int8)
        book[:1 << bits] = np.linspace(-127, 127, 1 << bits).round()
        m = oracle.nf_pack(idx, np.full(oracle.lib().k2o_nf_scale_count(rows, cols, 1), 0x3F80, np.uint16), bits, 1, book)
    _check(ctx, oracle, m, x)


class Image(C.Structure):
    _fields_ = [("img", C.c_void_p), ("scales", C.c_void_p), ("zero", C.c_void_p)]


def _converted(ctx, oracle, fmt, rows, cols, n_tok, sm_count):
    """The launch itself on a batch with chunks of zeros, and the oracle's product."""
    import torch

    from k2t_internal import internal
    launch = internal("launch_gemm_f16", C.c_int, C.c_void_p, C.c_void_p, C.c_void_p, C.c_void_p, C.c_uint32, C.POINTER(Image), C.c_void_p, C.c_size_t, C.c_int, C.c_void_p,
                      C.c_void_p, C.c_bool, C.c_bool)
    x = normal(n_tok * 7 + rows, (n_tok, cols))
    x[n_tok - 1, cols - 64:] = 0.0
    x[n_tok // 2, :] = 0.0
    if cols > 1024:
        x[:, 960:1024] = 0.0
    m = _wide_matrix(oracle, fmt, rows, cols)
    act = oracle.act_populate_fwht(x)
    want = oracle.nibble4_gemv(oracle.nibble4_from_bipolar(m, False), act) if m.kind == 0 else oracle.nf_gemv(m, act)
    q, s = torch.from_numpy(np.array(act.q)).cuda(), torch.from_numpy(np.array(act.scales)).cuda()
    pad = (n_tok + 127) // 128 * 128
    img, rec = (torch.full((n,), 0x7F, dtype=torch.uint8, device="cuda") for n in (pad * cols * 2 + 1024, pad // 32 * (cols // 64) * 144))
    out, err = torch.zeros(n_tok, rows, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    image = Image((img.data_ptr() + 1023) // 1024 * 1024, rec.data_ptr(), None)
    dm = upload(ctx, m)          # its handle: a KronosCudaMatrix, the DeviceMatrix first
    try:
        e = launch(torch.cuda.current_stream().cuda_stream, dm.handle, q.data_ptr(), s.data_ptr(), n_tok, C.byref(image), out.data_ptr(), rows, sm_count, err.data_ptr(), None, False, False)
        torch.cuda.synchronize()
    finally:
        dm.free()
    assert e == 0 and err.item() == 0
    return out.cpu().numpy(), want


@pytest.mark.parametrize("fmt", FORMATS)
@pytest.mark.parametrize("rows,cols,n_tok", [(54, 64, 16), (71, 1536, 17), (300, 2112, 33), (129, 576, 128), (260, 4160, 100), (18944, 128, 64), (18944, 192, 131)])
def test_product_of_converted_activations(ctx, oracle, fmt, rows, cols, n_tok):
    """The same sizes by the launch itself: kronos_cuda_linear leaves batches that the integer GEMM multiplies faster to it."""
    got, want = _converted(ctx, oracle, fmt, rows, cols, n_tok, 148)
    assert np.array_equal(got, want)


@pytest.mark.parametrize("fmt", FORMATS)
@pytest.mark.parametrize("rows,cols,n_tok,sm_count", [
    (54, 2048, 16, 148), (300, 2048, 20, 3), (129, 2560, 33, 1), (257, 4096, 64, 3), (300, 4608, 77, 3), (131, 2048, 128, 2), (300, 2048, 130, 3), (384, 2560, 500, 2), (1025, 2048, 97, 4)])
def test_products_of_long_rows(ctx, oracle, fmt, rows, cols, n_tok, sm_count):
    """Rows of 32 chunks and more, for as many CTAs as sm_count says: every width of a tile (32 to 192 tokens), the last one partly filled, several
    tiles per CTA, ragged rows, last passes of 8 chunks and more."""
    got, want = _converted(ctx, oracle, fmt, rows, cols, n_tok, sm_count)
    assert np.array_equal(got, want)
