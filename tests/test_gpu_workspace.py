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


@pytest.mark.parametrize("kv_bits,window,past,max_seq", [(8, 0, 7100, 8300), (4, 0, 700, 8300), (8, 8000, 8200, 9000)])
def test_scores_in_portions(kv_bits, window, past, max_seq):
    """Batches of more tokens than the score scratch holds (half a GB: 504 tokens of 32 heads over 8320 rows): as batches of 256 give it, bit for
    bit.  Contexts that the row-sharing attention leaves alone."""
    import kronos_2t_b200 as k2
    from kronos_2t_b200 import synth
    n = 512
    cfg = dict(hidden=64, layers=2, n_q=32, n_kv=4, head_dim=64, inter=64, vocab=128, max_seq=max_seq, eps=1e-5, theta=1e4, kv_bits=kv_bits, kv_window=window, kv_sinks=4)
    assert 256 <= (512 << 20) // (32 * (max_seq if not window else window + 512) * 4) < 512
    tokens = np.random.Generator(np.random.PCG64(n)).integers(0, 128, past + n).astype(np.uint32)
    ctx = k2.Context(0)
    a, b = (k2.Engine(ctx, synth.random_model(cfg, "b4", seed=4)) for _ in range(2))
    try:
        for e in (a, b):
            e.forward_token_ids(tokens[:past])
        got = a.forward_token_ids(tokens[past:], pos_start=past, want_all=True)
        want = np.concatenate([b.forward_token_ids(tokens[p:p + 256], pos_start=p, want_all=True) for p in range(past, past + n, 256)])
        assert np.array_equal(got, want)
        assert np.array_equal(a.read_attention(), b.read_attention())
        p = past + n
        assert np.array_equal(a.forward_token_ids(tokens[:1], pos_start=p), b.forward_token_ids(tokens[:1], pos_start=p))
    finally:
        a.close(); b.close(); ctx.close()


def test_score_scratch_of_a_long_cache():
    """32 heads over 32768 positions: scores of 256 tokens (1.07 GB), whatever the batch."""
    import torch

    import kronos_2t_b200 as k2
    from kronos_2t_b200 import synth
    cfg = dict(hidden=64, layers=1, n_q=32, n_kv=4, head_dim=64, inter=64, vocab=128, max_seq=32768, eps=1e-5, theta=1e4)
    spec = synth.random_model(cfg, "b4", seed=4)
    ctx = k2.Context(0)
    k2.Engine(ctx, synth.random_model(dict(cfg, max_seq=64), "b4", seed=4)).close()
    torch.cuda.synchronize()
    before, _ = torch.cuda.mem_get_info()
    e = k2.Engine(ctx, spec)
    try:
        taken = before - torch.cuda.mem_get_info()[0]
        scores, cache = 256 * 32 * (32768 + 256) * 4, 4 * 32768 * 64 * 3
        rest = 512 * (4 * 40 * 64 * 4 + 2048 * 12 + 128 * 4)          # vectors, activations, image
        assert taken < scores + cache + rest + 64 * MB
    finally:
        e.close(); ctx.close()


@pytest.mark.parametrize("left_mb", [3000, 2200, 1400, 800])
def test_engine_with_smaller_batches_where_memory_is_short(left_mb):
    """Weights of 0.1 GB, a workspace of 1.74 GB for batches of 512 tokens, 0.87 for 256, 0.44 for 128.  3 GB hold 512 and the spare half;
    2.2 GB not the spare half, 1.4 GB not 512, 0.8 GB not 256.  Same bits as an engine with all the memory."""
    import torch

    import kronos_2t_b200 as k2
    from kronos_2t_b200 import synth
    torch.zeros(1, device="cuda")
    cfg = dict(hidden=64, layers=2, n_q=2, n_kv=1, head_dim=64, inter=64 * 2048, vocab=524288, max_seq=640, eps=1e-5, theta=1e4)
    spec = synth.random_model(cfg, "b4", seed=4)
    tokens = np.random.Generator(np.random.PCG64(3)).integers(0, 128, 600).astype(np.uint32)
    ctx = k2.Context(0)
    try:
        e = k2.Engine(ctx, spec)
        want = e.forward_token_ids(tokens), e.forward_token_ids(tokens[:1], pos_start=600)
        e.close()
        with Full(left_mb * MB):
            e = k2.Engine(ctx, spec)
            got = e.forward_token_ids(tokens), e.forward_token_ids(tokens[:1], pos_start=600)
            e.close()
        assert all(np.array_equal(a, b) for a, b in zip(got, want))
    finally:
        ctx.close()
