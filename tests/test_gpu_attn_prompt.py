"""Attention of prompt batches (rows of a kv head side by side) against the kernels that take one token and head each: the same
tokens in portions of fewer than sixteen, logits and cache rows bit for bit."""
import ctypes as C

import numpy as np
import pytest

from k2t_internal import internal

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import kronos_2t_b200 as k2
    c = k2.Context(0)
    yield c
    c.close()


# contexts around the ends of 256-position tiles and of groups of eight and four positions; batches that end inside a tile of rows
@pytest.mark.parametrize("n_q,n_kv,head_dim,past,n", [
    (4, 4, 64, 0, 16), (4, 4, 64, 3, 17), (3, 1, 64, 240, 33), (8, 1, 64, 250, 21), (7, 1, 128, 500, 29), (2, 2, 128, 1021, 40), (4, 1, 128, 0, 259),
    (2, 1, 64, 3419, 40), (2, 1, 64, 4096, 16), (2, 1, 128, 3395, 50), (1, 1, 64, 6850, 60)])
def test_prompt_attention(ctx, n_q, n_kv, head_dim, past, n):
    _compare(ctx, n_q, n_kv, head_dim, past, n, past + n + 5)


# batches of 1536 rows and more, which share rows behind any context: as many rows per CTA as their scores leave room for - sixteen up to 3424
# (head size 64) and 3344 (128) positions, eight up to 6944 and 6864, none beyond (the two kernels then).  The cache holds the batch and
# no more, so that its rows, rounded up to 32, are the context that the launch is sized for
@pytest.mark.parametrize("n_q,n_kv,head_dim,past,n,rows", [
    (32, 8, 64, 240, 49, 16), (32, 4, 64, 250, 53, 16), (28, 4, 128, 500, 61, 16), (32, 32, 64, 1021, 48, 16), (24, 3, 128, 2000, 70, 16),
    (32, 4, 64, 3424 - 51, 51, 16), (32, 4, 64, 3424 - 50, 51, 8), (32, 8, 128, 3328 - 50, 50, 16), (32, 8, 128, 3328 - 49, 50, 8),
    (32, 4, 64, 5000, 260, 8), (32, 4, 64, 6944 - 51, 51, 8), (32, 4, 64, 6944 - 50, 51, 0), (32, 8, 128, 6848 - 50, 50, 8), (32, 8, 128, 6848 - 49, 50, 0)])
def test_many_rows(ctx, n_q, n_kv, head_dim, past, n, rows):
    at = -(-(past + n) // 32) * 32
    assert internal("attention_prompt_rows", C.c_uint32, C.c_uint32, C.c_uint32)(head_dim, min(at, -(-(past + n) // 128) * 128)) == rows
    assert internal("attention_prompt_pays", C.c_bool, *[C.c_uint32] * 5)(n, n_q, n_kv, head_dim, at)
    _compare(ctx, n_q, n_kv, head_dim, past, n, past + n)


def _compare(ctx, n_q, n_kv, head_dim, past, n, max_seq):
    import kronos_2t_b200 as k2
    from kronos_2t_b200 import synth
    cfg = dict(hidden=128, layers=2, n_q=n_q, n_kv=n_kv, head_dim=head_dim, inter=128, vocab=128, max_seq=max_seq, eps=1e-5, theta=1e4)
    spec = synth.random_model(cfg, "b5", seed=n_q * 1000 + past, qkv_bias=True)
    rng = np.random.Generator(np.random.PCG64(past + n))
    tokens = rng.integers(0, cfg["vocab"], past + n)
    a, b = k2.Engine(ctx, spec), k2.Engine(ctx, spec)
    try:
        if past:
            a.forward_token_ids(tokens[:past])
            b.kv_import(a.kv_export(0, past), past)
        got = a.forward_token_ids(tokens[past:], pos_start=past, want_all=True)
        want = np.concatenate([b.forward_token_ids(tokens[p:min(p + 15, past + n)], pos_start=p, want_all=True) for p in range(past, past + n, 15)])
        assert np.array_equal(got, want)
        assert np.array_equal(a.read_attention(), b.read_attention())
        assert np.array_equal(a.kv_export(past, past + n), b.kv_export(past, past + n))
    finally:
        a.close()
        b.close()
