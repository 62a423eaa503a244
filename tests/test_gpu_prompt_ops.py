"""Norm, SwiGLU and head preparation of prompt batches (eight lanes per 64-value block) against the oracle's token by token run, bit for bit."""
import numpy as np
import pytest

import k2t_models as km

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("head_dim,n_q,n_kv,hidden,inter,n_tok,kw,after", [
    (64, 3, 3, 192, 320, 16, dict(), 0),                                       # 9 heads, 5 chunks: partial warps and CTAs
    (64, 4, 2, 64, 64, 17, dict(qkv_bias=True, qk_norm=True), 0),              # one chunk, an odd number of tokens
    (128, 2, 1, 2112, 192, 33, dict(qk_norm=True), 1),                         # 33 chunks, norm after the rotation by position
    (128, 3, 1, 128, 2112, 131, dict(qkv_bias=True), 0),                       # more than one tile of 128 tokens
])
def test_small_operators_of_a_batch(oracle, head_dim, n_q, n_kv, hidden, inter, n_tok, kw, after):
    import kronos_2t_b200 as k2
    cfg = dict(hidden=hidden, layers=2, n_q=n_q, n_kv=n_kv, head_dim=head_dim, inter=inter, vocab=320, max_seq=160, eps=1e-6, theta=1e6, qk_norm_after_rope=after)
    spec = km.build(oracle, cfg, "b5", seed=n_tok, tied=False, **kw)
    tokens = [int(t) for t in np.random.Generator(np.random.PCG64(n_tok)).integers(0, 320, n_tok)]
    spec["embed_bf16"][tokens[5], :64] = 0          # a chunk of one token without a scale
    ctx = k2.Context(0)
    eng, ref = k2.Engine(ctx, spec), oracle.Model(spec)
    try:
        want = np.stack([ref.forward_token(t, threads=4) for t in tokens])
        assert np.array_equal(eng.forward_token_ids(tokens, want_all=True), want)
        assert np.array_equal(eng.forward_token_ids(tokens[:1], pos_start=n_tok), ref.forward_token(tokens[0], threads=4))          # the cache rows
    finally:
        eng.close(); ref.close(); ctx.close()
