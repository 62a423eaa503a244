"""Expert projections of a prompt, an expert's (token, route) pairs side by side on the tensor cores, against the oracle's token by token
run, bit for bit."""
import numpy as np
import pytest

import k2t_models as km

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits,sgc,n_experts,top_k,hidden,d_ff,n_tok", [
    (3, 2, 3, 1, 256, 128, 90),       # more than one tile of 32 per expert
    (4, 1, 70, 3, 320, 192, 41),      # odd chunk counts, most experts with one or two pairs, some with none
    (5, 1, 6, 2, 64, 64, 33),         # one chunk
    (2, 2, 4, 4, 384, 128, 34),       # every token takes every expert: 34 pairs each
    (3, 1, 33, 2, 2112, 64, 64),      # a pass boundary of 32 chunks
])
def test_prompt_pairs_by_expert(oracle, bits, sgc, n_experts, top_k, hidden, d_ff, n_tok):
    import ctypes as C

    import kronos_2t_b200 as k2
    from k2t_internal import internal
    assert internal("experts_grouped", C.c_bool, *[C.c_uint32] * 6)(n_tok, n_tok * top_k, n_experts, hidden, d_ff, bits), "a GEMV per pair"
    cfg = dict(hidden=hidden, layers=2, n_q=4, n_kv=2, head_dim=64, inter=256, vocab=320, max_seq=96, eps=1e-6, theta=1e6)
    spec = km.build(oracle, cfg, "nf4", seed=bits + n_experts, moe=dict(layers=[0, 1], n_experts=n_experts, top_k=top_k, d_ff=d_ff, bits=bits, sgc=sgc))
    if hidden > 64:
        spec["layers"][0]["post_norm"][64:128] = 0.0          # a chunk whose activation scale is zero
    tokens = [int(t) for t in np.random.Generator(np.random.PCG64(n_tok)).integers(0, 320, n_tok)]
    ctx = k2.Context(0)
    eng, ref = k2.Engine(ctx, spec), oracle.Model(spec)
    try:
        want = np.stack([ref.forward_token(t, threads=4) for t in tokens])
        assert np.array_equal(eng.forward_token_ids(tokens, want_all=True), want)
    finally:
        eng.close(); ref.close(); ctx.close()
