"""The router of prompt batches in one launch (fewer than 14336 pairs of a token and an expert at this width) and in two: experts and tokens on both
sides of the tiles of 16, against the oracle's token-by-token run, logits and routes bit for bit."""
import numpy as np
import pytest

import k2t_models as km
from test_gpu_model import ctx, make  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_experts,n_tok", [(3, 15), (3, 16), (16, 17), (17, 33), (40, 31), (256, 55), (256, 56), (250, 65), (33, 440), (129, 113)])
def test_routes_of_a_batch(ctx, oracle, n_experts, n_tok):  # noqa: F811
    cfg = dict(km.MOE_TINY, max_seq=max(n_tok + 8, km.MOE_TINY["max_seq"]))
    spec, eng, ref = make(ctx, oracle, cfg, "nf4g128", seed=5, moe=dict(layers=[0, 2], n_experts=n_experts, top_k=3, d_ff=64, bits=3, sgc=2, bias=n_experts == 17))
    try:
        tokens = np.random.Generator(np.random.PCG64(n_tok)).integers(0, km.MOE_TINY["vocab"], n_tok).tolist()
        want = np.stack([ref.forward_token(t, threads=2) for t in tokens])
        assert np.array_equal(eng.forward_token_ids(tokens, want_all=True), want)
        for layer in (0, 2):
            assert all(np.array_equal(g, w) for g, w in zip(eng.read_routes(layer), ref.last_routes(layer)))
    finally:
        eng.close()
        ref.close()
