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


SWITCH = """
import sys, zlib
import numpy as np
import kronos_2t_b200 as k2
from kronos_2t_b200 import synth
cfg = dict(hidden=192, layers=2, n_q=4, n_kv=2, head_dim=64, inter=320, vocab=320, max_seq=160, eps=1e-6, theta=1e6)
ctx, crc = k2.Context(0), 0
for kv_bits in (8, 4):
    for moe in (None, dict(n_experts=4, top_k=2, d_ff=128, bits=3, sgc=1)):
        eng = k2.Engine(ctx, synth.random_model(dict(cfg, kv_bits=kv_bits), "nf4", seed=5, **(dict(moe=moe) if moe else {})))
        tokens, pos = np.random.Generator(np.random.PCG64(1)).integers(0, 320, 120).astype(np.uint32), 0
        for n in (60, 3, 1, 16, 1, 5):
            crc = zlib.crc32(eng.forward_token_ids(tokens[pos:pos + n], pos_start=pos, want_all=True).tobytes(), crc)
            pos += n
        toks, logits = eng.decode_greedy(int(tokens[pos]), pos, 4, want_logits=True)
        crc = zlib.crc32(logits.tobytes(), zlib.crc32(np.asarray(toks).tobytes(), crc))
        eng.close()
print(crc)
"""


def test_tensor_core_switch_changes_no_bits():
    """KRONOS_CUDA_TC_MIN_TOKENS: never, from one token on (single steps included), as it is: prompts, short ones and decoding."""
    from test_prompt_rules import in_process
    assert len({in_process(SWITCH, KRONOS_CUDA_TC_MIN_TOKENS=v) for v in ("0", "1", "4", "16", "100")}) == 1
