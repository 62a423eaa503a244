"""The experts of a prompt in tiles of 32 pairs: more tiles than CTAs, experts with one pair to two tiles, rows of a few chunks that are no whole slots, rows of
32 chunks and more, ragged last row tiles, every width of an expert's codes, bit for bit."""
import ctypes as C

import numpy as np
import pytest

import k2t_models as km
from k2t_internal import internal
from test_gpu_model import ctx, make  # noqa: F401

pytestmark = pytest.mark.gpu


def check(ctx, oracle, bits, hidden, d_ff, sgc, n_tok, n_experts, k):  # noqa: F811
    cfg = dict(km.MOE_TINY, hidden=hidden, layers=2, max_seq=160)
    assert internal("experts_grouped", C.c_bool, *[C.c_uint32] * 6)(n_tok, n_tok * k, n_experts, cfg["hidden"], d_ff, bits)
    spec, eng, ref = make(ctx, oracle, cfg, "nf4g128", seed=bits, moe=dict(layers=[0, 1], n_experts=n_experts, top_k=k, d_ff=d_ff, bits=bits, sgc=sgc))
    try:
        tokens = np.random.Generator(np.random.PCG64(bits)).integers(0, cfg["vocab"], n_tok)
        want = np.stack([ref.forward_token(int(t), threads=4) for t in tokens])
        assert np.array_equal(eng.forward_token_ids(tokens, want_all=True), want)
    finally:
        eng.close()
        ref.close()


@pytest.mark.parametrize("bits,d_ff,sgc", [(2, 320, 1), (3, 320, 1), (3, 384, 2), (4, 320, 1), (5, 320, 1)])
def test_experts_of_a_prompt(ctx, oracle, bits, d_ff, sgc):  # noqa: F811
    check(ctx, oracle, bits, 640, d_ff, sgc, 150, 32, 8)


# gate_up of 32, 33 and 40 chunks (a whole pass, one chunk more, a pass of whole slots behind it; 2112: down's last row tile is half full), down of 33 chunks
@pytest.mark.parametrize("bits", [2, 3, 4, 5])
@pytest.mark.parametrize("hidden,d_ff,sgc", [(2048, 64, 1), (2048, 128, 2), (2112, 64, 1), (2560, 128, 2), (192, 2112, 1)])
def test_long_rows(ctx, oracle, bits, hidden, d_ff, sgc):  # noqa: F811
    check(ctx, oracle, bits, hidden, d_ff, sgc, 70, 5, 2)
