"""Norms of long prompts (a few threads per token, the vector in registers) against the same prompt in portions, which the other form takes."""
import numpy as np
import pytest

import folizen_models as fm
import zasesun_models as zm
from test_gpu_folizen import TOL, ctx, engine, portions, tokens_of  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width", [516, 1092, 2052])          # two, four and eight quadruples per thread, the last ones partly filled
@pytest.mark.parametrize("design", ["folizen", "zasesun"])
def test_long_prompt_and_portions(engine, design, width):  # noqa: F811
    """Norm behind a sublayer alone, with the next one's in front, and with routed pairs added."""
    model = (fm.make(width, 40, [fm.attention(2, 1, 16, 16, 20, ff=64), fm.delta(1, 16)]) if design == "folizen"
             else zm.make(width, 40, [zm.latent(2, 16, 8, 16, 24, 32, zm.moe(5, 2, 32, 16)), zm.latent(2, 16, 8, 16, 24, 32, zm.dense(64))]))
    toks = tokens_of(model, 743)
    eng = engine(model, "float32")
    whole = eng.forward_token_ids(toks, want_all=True).astype(np.float64)
    assert fm.error(portions(eng, toks, [380]), whole).max() < 2 * TOL["float32"]          # either stays within TOL of the exact values


# sublayers whose own results do not depend on the portion (window attention in bfloat16 has tiles of the batch)
BLOCKS = {
    "folizen": lambda width: fm.make(width, 40, [fm.delta(2, 16, ff=64), fm.delta(1, 16)]),
    "zasesun": lambda width: zm.make(width, 40, [zm.latent(2, 16, 8, 16, 24, 32, zm.moe(5, 2, 32, 16)), zm.latent(2, 16, 8, 16, 24, 32, zm.dense(64))]),
}


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("width", [516, 1024, 1092, 2048, 2052, 4096])
@pytest.mark.parametrize("design", ["folizen", "zasesun"])
def test_bits_of_the_other_form(engine, design, width, dtype):  # noqa: F811
    """Either form sums in the same order: the residual stream of a prompt's last token does not depend on the portion that it is in."""
    model = BLOCKS[design](width)
    toks = tokens_of(model, 743)
    eng = engine(model, dtype)
    whole = eng.forward_token_ids(toks, want_all=True)
    stream = eng.read_hidden()
    assert np.array_equal(portions(eng, toks, [372, 371]), whole)
    assert np.array_equal(eng.read_hidden(), stream)
