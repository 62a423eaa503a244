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
