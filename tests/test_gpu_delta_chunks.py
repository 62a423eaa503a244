"""The recurrence of prompts in chunks: lengths at the edges of a chunk, every padded head size, and decay scales for which a chunk holds fewer
tokens (a decay is at least exp(-scale), and its products over a chunk must not underflow)."""
import math

import numpy as np
import pytest

import folizen_models as fm
import folizen_ref as ref
from test_gpu_folizen import TOL, ctx, engine, portions, tokens_of  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim", [20, 100, 130, 200])
@pytest.mark.parametrize("scale", [math.exp(-0.5), 2.5, 2.6, 13.0, 60.0, 300.0])
def test_decay_scales(engine, monkeypatch, dim, scale):  # noqa: F811
    from kronos_2t_b200 import models
    sig = ref.sigmoid
    monkeypatch.setattr(models, "DELTA_DECAY_SCALE", scale)
    monkeypatch.setattr(ref, "delta_coefficients", lambda d, a, k: (np.exp(-scale * sig(d)), sig(a), k / np.sqrt(np.sum(k * k, axis=-1, keepdims=True) + 1e-6)))
    model = fm.make(64, 30, [fm.delta(2, dim, rank=5)], side=4, seed=dim)
    toks = tokens_of(model, 49)
    want, _ = ref.forward(model, toks)
    eng = engine(model, "float32", 64)
    for n in (2, 15, 16, 17, 33, 49):
        assert fm.error(eng.forward_token_ids(toks[:n], want_all=True), want[:n]).max() < TOL["float32"], n
    assert fm.error(portions(eng, toks, [17, 3, 1, 16]), want).max() < TOL["float32"]
