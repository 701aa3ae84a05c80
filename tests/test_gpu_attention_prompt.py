"""Batched attention at the edges of its tiles: token counts around the row tiles, contexts around the position chunks and the
softmax's two forms, a context that is no multiple of four, and a window - one-layer models against the oracle."""
import numpy as np
import pytest

import helpers as H
from brisk_llm_b200 import engine, synth

pytestmark = pytest.mark.gpu
SHAPES = {"group2": synth.QWEN3_0_6B, "heads64": synth.LLAMA_3_2_1B, "wide": synth.GEMMA3_1B}


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("context,before,n", [(256, 0, 25), (1101, 30, 97), (1101, 990, 40), (1101, 1020, 77)])
def test_tiles_and_chunks(shape, context, before, n):
    kw = {"sliding_window": 64} if shape == "wide" else {}
    spec = synth.tiny(SHAPES[shape], layers=1, vocab=256, context=context, **kw)
    m = synth.perturb_norms(synth.generate(spec, seed=1))
    toks = synth.random_tokens(spec, before + n, seed=2)
    o = H.OracleSession(m)
    with engine.CudaSession(m) as s:
        if before:
            s.eval(toks[:before])
            o.eval(toks[:before])
        got, want = s.eval(toks[before:]), o.eval(toks[before:])
        assert np.array_equal(got, want)
