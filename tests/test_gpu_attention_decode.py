"""Single-token attention (csrc/attn_decode.cu) at the edges of its tiles: positions around the 128 of a product tile, the 256 of
a scores CTA and the tiles requested ahead, for each head width, odd head groups and a window - against the oracle."""
import numpy as np
import pytest

import helpers as H
from brisk_llm_b200 import abi, engine, synth

pytestmark = pytest.mark.gpu
SHAPES = {"group2": (synth.QWEN3_0_6B, {}), "heads64": (synth.LLAMA_3_2_1B, {}), "group3": (synth.QWEN3_0_6B, {"heads": 6, "kv_heads": 2}),
          "wide": (synth.GEMMA3_1B, {"sliding_window": 130})}


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("before", [1, 30, 126, 254, 383, 511])
def test_edges(shape, before):
    base, kw = SHAPES[shape]
    spec = synth.tiny(base, layers=1, vocab=256, context=600, **kw)
    m = synth.perturb_norms(synth.generate(spec, seed=1))
    toks = synth.random_tokens(spec, before + 3, seed=2)
    o = H.OracleSession(m)
    with engine.CudaSession(m, flags=abi.FLAG_NO_PERSISTENT) as s:
        s.eval(toks[:before])
        o.eval(toks[:before])
        for t in toks[before:]:
            got, want = s.eval([t]), o.eval([t])
            assert np.array_equal(got, want), (shape, s.position())
