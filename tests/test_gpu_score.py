"""log_likelihood against a log-softmax of the rows eval_all returns: lengths around the chunk, row-slice and batch edges."""
import numpy as np
import pytest

from brisk_llm_b200 import engine, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,chunk", [(2, 64), (64, 64), (65, 7), (129, 64), (513, 64), (578, 33)])
def test_log_likelihood_is_the_log_softmax_of_the_rows(n, chunk):
    spec = synth.tiny(synth.QWEN3_0_6B, layers=1, vocab=777, context=600)
    toks = synth.random_tokens(spec, n, seed=n)
    with engine.CudaSession(synth.generate(spec, seed=3)) as s:
        rows = np.concatenate([s.eval_all(toks[i:i + 64]) for i in range(0, n, 64)])[:-1]
        diff = rows - rows.max(axis=1, keepdims=True)
        want = (diff[np.arange(n - 1), toks[1:]].astype(np.float64) - np.log(np.exp(diff.astype(np.float64)).sum(axis=1))).sum()
        s.rollback(0)
        assert abs(s.log_likelihood(toks, chunk) - want) < 1e-9 * abs(want)
        assert s.position() == n
        # an error of a later chunk leaves the chunks before it appended
        s.rollback(0)
        bad = toks.copy()
        bad[-1] = spec.vocab
        with pytest.raises(RuntimeError, match="out of range"):
            s.log_likelihood(bad, chunk)
        assert s.position() == (n - 1) // chunk * chunk


def test_an_error_of_a_later_chunk_scores_nothing():
    """The chunks before the error are appended without the output head: no log-probability leaves the device, and the sequence
    goes on as if they had been evaluated."""
    spec = synth.tiny(synth.QWEN3_0_6B, layers=1, vocab=777, context=600)
    toks = synth.random_tokens(spec, 130, seed=1)
    bad = np.append(toks, np.int32(spec.vocab))
    with engine.CudaSession(synth.generate(spec, seed=3)) as s:
        s.eval(toks[:128])
        want = s.eval(toks[128:])
        s.rollback(0)
        with pytest.raises(RuntimeError, match="out of range"):
            s.log_likelihood(bad, 64)
        assert s.position() == 128
        assert s.stats()["d2h_bytes"] == 0
        assert np.array_equal(s.eval(toks[128:]), want)
