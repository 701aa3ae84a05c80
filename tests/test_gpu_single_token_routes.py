"""Which kernels take a session's single tokens, at the lines between them: what a call reports about the persistent kernel
(brisk_cuda_stats.persistent_steps, launches), and that the results do not depend on it. The kernels for prompts with one
token (FLAG_NO_MEGAKERNEL), which know no such lines, are the general path compared with."""
import numpy as np
import pytest

from brisk_llm_b200 import abi, engine, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("runs_out", [False, True])
def test_replayed_persistent_steps_are_counted_and_dropped_with_the_kernel(runs_out, monkeypatch):
    """The error word of the persistent kernel is read after calls that counted a persistent step. With the barrier form in a
    captured graph (BRISK_CUDA_STEP_GRAPH=1) a step is recorded once and replayed from then on: every call counts its steps.
    Once a wait has run out (the word as such a wait leaves it) nothing replays the kernel any more."""
    monkeypatch.setenv("BRISK_CUDA_STEP_SYNC", "barrier")
    monkeypatch.setenv("BRISK_CUDA_STEP_GRAPH", "1")
    if runs_out:
        monkeypatch.setenv("BRISK_CUDA_TEST_POLL_TIMEOUT", "1")
    spec = synth.tiny(synth.QWEN3_0_6B, layers=2, vocab=512, context=128)
    model = synth.generate(spec, seed=1)
    toks = synth.random_tokens(spec, 12, seed=2)
    with engine.CudaSession(model) as s, engine.CudaSession(model, flags=abi.FLAG_NO_MEGAKERNEL) as general:
        assert "on: grid barriers" in s.step_path()
        s.eval(toks[:8])
        general.eval(toks[:8])
        if runs_out:
            with pytest.raises(RuntimeError, match="timed out"):
                s.eval(toks[8:9])
            assert s.position() == 8
        for t in toks[8:]:
            assert np.array_equal(s.eval([t]), general.eval([t]))
            assert s.stats()["persistent_steps"] == (0 if runs_out else 1)
            assert (s.stats()["kernel_launches"] > 3) == runs_out  # embedding, layers, head; or one kernel per operation
        assert np.array_equal(s.generate_greedy(int(toks[0]), 5), general.generate_greedy(int(toks[0]), 5))
        assert s.stats()["persistent_steps"] == (0 if runs_out else 5)


@pytest.mark.parametrize("context,fits", [(26497, True), (33792, True), (33793, False)])
def test_long_sessions_keep_the_single_token_kernels(context, fits):
    """24 heads of 128 values: the softmax + weighted-sum kernel of csrc/attn_decode.cu takes contexts up to 33792 (their
    probabilities and its tiles in 200 KB of shared memory). The older kernel, for which 26496 is the end, does not decide."""
    spec = synth.tiny(synth.QWEN3_0_6B, layers=1, vocab=256, context=context, heads=24, kv_heads=8)
    model = synth.generate(spec, seed=3)
    toks = synth.random_tokens(spec, context, seed=4)
    with engine.CudaSession(model, max_context=1024, flags=abi.FLAG_NO_PERSISTENT) as s:
        s.eval(toks[:600])
        s.eval(toks[600:601])
        usual = s.stats()["kernel_launches"]
    with engine.CudaSession(model, flags=abi.FLAG_NO_PERSISTENT) as s, engine.CudaSession(model, flags=abi.FLAG_NO_MEGAKERNEL) as general:
        for at in (600, context - 2):  # early, and the context's last positions
            for session in (s, general):
                session.eval(toks[session.position():at])
            for t in toks[at:at + 2]:
                assert np.array_equal(s.eval([t]), general.eval([t])), s.position()
                assert (s.stats()["kernel_launches"] == usual) == fits
