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


@pytest.mark.parametrize("layers,context,positions", [
    (2, 40960, {300: 1, 1100: 1, 2600: 1}),          # the other side would be the batched path
    (19, 40960, {20: 1}),                            # ... for layers past 160 MB too
    (2, 36000, {300: 1, 2499: 1, 2500: 0, 2501: 0}),  # the older attention kernels, faster from 2501 visible positions on
])
def test_contexts_too_long_for_the_single_token_attention(layers, context, positions):
    """Past 33 792 positions the kernels of csrc/attn_decode.cu do not run, and what was measured with them decides nothing. (0.6B files
    state 40 960 positions, and a session takes what the file states.)"""
    spec = synth.tiny(synth.QWEN3_0_6B, layers=layers, vocab=512, context=context)
    model = synth.perturb_norms(synth.generate(spec, seed=10, share_layers=True))
    toks = synth.random_tokens(spec, 2600, seed=11)
    with engine.CudaSession(model) as s, engine.CudaSession(model, flags=abi.FLAG_NO_MEGAKERNEL) as general:
        for at, persistent in positions.items():
            for session in (s, general):
                if session.position() < at:
                    session.eval(toks[session.position():at])
            assert np.array_equal(s.eval([5]), general.eval([5])), at
            assert s.stats()["persistent_steps"] == persistent, at
            for session in (s, general):
                session.rollback(at)


@pytest.mark.parametrize("layers,context,says", [(2, 640, "kernel on: tagged exchange"), (2, 640, ", up to 1024 positions"), (12, 640, ", from 513 to 1024 positions"),
                                                 (19, 640, "kernel off: layers of 16"), (19, 40960, "kernel on: tagged exchange"), (2, 36000, ", up to 2500 positions")])
def test_the_step_path_names_what_runs(layers, context, says):
    """Where no token of a session takes the persistent kernel it is not built, and the session says so."""
    spec = synth.tiny(synth.QWEN3_0_6B, layers=layers, vocab=512, context=context)
    with engine.CudaSession(synth.generate(spec, seed=12, share_layers=True)) as s:
        path = s.step_path()
        assert says in path, path
        s.eval(synth.random_tokens(spec, 513, seed=13))
        s.eval([1])
        assert s.stats()["persistent_steps"] == (0 if "off" in path else 1)


@pytest.mark.parametrize("layers", [11, 12])
def test_the_switch_at_512_positions(layers):
    """Layers past 100 MB (12 of this shape; 11 stay below): one kernel per operation up to 512 positions, the persistent
    kernel from there on, in one call and between calls; smaller models stay persistent."""
    spec = synth.tiny(synth.QWEN3_0_6B, layers=layers, vocab=512, context=640)
    model = synth.perturb_norms(synth.generate(spec, seed=5, share_layers=True))
    toks = synth.random_tokens(spec, 512, seed=6)
    with engine.CudaSession(model) as s, engine.CudaSession(model, flags=abi.FLAG_NO_MEGAKERNEL) as general:
        for session in (s, general):
            session.eval(toks[:509])
        for at in range(509, 512):
            assert np.array_equal(s.eval(toks[at:at + 1]), general.eval(toks[at:at + 1]))
            assert s.stats()["persistent_steps"] == (1 if layers < 12 else 0)
        for session in (s, general):
            session.rollback(506)
        ids, logits = s.generate_greedy(7, 10, want_logits=True)  # the tokens at 512 and later see more than 512 positions
        assert s.stats()["persistent_steps"] == (10 if layers < 12 else 4)
        want_ids, want = general.generate_greedy(7, 10, want_logits=True)
        assert np.array_equal(ids, want_ids) and np.array_equal(logits, want)
        assert np.array_equal(s.eval([3]), general.eval([3])) and s.stats()["persistent_steps"] == 1


@pytest.mark.parametrize("layers,before,after", [(2, 1, 0), (18, 1, 0), (19, 0, 0)])
def test_the_switch_at_1024_positions(layers, before, after):
    """The persistent kernel's upper lines: layers past 160 MB (19 of this shape; 18 stay below) leave it past 512 positions too,
    and no model takes it past 1024 visible ones."""
    spec = synth.tiny(synth.QWEN3_0_6B, layers=layers, vocab=512, context=1152)
    model = synth.perturb_norms(synth.generate(spec, seed=8, share_layers=True))
    toks = synth.random_tokens(spec, 1026, seed=9)
    with engine.CudaSession(model) as s, engine.CudaSession(model, flags=abi.FLAG_NO_MEGAKERNEL) as general:
        for session in (s, general):
            session.eval(toks[:1022])
        for at in range(1022, 1026):
            assert np.array_equal(s.eval(toks[at:at + 1]), general.eval(toks[at:at + 1]))
            assert s.stats()["persistent_steps"] == (before if at + 1 <= 1024 else after), at
        for session in (s, general):
            session.rollback(1021)
        ids, logits = s.generate_greedy(7, 5, want_logits=True)  # one call over the line
        assert s.stats()["persistent_steps"] == 3 * before + 2 * after
        want_ids, want = general.generate_greedy(7, 5, want_logits=True)
        assert np.array_equal(ids, want_ids) and np.array_equal(logits, want)
