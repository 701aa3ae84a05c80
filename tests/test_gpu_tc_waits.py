"""The bounded waits of the multiplies in tensor memory (csrc/gemm_k_tc.cu, csrc/gemm_tc.cu): a wait that ran out sets a word, and the
call whose multiply it was - no other - reports it. Nothing here faults or hangs: BRISK_CUDA_TEST_TC_TIMEOUT=1 sets the word as such a
wait leaves it, 2 + k has a kernel never ask for the weights of a CTA's step k, so that the waits for them run out after 50 us."""
import numpy as np
import pytest

import helpers as H
from brisk_llm_b200 import engine, formats as F, synth

pytestmark = pytest.mark.gpu


def small_model():
    spec = synth.tiny(synth.LLAMA_3_2_1B, layers=1, vocab=256, context=256, hidden=512, heads=4, kv_heads=2, head_dim=128, ffn=8448, fmt=F.Q4_K,
                      fmt_overrides={"embd": F.Q8_0})
    return spec, synth.perturb_norms(synth.generate(spec, seed=5))


def test_a_wait_that_ran_out_is_reported_by_its_own_session(monkeypatch):
    """Two sessions of one device. The one whose wait did not run out ends its call first: its results stand, and the other still
    learns of its own."""
    spec, model = small_model()
    tokens = synth.random_tokens(spec, 70, seed=6)
    want = H.OracleSession(model).eval(tokens)
    monkeypatch.setenv("BRISK_CUDA_TEST_TC_TIMEOUT", "1")
    with engine.CudaSession(model) as failed:
        monkeypatch.delenv("BRISK_CUDA_TEST_TC_TIMEOUT")
        with engine.CudaSession(model) as sound:
            assert np.array_equal(sound.eval(tokens), want)
            with pytest.raises(RuntimeError, match="ran out"):
                failed.eval(tokens)
            sound.rollback(0)
            assert np.array_equal(sound.eval(tokens), want)
            failed.rollback(0)
            assert np.array_equal(failed.eval(tokens), want)  # reported once


def test_a_standalone_multiply_reports_its_wait(monkeypatch):
    rows, cols, n = 9088, 512, 130
    wb = np.zeros(rows * F.row_bytes(F.Q4_K, cols), np.uint8)
    x = np.ones((n, cols), np.float32)
    monkeypatch.setenv("BRISK_CUDA_TEST_TC_TIMEOUT", "1")
    with pytest.raises(RuntimeError, match="ran out"):
        engine.matmul(F.Q4_K, wb, rows, cols, x)
    with pytest.raises(RuntimeError, match="ran out"):
        engine.matmul_seconds(F.Q4_K, wb, rows, cols, n, 1, 1)
    monkeypatch.delenv("BRISK_CUDA_TEST_TC_TIMEOUT")
    assert not engine.matmul(F.Q4_K, wb, rows, cols, x).any()


@pytest.mark.parametrize("fmt,ffn,n", [(F.Q4_K, 18944, 70), (F.Q4_K, 8448, 131), (F.Q5_K, 8448, 131), (F.Q6_K, 8448, 131), (F.TQ2_0, 8448, 131), (F.Q4_0, 4352, 131)],
                         ids=["Q4_K-70", "Q4_K", "Q5_K", "Q6_K", "TQ2_0", "Q4_0"])
@pytest.mark.parametrize("step", [0, 1, 3, 7])
def test_waits_that_run_out_end_the_kernel_and_leave_the_device_sound(fmt, ffn, n, step, monkeypatch):
    """Steps at which nothing, one, a full ring and more than a ring of a CTA's copies and MMAs have been asked for; tiles of 64 and 128
    tokens of gate/up pairs, whose warps also meet at barriers (8 to 12 steps a CTA); Q4_0: the kernel of csrc/gemm_tc.cu. The call raises,
    nothing of it is left, and another session of the process goes on with the bits it had."""
    monkeypatch.setenv("BRISK_CUDA_GEMM", "tc")
    spec = synth.tiny(synth.BITNET_2B if fmt == F.TQ2_0 else synth.LLAMA_3_2_1B, layers=1, vocab=256, context=256, hidden=1024, heads=4, kv_heads=2,
                      head_dim=128, ffn=ffn, fmt=fmt, fmt_overrides={"embd": F.Q8_0})
    model = synth.perturb_norms(synth.generate(spec, seed=7))
    tokens = synth.random_tokens(spec, n, seed=8)
    with engine.CudaSession(model) as sound:
        want = sound.eval(tokens)
        monkeypatch.setenv("BRISK_CUDA_TEST_TC_TIMEOUT", str(2 + step))
        with engine.CudaSession(model) as failed:
            for _ in range(3):
                with pytest.raises(RuntimeError, match="ran out"):
                    failed.eval(tokens)
                assert failed.position() == 0
                sound.rollback(0)
                assert np.array_equal(sound.eval(tokens), want)
