"""The super-block multiply in tensor memory (csrc/gemm_k_tc.cu) where it can go wrong: row and token counts around its tiles (128
rows, or 64 of a gate/up pair; 64 and 128 tokens), one super-block per row and several tiles per CTA, several matrices in one launch,
the sum with what is there, quants, scales and minimums of every value (the digits at their ends, the accumulators at their largest).
takes() says by which kernel, and with which tile, a multiply is done; each test but the first states what it needs. Integer arithmetic
in the reference's float order: the oracle's bits."""
import ctypes as C

import numpy as np
import pytest

import helpers as H
from brisk_llm_b200 import abi, engine, formats as F, synth

pytestmark = pytest.mark.gpu
FORMATS = (F.Q4_K, F.Q5_K, F.Q6_K, F.TQ2_0)


def takes(fmt, rows, cols, n, pair=False):
    """Tokens of the tile in tensor memory on a B200 (148 SMs); 0: the multiply stays with csrc/gemm_k.cu."""
    ask = abi.load_library().brisk_cuda_super_block_tokens
    ask.restype = C.c_uint32
    ask.argtypes = [C.c_int32, C.POINTER(C.c_uint32), C.c_uint32, C.c_uint32, C.c_uint32, C.c_int32, C.c_uint32]
    return ask(fmt, (C.c_uint32 * len(rows))(*rows), len(rows), cols, n, pair, 148)


def any_blocks(fmt, rows, cols, seed):
    """Blocks of random bytes - every quant, scale and minimum - with scales d (and dmin) of ordinary size."""
    rng = np.random.default_rng(seed)
    blocks = rng.integers(0, 256, (rows * cols // 256, F.row_bytes(fmt, 256)), dtype=np.uint8)
    d = (rng.uniform(-1.0, 1.0, (len(blocks), 2)) * 0.01).astype(np.float16)
    if fmt in (F.Q4_K, F.Q5_K):
        blocks[:, :4] = d.view(np.uint8)
    else:
        blocks[:, -2:] = d[:, :1].copy().view(np.uint8)
    return blocks.reshape(-1)


@pytest.mark.parametrize("fmt", FORMATS, ids=lambda f: F.NAMES[f])
@pytest.mark.parametrize("rows,cols,tokens", [(9001, 256, (64, 65)), (9088, 512, (128, 129, 200)), (4225, 2304, (191, 257)), (20000, 256, (130,))])
def test_rows_tokens_and_values(fmt, rows, cols, tokens):
    """On either side of the rule between the two kernels."""
    wb = any_blocks(fmt, rows, cols, seed=rows)
    x = np.random.default_rng(cols).standard_normal((max(tokens), cols)).astype(np.float32)
    x[1], x[2] = 1.0, -1.0  # quants of 127 and -127 throughout: sums at their largest
    x[3] = 0.0
    want = H.oracle_matmul(fmt, wb, rows, cols, x)
    for n in tokens:
        assert np.array_equal(engine.matmul(fmt, wb, rows, cols, x[:n]), want[:n]), n


@pytest.mark.parametrize("fmt", FORMATS, ids=lambda f: F.NAMES[f])
@pytest.mark.parametrize("rows,cols,tiles", [(40001, 256, {129: 64, 193: 128}), (9001, 2048, {65: 64, 128: 64, 129: 128}),
                                             (4225, 2304, {191: 64, 257: 128}), (18300, 1024, {65: 128, 128: 128, 193: 128})])
def test_in_tensor_memory(fmt, rows, cols, tiles):
    wb = any_blocks(fmt, rows, cols, seed=rows)
    x = np.random.default_rng(cols).standard_normal((max(tiles), cols)).astype(np.float32)
    x[1], x[2], x[3] = 1.0, -1.0, 0.0
    want = H.oracle_matmul(fmt, wb, rows, cols, x)
    for n, tile in tiles.items():
        assert takes(fmt, [rows], cols, n) == tile, n
        assert np.array_equal(engine.matmul(fmt, wb, rows, cols, x[:n]), want[:n]), n


@pytest.mark.parametrize("fmt", FORMATS, ids=lambda f: F.NAMES[f])
@pytest.mark.parametrize("hidden,n,v,tile,adds", [(4096, 130, None, 64, True), (1024, 200, None, 128, False), (1024, 200, F.Q6_K, 128, False)], ids=["added", "q-k-v", "q-k"])
def test_several_matrices_and_the_sum_with_what_is_there(fmt, hidden, n, v, tile, adds):
    """q, k and v (or q and k, V of another type) as one launch; the output projection adds to the residual stream."""
    base = synth.BITNET_2B if fmt == F.TQ2_0 else synth.LLAMA_3_2_1B
    overrides = {"embd": F.Q8_0, "gate": F.Q8_0, "up": F.Q8_0, "down": F.Q8_0}
    if v is not None and fmt != v:
        overrides["v"] = v
    spec = synth.tiny(base, layers=1, vocab=256, context=256, hidden=hidden, heads=32, kv_heads=8, head_dim=128, ffn=512, fmt=fmt, fmt_overrides=overrides)
    assert takes(fmt, [4096, 1024] if "v" in overrides else [4096, 1024, 1024], hidden, n) == tile
    assert not adds or takes(fmt, [hidden], 4096, n) == tile
    model = synth.perturb_norms(synth.generate(spec, seed=hidden))
    tokens = synth.random_tokens(spec, n, seed=n)
    oracle = H.OracleSession(model)
    with engine.CudaSession(model) as s:
        got, want = s.eval(tokens), oracle.eval(tokens)
        assert np.array_equal(s.debug_buffer("hidden", n * spec.hidden), oracle.debug_buffer("hidden", n * spec.hidden))
        assert np.array_equal(got, want)


@pytest.mark.parametrize("fmt", FORMATS, ids=lambda f: F.NAMES[f])
@pytest.mark.parametrize("ffn,n", [(4352, 131), (8448, 70)])
def test_gate_and_up_with_the_activation(fmt, ffn, n):
    base = synth.BITNET_2B if fmt == F.TQ2_0 else synth.LLAMA_3_2_1B
    spec = synth.tiny(base, layers=1, vocab=256, context=256, hidden=512, heads=4, kv_heads=2, head_dim=128, ffn=ffn, fmt=fmt, fmt_overrides={"embd": F.Q8_0})
    assert takes(fmt, [ffn, ffn], spec.hidden, n, pair=True) == 128
    model = synth.perturb_norms(synth.generate(spec, seed=ffn))
    tokens = synth.random_tokens(spec, n, seed=n)
    oracle = H.OracleSession(model)
    with engine.CudaSession(model) as s:
        got, want = s.eval(tokens), oracle.eval(tokens)
        assert np.array_equal(s.debug_buffer("hidden", n * spec.hidden), oracle.debug_buffer("hidden", n * spec.hidden))
        assert np.array_equal(got, want)
