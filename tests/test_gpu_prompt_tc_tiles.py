"""The prompt pass's tensor-core product (prompt_tc_gemm_kernel) in each of its forms, against the oracle's one-token steps, bit for bit.

Each case names the matrices that the rule (wd_prompt_tile) gives to the kernel, with the tokens per tile: token tiles of 32, 48 and 64 with a full, a nearly
empty and a nearly full last tile, row tiles of 128 with a remainder, rows of one, two, three and more groups of 32 blocks with and without a short last
group, Q4_0 and Q8_0, prompts of two passes, and a shorter prompt on the same workspace."""
import numpy as np
import pytest

from test_y_dense_decoder import _oracle_for

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def wd():
    import warpdecode_b200 as w
    w.lib()
    return w


CASES = [
    # hidden, heads, kv, head_dim, ffn, prompt, q8 (all matrices but the output product's), {matrix: tokens per tile}
    (1024, 16, 4, 64, 5120, 65, False, {"gate_up": 32}),                    # one group of 32 blocks
    (1024, 16, 4, 64, 5120, 65, True, {"gate_up": 32}),
    (1024, 16, 4, 64, 9472, 449, False, {"qkv": 48, "gate_up": 64}),
    (1024, 16, 4, 64, 9472, 512, True, {"qkv": 48, "gate_up": 64, "down": 32}),     # ten groups, the last one short
    (1024, 16, 4, 64, 5120, 700, False, {"qkv": 48, "gate_up": 64}),                   # two passes; the second of 188 positions
    (2048, 32, 8, 64, 2816, 300, False, {"qkv": 64, "wo": 48, "gate_up": 64, "down": 48}),       # three groups, the last one short
    (2048, 32, 8, 64, 2816, 449, True, {"qkv": 48, "wo": 64, "gate_up": 48, "down": 64}),
    (2048, 17, 1, 64, 6176, 319, False, {"wo": 48, "gate_up": 64}),         # 34 blocks: two groups, the last one nearly empty
    (2048, 22, 2, 96, 6176, 300, True, {"qkv": 48, "wo": 48, "gate_up": 64}),      # 66 blocks: three; 193: seven
    (2048, 32, 8, 64, 8192, 65, False, {"gate_up": 48}),
    (2048, 32, 8, 64, 8192, 128, True, {"gate_up": 64}),
    (4096, 11, 1, 96, 3104, 97, False, {"gate_up": 48}),
]


def tiles_of(wd, hidden, heads, kv, head_dim, ffn, prompt, q8):
    q = wd.TYPE_Q8_0 if q8 else wd.TYPE_Q4_0
    shapes = {"qkv": ((heads + 2 * kv) * head_dim, hidden, q), "wo": (hidden, heads * head_dim, wd.TYPE_Q4_0), "gate_up": (2 * ffn, hidden, q), "down": (hidden, ffn, q)}
    return {k: t for k, v in shapes.items() if (t := wd.prompt_tile(*v, min(prompt, 512)))}


@pytest.mark.parametrize("hidden,heads,kv,head_dim,ffn,prompt,q8,tiles", CASES)
def test_prompt_takes_the_tiles_it_names(wd, oracle, hidden, heads, kv, head_dim, ffn, prompt, q8, tiles):
    from warpdecode_b200 import synth
    assert tiles_of(wd, hidden, heads, kv, head_dim, ffn, prompt, q8) == tiles
    vocab, ctx = 96, prompt + 4
    cfg = dict(hidden=hidden, n_heads=heads, n_kv_heads=kv, head_dim=head_dim, ffn=ffn, vocab=vocab, n_layers=1, max_ctx=ctx, rms_eps=1e-5)
    dec = wd.DenseDecoder(hidden, heads, kv, head_dim, ffn, vocab, 1, ctx, 1e-5, 500000.0)
    dec.synth(11, 0.05)
    rng = np.random.Generator(np.random.PCG64(hidden + ffn + prompt))
    if q8:
        for which in (wd.DT_W_DOWN, wd.DT_W_GATE_UP, wd.DT_WQKV):
            w = (rng.standard_normal(dec.shape(which)) * 0.05).astype(np.float32)
            dec.set_tensor(0, which, synth.quantize_q8_0(w).reshape(-1), wd.TYPE_Q8_0)
    tokens = rng.integers(0, vocab, prompt).astype(np.int32)
    ref = _oracle_for(wd, oracle, dec, cfg, 500000.0)
    got, _ = dec.decode(tokens, 3)
    want = ref.decode(tokens, 3)
    assert np.array_equal(got, want)
    logits, hid = dec.read()
    assert np.array_equal(logits.view(np.uint32), ref.logits.view(np.uint32))
    assert np.array_equal(hid.view(np.uint32), ref.hidden.view(np.uint32))
    short = tokens[:prompt // 2]                # on the caches and the workspace as they are now
    got, _ = dec.decode(short, 1)
    assert np.array_equal(got, ref.decode(short, 1))
    assert np.array_equal(dec.read()[0].view(np.uint32), ref.logits.view(np.uint32))
    dec.close()
