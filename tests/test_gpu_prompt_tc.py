"""The prompt pass's tensor-core product (prompt_tc_gemm_kernel) where it can go wrong, against the oracle's one-token steps, bit for bit.

A model that is wide enough for the rule to pick the kernel: token tiles of 32, 48 and 64 with a full, a nearly empty and a nearly full last tile,
row tiles of 128 with a remainder, Q4_0 and Q8_0. Which product takes which tile, and the other lengths of rows: test_gpu_prompt_tc_tiles.py."""
import numpy as np
import pytest

from test_y_dense_decoder import _oracle_for

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def wd():
    import warpdecode_b200 as w
    w.lib()
    return w


# where the rule picks the kernel: gate/up everywhere
@pytest.mark.parametrize("hidden,heads,kv,head_dim,ffn,prompt,q8", [
    (1024, 16, 4, 64, 9472, 449, False), (1024, 16, 4, 64, 9472, 512, True), (2048, 17, 1, 64, 6176, 319, False), (2048, 22, 2, 96, 6176, 300, True),
    (2048, 32, 8, 64, 8192, 65, False), (2048, 32, 8, 64, 8192, 128, True), (4096, 11, 1, 96, 3104, 97, False)])
def test_prompt_on_tensor_cores(wd, oracle, hidden, heads, kv, head_dim, ffn, prompt, q8):
    from warpdecode_b200 import synth
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
    dec.close()
