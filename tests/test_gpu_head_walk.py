"""The dense decoder's output head where it asks for its next blocks ahead (rows of 64 blocks or more, four passes over the grid): the last pass with
rows for some warps only, both block types, both lengths of the norm. Logits and tokens bit for bit against the oracle."""
import numpy as np
import pytest

import oracle_lib as ol
from test_y_dense_decoder import _oracle_for

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def wd():
    import warpdecode_b200 as w
    w.lib()
    return w


# 4 * 4 * 16 * 296 = 75,776 rows on a GPU of 148 SMs: the first ones that take the walk, with remainders of 1 and 37 rows
@pytest.mark.parametrize("hidden,vocab,q8", [(2048, 75776, False), (2048, 75813, True), (4096, 75777, False)])
def test_head_walk(wd, oracle, hidden, vocab, q8):
    from warpdecode_b200 import synth
    cfg = dict(hidden=hidden, n_heads=4, n_kv_heads=2, head_dim=64, ffn=256, vocab=vocab, n_layers=1, max_ctx=8, rms_eps=1e-5)
    dec = wd.DenseDecoder(hidden, 4, 2, 64, 256, vocab, 1, 8, 1e-5, 500000.0)
    dec.synth(5, 0.05)
    if q8:
        rng = np.random.Generator(np.random.PCG64(vocab))
        w = np.tile((rng.standard_normal((1024, hidden)) * 0.05).astype(np.float32), (vocab // 1024 + 1, 1))[:vocab]
        w[-1] *= 1.5
        dec.set_tensor(0, wd.DT_OUTPUT, synth.quantize_q8_0(w).reshape(-1), wd.TYPE_Q8_0)
    ref = _oracle_for(wd, oracle, dec, cfg, 500000.0)
    got, _ = dec.decode(np.array([7, 11]), 4)
    assert np.array_equal(got, ref.decode(np.array([7, 11]), 4))
    logits, hid = dec.read()
    assert np.array_equal(ol.fbits(logits), ol.fbits(ref.logits)) and np.array_equal(ol.fbits(hid), ol.fbits(ref.hidden))
    dec.close()
