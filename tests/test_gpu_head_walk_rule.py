"""The dense decoder's output head on both sides of the line from which Q4_0 rows of fewer than 128 blocks ask for their next blocks ahead (six passes over
the grid). Logits and tokens bit for bit against the oracle."""
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


# 6 * 4 * 16 * 296 = 113,664 rows on a GPU of 148 SMs: the first that take the walk, and the last that do not
@pytest.mark.parametrize("hidden,vocab", [(2048, 113664), (2048, 113663)])
def test_head_walk_rule(wd, oracle, hidden, vocab):
    from warpdecode_b200 import synth
    cfg = dict(hidden=hidden, n_heads=4, n_kv_heads=2, head_dim=64, ffn=256, vocab=vocab, n_layers=1, max_ctx=8, rms_eps=1e-5)
    dec = wd.DenseDecoder(hidden, 4, 2, 64, 256, vocab, 1, 8, 1e-5, 500000.0)
    dec.synth(5, 0.05)
    ref = _oracle_for(wd, oracle, dec, cfg, 500000.0)
    got, _ = dec.decode(np.array([7, 11]), 4)
    assert np.array_equal(got, ref.decode(np.array([7, 11]), 4))
    logits, hid = dec.read()
    assert np.array_equal(ol.fbits(logits), ol.fbits(ref.logits)) and np.array_equal(ol.fbits(hid), ol.fbits(ref.hidden))
    dec.close()
