"""Decode attention of heads of 64 on both sides of the line from which the values are summed in batches of 32 positions' loads (a longest context of 641
positions: two CTAs' rings no longer hold it): contexts shorter than a batch, at the ends of batches and chunks, and refilled. Bit for bit against the oracle."""
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


@pytest.mark.parametrize("max_ctx,prompt,gen", [(640, 2, 130), (641, 2, 130), (641, 600, 40), (8192, 2, 70), (8192, 1270, 20)])
def test_contexts_around_batches(wd, oracle, max_ctx, prompt, gen):
    cfg = dict(hidden=256, n_heads=2, n_kv_heads=1, head_dim=64, ffn=64, vocab=500, n_layers=1, max_ctx=max_ctx, rms_eps=1e-5)
    dec = wd.DenseDecoder(256, 2, 1, 64, 64, 500, 1, max_ctx, 1e-5, 500000.0)
    dec.synth(13, 0.05)
    tokens = np.random.Generator(np.random.PCG64(max_ctx + prompt)).integers(0, 500, prompt)
    got, _ = dec.decode(tokens, gen)
    logits, hidden = dec.read()
    ref = _oracle_for(wd, oracle, dec, cfg, 500000.0)
    assert np.array_equal(got, ref.decode(tokens, gen))
    assert np.array_equal(ol.fbits(logits), ol.fbits(ref.logits)) and np.array_equal(ol.fbits(hidden), ol.fbits(ref.hidden))
    dec.close()
