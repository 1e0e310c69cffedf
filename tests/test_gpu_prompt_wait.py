"""The prompt pass when a wait of its tensor-core products runs out: the warp that asks for the copies stops at a tile that the host names, in front of
the first copy or with copies and MMAs under way. The call returns an error, and the decoder is as good as new."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("stop_at", [0, 1, 2])
def test_a_wait_that_runs_out_is_an_error(monkeypatch, stop_at):
    import warpdecode_b200 as wd
    hidden, heads, kv, ffn, vocab, prompt = 2048, 32, 8, 8192, 96, 400      # gate/up: 128 x 7 tiles, more than two per CTA
    tokens = np.random.Generator(np.random.PCG64(3)).integers(0, vocab, prompt).astype(np.int32)

    def decoder():
        dec = wd.DenseDecoder(hidden, heads, kv, 64, ffn, vocab, 1, prompt + 40, 1e-5, 500000.0)
        dec.synth(11, 0.05)
        return dec

    good = decoder()
    want, _ = good.decode(tokens, 3)
    short, _ = good.decode(tokens[:20], 3)
    monkeypatch.setenv("WD_PROMPT_STOP_AT", str(stop_at))
    bad = decoder()
    monkeypatch.delenv("WD_PROMPT_STOP_AT")
    for _ in range(2):
        with pytest.raises(wd.WdError, match="status 2"):
            bad.decode(tokens, 3)
        # a prompt that the other product reads: the status of the call before is gone
        got, _ = bad.decode(tokens[:20], 3)
        assert np.array_equal(got, short)
    got, _ = good.decode(tokens, 3)
    assert np.array_equal(got, want)
    bad.close()
    good.close()
