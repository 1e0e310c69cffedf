"""The prompt pass of the plain decoder (all prompt positions of a chunk in one read of the weights) against the CPU
restatement of the one-token step: tokens, the last step's logits and the residual stream, bit for bit, at the edges of
its tiles (8 / 16 / 32 tokens, 32 / 64 rows, blocks that do not fill 32 lanes, the chunk of 512 positions)."""
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


#            hidden heads kv  hd   ffn  layers prompt gen  style
CASES = [(256, 4, 2, 64, 512, 2, 2, 3, "q4"),
         (256, 4, 2, 64, 512, 2, 9, 1, "q4"),
         (512, 3, 1, 96, 928, 2, 17, 4, "q4"),           # 29 blocks per ffn row: lanes without a block
         (256, 2, 1, 128, 1056, 2, 33, 0, "q4"),         # 33 blocks: one lane with two; nothing generated
         (1024, 8, 8, 32, 2816, 1, 40, 5, "file"),       # Q8_0 matrices, biases, head norms
         (2048, 32, 8, 64, 8192, 1, 70, 2, "q4"),        # the benchmark width: the wide row tile
         (512, 4, 2, 128, 512, 1, 300, 4, "q4"),         # more positions than the value ring of the decode attention holds
         (256, 4, 1, 64, 256, 1, 530, 3, "q4")]          # two chunks; likewise


@pytest.mark.parametrize("H,nh,nkv,hd,F,L,P,G,style", CASES)
def test_prompt_pass_equals_the_one_token_steps(wd, oracle, H, nh, nkv, hd, F, L, P, G, style):
    V = 1000
    cfg = dict(hidden=H, n_heads=nh, n_kv_heads=nkv, head_dim=hd, ffn=F, vocab=V, n_layers=L, max_ctx=P + G + 1, rms_eps=1e-5)
    dec = wd.DenseDecoder(H, nh, nkv, hd, F, V, L, P + G + 1, 1e-5, 500000.0)
    dec.synth(7, 0.05)
    rng = np.random.Generator(np.random.PCG64(P))
    for l in range(L):
        for which in (wd.DT_ATTN_NORM, wd.DT_FFN_NORM):
            dec.set_tensor(l, which, (1.0 + 0.1 * rng.standard_normal(H)).astype(np.float32))
        if style == "file":
            from warpdecode_b200 import synth
            for which in (wd.DT_WQKV, wd.DT_W_DOWN):
                shp = dec.shape(which)
                w = (rng.standard_normal(shp) * 0.05).astype(np.float32)
                dec.set_tensor(l, which, synth.quantize_q8_0(w).reshape(-1), wd.TYPE_Q8_0)
            dec.set_tensor(l, wd.DT_BQKV, (0.2 * rng.standard_normal(dec.vector_len(wd.DT_BQKV))).astype(np.float32))
            for which in (wd.DT_Q_NORM, wd.DT_K_NORM):
                dec.set_tensor(l, which, (1.0 + 0.2 * rng.standard_normal(hd)).astype(np.float32))
    prompt = rng.integers(0, V, P)
    got, _ = dec.decode(prompt, G)
    logits, hidden = dec.read()
    ref = _oracle_for(wd, oracle, dec, cfg, 500000.0)
    want = ref.decode(prompt, G)
    assert np.array_equal(got, want)
    assert np.array_equal(ol.fbits(logits), ol.fbits(ref.logits))
    assert np.array_equal(ol.fbits(hidden), ol.fbits(ref.hidden))
    again, _ = dec.decode(prompt[:max(2, P // 2)], 1)          # a shorter prompt on the used caches and workspace
    assert np.array_equal(again, ref.decode(prompt[:max(2, P // 2)], 1))
    dec.close()


@pytest.mark.parametrize("H,hd,F,V,q8", [(4096, 128, 64, 700, False),           # the norm's elements in two passes over the threads
                                         (4096, 128, 96, 9441, True), (256, 64, 512, 9441, False),       # two head rows per warp, a ragged end
                                         (512, 64, 320, 20003, False), (512, 64, 320, 20003, True)])     # four rows per warp, a walk over the rows
def test_norm_and_product_in_one_kernel(wd, oracle, H, hd, F, V, q8):
    from warpdecode_b200 import synth
    cfg = dict(hidden=H, n_heads=2, n_kv_heads=1, head_dim=hd, ffn=F, vocab=V, n_layers=2, max_ctx=12, rms_eps=1e-5)
    dec = wd.DenseDecoder(H, 2, 1, hd, F, V, 2, 12, 1e-5, 500000.0)
    dec.synth(3, 0.05)
    rng = np.random.Generator(np.random.PCG64(V))
    if q8:
        for l, which in ((0, wd.DT_W_GATE_UP), (1, wd.DT_WQKV), (-1, wd.DT_OUTPUT)):
            w = (rng.standard_normal(dec.shape(which)) * 0.05).astype(np.float32)
            dec.set_tensor(l, which, synth.quantize_q8_0(w).reshape(-1), wd.TYPE_Q8_0)
    prompt = rng.integers(0, V, 3)
    got, _ = dec.decode(prompt, 6)
    logits, hidden = dec.read()
    ref = _oracle_for(wd, oracle, dec, cfg, 500000.0)
    assert np.array_equal(got, ref.decode(prompt, 6))
    assert np.array_equal(ol.fbits(logits), ol.fbits(ref.logits))
    assert np.array_equal(ol.fbits(hidden), ol.fbits(ref.hidden))
    dec.close()


@pytest.mark.parametrize("nh,nkv,hd,P,style", [(4, 2, 64, 322, "q4"),           # one position and one chunk beyond the single ring
                                               (4, 2, 64, 640, "file"), (2, 1, 64, 1090, "q4"),         # values refilled behind the scores
                                               (3, 1, 96, 500, "q4"), (3, 1, 96, 1350, "q4"), (2, 1, 128, 1400, "q4")])
def test_attention_over_a_cluster(wd, oracle, nh, nkv, hd, P, style):
    test_prompt_pass_equals_the_one_token_steps(wd, oracle, 256, nh, nkv, hd, 320, 1, P, 3, style)


def test_attention_of_a_long_decoder_at_its_first_positions(wd, oracle):
    """The cluster form is chosen by the longest context; the first positions leave some of its CTAs without keys."""
    cfg = dict(hidden=256, n_heads=2, n_kv_heads=1, head_dim=128, ffn=64, vocab=500, n_layers=1, max_ctx=2000, rms_eps=1e-5)
    dec = wd.DenseDecoder(256, 2, 1, 128, 64, 500, 1, 2000, 1e-5, 500000.0)
    dec.synth(5, 0.05)
    got, _ = dec.decode(np.arange(2), 130)
    ref = _oracle_for(wd, oracle, dec, cfg, 500000.0)
    assert np.array_equal(got, ref.decode(np.arange(2), 130))
    dec.close()


@pytest.mark.parametrize("P", [1021, 1100, 8186])
def test_attention_with_the_fewest_slots(wd, oracle, P):
    """Heads of 128 and the longest context leave four slots of 256 positions per CTA: the first refilled chunk, the one behind
    it, and the end of the range."""
    cfg = dict(hidden=256, n_heads=1, n_kv_heads=1, head_dim=128, ffn=64, vocab=500, n_layers=1, max_ctx=8192, rms_eps=1e-5)
    dec = wd.DenseDecoder(256, 1, 1, 128, 64, 500, 1, 8192, 1e-5, 500000.0)
    dec.synth(11, 0.05)
    prompt = np.random.Generator(np.random.PCG64(P)).integers(0, 500, P)
    got, _ = dec.decode(prompt, 6)
    logits, hidden = dec.read()
    ref = _oracle_for(wd, oracle, dec, cfg, 500000.0)
    assert np.array_equal(got, ref.decode(prompt, 6))
    assert np.array_equal(ol.fbits(logits), ol.fbits(ref.logits))
    assert np.array_equal(ol.fbits(hidden), ol.fbits(ref.hidden))
    dec.close()


def test_a_decoder_without_room_for_the_prompt_workspace(wd):
    """The prompt pass wants 78 MB beside this decoder's tensors. With less left it reads fewer positions at a time, with nearly
    nothing the steps read the prompt: tokens and logits are the same, and so they are after tensors have changed their type."""
    import gc
    import torch
    from warpdecode_b200 import synth
    P, G, V, F = 400, 40, 500, 16384
    prompt = np.random.Generator(np.random.PCG64(1)).integers(0, V, P)
    q8 = synth.quantize_q8_0((np.random.Generator(np.random.PCG64(2)).standard_normal((256, F)) * 0.05).astype(np.float32)).reshape(-1)

    def run(dec):
        dec.synth(4, 0.05)
        a = dec.decode(prompt, G)[0].copy(), dec.read()[0].copy()
        dec.close()
        return a

    def create():
        return wd.DenseDecoder(256, 2, 1, 64, F, V, 1, 512, 1e-5, 500000.0)

    def run_q8(dec):
        dec.synth(4, 0.05)
        dec.set_tensor(0, wd.DT_W_DOWN, q8, wd.TYPE_Q8_0)
        a = dec.decode(prompt, G)[0].copy(), dec.read()[0].copy()
        dec.close()
        return a
    want, want8 = run(create()), run_q8(create())
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    least = None
    for left in list(range(12, 64, 2)):                     # the least memory this decoder can be created in
        hog = torch.empty(free - (left << 20), dtype=torch.uint8, device="cuda")
        try:
            create().close()
            least = left
        except wd.WdError:
            pass
        del hog
        gc.collect()
        torch.cuda.empty_cache()
        if least is not None:
            break
    assert least is not None
    for more in (16, 90, 110, 200):
        hog = torch.empty(free - ((least + more) << 20), dtype=torch.uint8, device="cuda")
        for got, ref in ((run(create()), want), (run_q8(create()), want8)):
            assert np.array_equal(got[0], ref[0]) and np.array_equal(ol.fbits(got[1]), ol.fbits(ref[1])), more
        del hog
        gc.collect()
        torch.cuda.empty_cache()


@pytest.mark.parametrize("H,nh,nkv,hd,F", [(256, 16, 4, 128, 320), (512, 9, 3, 96, 32)])
def test_more_head_elements_than_hidden_or_ffn(wd, oracle, H, nh, nkv, hd, F):
    """The output product's input is the longest row of the model."""
    test_prompt_pass_equals_the_one_token_steps(wd, oracle, H, nh, nkv, hd, F, 2, 19, 6, "file")
