"""Wide tiles (one 4-bit code per weight) against the CPU oracle and against the compact tiles, at every number of
superblocks per row, for both codebooks and their mixture, in one-token and batch calls and in a stack step."""
import numpy as np
import pytest

import oracle_lib as ol
from warpdecode_b200 import synth

pytestmark = pytest.mark.gpu
bits = ol.fbits


@pytest.mark.parametrize("H,F,gate,down", [(256, 256, 21, 21), (512, 512, 22, 22), (1024, 256, 22, 21), (2048, 512, 21, 21),
                                           (4096, 1024, 21, 21), (1024, 2048, 21, 21), (2048, 512, 22, 22)])
def test_wide_tiles_give_the_oracle_bits(oracle, monkeypatch, H, F, gate, down):
    import warpdecode_b200 as wd
    E, K, SF = 8, 2, 128
    m = synth.make_moe_block(H + F, H, F, E, K, SF, gate, down)
    rng = np.random.Generator(np.random.PCG64(H))
    for k in ("gate", "up"):
        m[k] = synth.random_blocks(rng, gate, E * F * H // 256)         # every code and scale, not only what the encoder picks
    m["down"] = synth.random_blocks(rng, down, E * H * F // 256)
    x = rng.standard_normal((3, H)).astype(np.float32)
    want = [oracle.moe_block(m, v) for v in x]
    size, res = {}, {}
    for wide in ("1", "0"):
        monkeypatch.setenv("WD_WIDE_TILES", wide)
        eng = wd.Engine(H, F, E, K, SF, 1, expert_type=gate, down_type=down, max_tokens=3)
        eng.load_block(0, m)
        size[wide] = eng.slot_bytes()
        out = eng.forward_host(0, x)
        one = eng.forward_host(0, x[0])
        for name in ("act", "expert_out"):
            assert np.array_equal(bits(eng.tap(name)), bits(want[0][name])), (wide, name)
        assert np.array_equal(bits(one), bits(want[0]["out"]))
        for t in range(3):
            assert np.array_equal(bits(out[t]), bits(want[t]["out"])), (wide, t)
        res[wide] = eng.stack_step_host(x[1])
        assert eng.device_status() == 0
        eng.close()
    assert size["1"] > size["0"] and np.array_equal(bits(res["1"]), bits(res["0"]))


def test_a_pool_that_only_fits_compact_keeps_compact_tiles():
    import warpdecode_b200 as wd
    H, F, E, L = 512, 256, 64, 4                        # compact: 168,960 bytes per expert, 41.3 MiB in all
    open_, tight = wd.Engine(H, F, E, 4, 128, L), wd.Engine(H, F, E, 4, 128, L, cache_mib=42)
    assert tight.slot_count() == open_.slot_count() == E * L
    assert tight.slot_bytes() == 168960 < open_.slot_bytes()
    open_.close(), tight.close()


@pytest.mark.parametrize("H,F,gate,up,down,f32", [(256 * 3, 64, 21, 21, 20, False), (2560, 640, 22, 22, 20, True), (1280, 192, 21, 22, 20, True),
                                                  (768, 768, 22, 22, 21, True), (4096, 256, 21, 21, 22, True), (1792, 512, 22, 21, 22, False)])
def test_wide_rows_of_the_plain_layout_path(oracle, monkeypatch, H, F, gate, up, down, f32):
    import warpdecode_b200 as wd
    E, K, SF = 8, 3, 128
    m = synth.make_moe_block(H + F, H, F, E, K, SF, gate, down, router_f32=f32)
    m["up_type"] = up
    rng = np.random.Generator(np.random.PCG64(F))
    m["gate"], m["up"] = (synth.random_blocks(rng, t, E * F * H // 256) for t in (gate, up))
    m["down"] = synth.random_blocks(rng, down, E * H * F // (32 if down == 20 else 256))
    x = rng.standard_normal((2, H)).astype(np.float32)
    want = [oracle.moe_block(m, v) for v in x]
    for wide in ("1", "0"):
        monkeypatch.setenv("WD_WIDE_TILES", wide)
        eng = wd.Engine(H, F, E, K, SF, 1, expert_type=gate, down_type=down, max_tokens=2, router_f32=f32)
        eng.load_block(0, m)
        assert eng.kernel_name() == "plain_gate_up_kernel"
        out = eng.forward_host(0, x)
        for t in range(2):
            for name in ("act", "expert_out"):
                assert np.array_equal(bits(eng.tap(name, t)), bits(want[t][name])), (wide, t, name)
            assert np.array_equal(bits(out[t]), bits(want[t]["out"])), (wide, t)
        assert eng.device_status() == 0
        eng.close()


@pytest.mark.parametrize("bad", [(1,), (0, 3), (0, 1, 2, 3)])
def test_a_batch_whose_early_picks_do_not_stand_is_decoded_again(oracle, bad):
    """Huge activations push most probabilities to zero: the k largest logits are then not the k rungs, and the tiles asked
    for before the proof belong to the wrong experts. One such token makes the whole batch decode again."""
    import warpdecode_b200 as wd
    H, F, E, K, SF = 512, 256, 64, 6, 128
    m = synth.make_moe_block(77, H, F, E, K, SF, 21, 22)
    x = np.random.Generator(np.random.PCG64(5)).standard_normal((4, H)).astype(np.float32)
    x[list(bad)] *= np.float32(1000.0)
    want = [oracle.moe_block(m, v) for v in x]
    eng = wd.Engine(H, F, E, K, SF, 1, expert_type=21, down_type=22, max_tokens=4)
    eng.load_block(0, m)
    for _ in range(3):
        out = eng.forward_host(0, x)
        for t in range(4):
            assert np.array_equal(eng.tap("ids", t), want[t]["ids"])
            for name in ("weights", "act", "expert_out"):
                assert np.array_equal(bits(eng.tap(name, t)), bits(want[t][name])), (t, name)
            assert np.array_equal(bits(out[t]), bits(want[t]["out"])), t
    assert eng.fallbacks() == 3 * len(bad) and eng.device_status() == 0
    eng.close()


@pytest.mark.parametrize("E,K,scale", [(8, 3, 1.0), (64, 10, 1000.0), (600, 10, 300.0), (16, 16, 30.0)])
def test_plain_layout_picks_from_a_threshold_or_the_rungs(oracle, E, K, scale):
    """Ordinary rows, and activations that push most probabilities to zero, where the k largest logits are not the k rungs."""
    import warpdecode_b200 as wd
    H, F, SF = 768, 64, 128
    m = synth.make_moe_block(E + K, H, F, E, K, SF, 21, 20)
    x = np.random.Generator(np.random.PCG64(E)).standard_normal((3, H)).astype(np.float32)
    x[1:] *= np.float32(scale)
    eng = wd.Engine(H, F, E, K, SF, 1, expert_type=21, down_type=20, max_tokens=3)
    eng.load_block(0, m)
    assert eng.kernel_name() == "plain_gate_up_kernel"
    out = eng.forward_host(0, x)
    for t in range(3):
        want = oracle.moe_block(m, x[t])
        assert np.array_equal(eng.tap("ids", t), want["ids"])
        assert np.array_equal(bits(eng.tap("weights", t)), bits(want["weights"]))
        assert np.array_equal(bits(out[t]), bits(want["out"])), t
    assert eng.device_status() == 0
    eng.close()
