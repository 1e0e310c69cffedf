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


@pytest.mark.parametrize("H,F,gate,down,f32", [(2048, 512, 22, 22, False), (2560, 640, 22, 20, True)])
def test_the_wide_form_leaves_the_program_its_memory(monkeypatch, H, F, gate, down, f32):
    """What the wide form takes beyond the file's form is at most a quarter of the memory that one would leave; an engine
    in the file's form serves where the wide one does not fit."""
    import gc
    import torch
    import warpdecode_b200 as wd
    monkeypatch.delenv("WD_WIDE_TILES", raising=False)
    E, L, GB = 512, 12, 1 << 30
    compact = L * E * (2 * F * (H // 256) * 82 + (H * (F // 32) * 18 if down == 20 else H * (F // 256) * 82))
    if f32:
        wide = L * E * 3 * H * F // 64 * 36
    else:
        wide = L * E * 3 * (F * (H // 256) // 32) * 4416

    def wide_engine(left):
        gc.collect()
        torch.cuda.empty_cache()
        hog = torch.empty(torch.cuda.mem_get_info()[0] - left, dtype=torch.uint8, device="cuda")
        before = torch.cuda.mem_get_info()[0]
        eng = wd.Engine(H, F, E, 8, 128, L, expert_type=gate, down_type=down, router_f32=f32)
        # the plain-layout path allocates the file's form when the tensors are set, the wide one at creation
        took = before - torch.cuda.mem_get_info()[0]
        eng.close()
        del hog
        return took > (wide + compact) // 2 if not f32 else took > wide // 2
    wd.Engine(H, F, E, 8, 128, 1, expert_type=gate, down_type=down, router_f32=f32).close()        # context, modules
    need = compact + 4 * (wide - compact)
    assert need > wide + 4 * GB                             # the quarter is the tighter bound at this size
    assert wide_engine(need + GB // 2)
    assert not wide_engine(need - GB)
    assert not wide_engine(wide + 4 * GB + GB // 2)         # fits, and would leave 4 GiB, but too little of the rest
    assert not wide_engine(compact + GB)


def test_two_plain_engines_created_before_their_tensors_are_set(oracle):
    """Each engine has its buffers when the next one looks at the free memory."""
    import warpdecode_b200 as wd
    H, F, E, K, SF = 768, 192, 16, 3, 128
    ms = [synth.make_moe_block(50 + i, H, F, E, K, SF, 21, 20) for i in range(2)]
    engs = [wd.Engine(H, F, E, K, SF, 1, expert_type=21, down_type=20) for _ in ms]
    x = np.random.Generator(np.random.PCG64(9)).standard_normal(H).astype(np.float32)
    for e, m in zip(engs, ms):
        e.load_block(0, m)
    for e, m in zip(engs, ms):
        assert np.array_equal(bits(e.forward_host(0, x)), bits(oracle.moe_block(m, x)["out"]))
        e.close()


def test_a_fused_gate_up_tensor_in_several_parts(oracle):
    """Three experts fit the staging buffer at this shape: eight go through it as 3 + 3 + 2 (down rows in ragged parts likewise)."""
    import warpdecode_b200 as wd
    H, F, E, K = 768, 576, 8, 4
    m = synth.make_moe_block(61, H, F, E, K, 128, 21, 20)
    eng = wd.Engine(H, F, E, K, 128, 1, expert_type=21, down_type=20)
    eng.load_block(0, m)
    x = np.random.Generator(np.random.PCG64(3)).standard_normal(H).astype(np.float32)
    want = bits(oracle.moe_block(m, x)["out"])
    assert np.array_equal(bits(eng.forward_host(0, x)), want)
    rng = np.random.Generator(np.random.PCG64(4))
    m2 = dict(m, gate=synth.random_blocks(rng, 21, E * F * H // 256), up=synth.random_blocks(rng, 21, E * F * H // 256))
    fused = np.concatenate([np.asarray(m2[k]).reshape(E, -1) for k in ("gate", "up")], axis=1).copy()
    down = np.ascontiguousarray(m2["down"])
    wd._check(wd.lib().wd_set_experts_fused(eng.h, 0, fused.ctypes.data, 21, down.ctypes.data, 20))
    assert np.array_equal(bits(eng.forward_host(0, x)), bits(oracle.moe_block(m2, x)["out"]))
    eng.close()
