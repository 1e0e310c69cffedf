"""Expert-parallel engines one at a time on one GPU, unconnected: what a rank computes of its share, on both tile forms. Nothing
here waits for another rank (tests/test_gpu_ep.py runs connected ranks and needs two GPUs)."""
import numpy as np
import pytest

import oracle_lib as ol
from warpdecode_b200 import synth

pytestmark = pytest.mark.gpu
bits = ol.fbits


@pytest.mark.parametrize("size", [2, 4, 8])
@pytest.mark.parametrize("H,F,E,K,down", [(512, 256, 64, 6, 21), (2048, 512, 64, 10, 22)])
def test_a_rank_computes_its_share_in_either_form(oracle, monkeypatch, H, F, E, K, down, size):
    import warpdecode_b200 as wd
    SF, L = 256, 2
    ms = [synth.make_moe_block(70 + l, H, F, E, K, SF, 21, down, bias_sigma=1.0) for l in range(L)]
    rng = np.random.Generator(np.random.PCG64(size))
    xs = rng.standard_normal((4, H)).astype(np.float32)
    xs[2] *= np.float32(1000.0)                 # most probabilities underflow: the early picks do not stand
    monkeypatch.setenv("WD_COMPILED_KERNEL", "0")
    for rank in sorted({0, size // 2, size - 1}):
        first, count, got = rank * (E // size), E // size, {}
        for wide in ("1", "0"):
            monkeypatch.setenv("WD_WIDE_TILES", wide)
            eng = wd.Engine(H, F, E, K, SF, L, expert_type=21, down_type=down, ep_rank=rank, ep_size=size)
            for l, m in enumerate(ms):
                eng.load_block(l, m)
            assert eng.kernel_name() == "moe_layer_kernel" and eng.slot_count() == L * count
            for i, x in enumerate(xs):
                for l, m in enumerate(ms):
                    out, want = eng.forward_host(l, x), oracle.moe_block(m, x)
                    assert np.array_equal(eng.tap("ids"), want["ids"]) and np.array_equal(bits(eng.tap("weights")), bits(want["weights"]))
                    acc, eo, act = np.zeros(H, np.float32), eng.tap("expert_out").reshape(K, H), eng.tap("act").reshape(K, F)
                    for j, e in enumerate(want["ids"]):
                        if first <= e < first + count:
                            row = want["expert_out"].reshape(K, H)[j]
                            assert np.array_equal(bits(act[j]), bits(want["act"].reshape(K, F)[j])), (wide, i, l, j)
                            assert np.array_equal(bits(eo[j]), bits(row)), (wide, i, l, j)
                            acc = (acc + row * want["weights"][j]).astype(np.float32)
                    acc = (acc + eng.tap("shared") * eng.tap("shared_gate")[0]).astype(np.float32)
                    assert np.array_equal(bits(out), bits(acc)), (wide, i, l)
            got[wide] = [eng.stack_step_host(x) for x in xs]            # both layers in one launch
            assert eng.device_status() == 0
            eng.close()
        assert all(np.array_equal(bits(a), bits(b)) for a, b in zip(got["1"], got["0"]))
