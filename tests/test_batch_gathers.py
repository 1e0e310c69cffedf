"""Who gathers a batch's activations (batch_task): where a list has tasks enough behind the places that a token's gathers start from, every
superblock of every token is handed to exactly one task. Lists shorter than a round leave the last ones to the tiles that need them."""
import pytest

import warpdecode_b200 as wd


@pytest.mark.parametrize("H,F,K", [(1024, 512, 8), (512, 1024, 8), (512, 512, 10), (2048, 512, 10), (512, 256, 4), (256, 2048, 4)])
@pytest.mark.parametrize("T", [2, 3, 4])
def test_no_gather_is_lost_to_another_tokens(H, F, K, T):
    nsb_f = F // 256
    t3 = H * nsb_f // 32
    wcta = 148 - T
    apt = min(K, ((K * t3 + wcta - 1) // wcta - 1) // t3 + 2) * nsb_f       # activation superblocks planned per token
    for cta in range(0, wcta, 7):
        desc, aux = wd.batch_tasks(H, F, K, T, T, True, 148, cta)
        desc, aux = desc.astype("int64").tolist(), aux.tolist()
        jobs = [((d >> 22) & 63) - 1 for d in desc if (d >> 22) & 63]
        assert len(set(jobs)) == len(jobs)
        wanted = sorted({a + s for d, a in zip(desc, aux) if d & 1 for s in range(nsb_f)})
        assert set(jobs) <= set(wanted)
        missing = [g for g in wanted if g not in jobs]
        assert not missing or len(desc) < 16 + len(wanted), (cta, missing)
