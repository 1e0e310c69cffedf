"""The tile lists of the batch kernel, walked on the CPU: sixteen warps per CTA, all CTAs of a grid together, every wait of the
kernel in place (a slot of the ring, the gate/up rows of other CTAs, a superblock of activations). Whatever the geometry, the
walk has to end: a warp that gathers activations may not stand in front of the gate/up tiles they come from."""
import numpy as np
import pytest

import warpdecode_b200 as wd

WARPS = 16


def walk(H, F, K, T, Tm, wide, n_cta, ring):
    """Tasks that were never finished (0: the walk ends), and the number of tiles of each kind."""
    nsb_h, nsb_f = H // 256, F // 256
    t2, t3 = F * nsb_h // 32, H * nsb_f // 32
    wcta = n_cta - (Tm if wide else 0)
    apt = min(K, ((K * t3 + wcta - 1) // wcta - 1) // t3 + 2) * nsb_f
    left = np.full((T * K, nsb_f), 8 * nsb_h)               # gate/up units of a superblock that are not published yet
    ctas = []
    for c in range(n_cta):
        desc, aux = wd.batch_tasks(H, F, K, T, Tm, wide, n_cta, c)
        d = desc.astype(np.int64)
        tasks = list(zip((d & 1).tolist(), ((d >> 1) & 3).tolist(), ((d >> 3) & 63).tolist(), ((d >> 9) & 4095).tolist(),
                         ((d >> 22) & 63).tolist(), aux.tolist()))
        jl0 = {t: p - t * K - (a - t * apt) // nsb_f for down, t, p, _, _, a in tasks if down}
        ctas.append(dict(tasks=tasks, jl0=jl0, eaten=[False] * len(tasks), half={}, state={}, at=[w for w in range(WARPS)],
                         busy=[None] * WARPS, job=[False] * WARPS))
    n_gu = sum(1 for c in ctas for t in c["tasks"] if not t[0])
    n_down = sum(len(c["tasks"]) for c in ctas) - n_gu

    def published(c, g):
        t, r = divmod(g, apt)
        return left[t * K + c["jl0"][t] + r // nsb_f, r % nsb_f] == 0

    def gather(c, w, g):
        """True when the superblock is there; a warp that asks first holds it until its rows are published."""
        if c["state"].get(g) == "done":
            return True
        if g not in c["state"]:
            c["state"][g] = w
        if c["state"][g] == w and published(c, g):
            c["state"][g] = "done"
            return True
        return False

    moved = True
    while moved:
        moved = False
        for c in ctas:
            for w in range(WARPS):
                while c["at"][w] < len(c["tasks"]):
                    i = c["at"][w]
                    down, t, pair, tile, job, aux = c["tasks"][i]
                    if not c["job"][w]:                     # the tile itself
                        if down and not all(gather(c, w, aux + s) for s in range(nsb_f)):
                            break
                        if i >= ring and not c["eaten"][i - ring]:
                            break
                        c["eaten"][i] = True
                        if not down:
                            k = (pair, tile)
                            c["half"][k] = c["half"].get(k, 0) + 1
                            if c["half"][k] == 2:
                                left[pair, tile // (8 * nsb_h)] -= 1
                        c["job"][w] = True
                        moved = True
                    g = job - 1
                    if job and (g not in c["state"] or c["state"][g] == w) and not gather(c, w, g):
                        break                               # this warp won the gather and polls
                    c["job"][w] = False
                    c["at"][w] += WARPS
                    moved = True
    return sum(len(c["tasks"]) for c in ctas) - sum(sum(c["eaten"]) for c in ctas), n_gu, n_down


@pytest.mark.parametrize("H,F,K,Tm,wide", [(2048, 1024, 8, 4, True), (2048, 1024, 8, 1, False), (2048, 1024, 16, 4, True), (2048, 512, 10, 4, True),
                                           (2048, 512, 10, 4, False), (1024, 1024, 12, 4, True), (512, 256, 4, 1, True), (256, 2048, 16, 2, True),
                                           (4096, 512, 8, 2, False), (1024, 2048, 3, 4, True), (4096, 256, 16, 4, True)])
def test_every_walk_ends(H, F, K, Tm, wide):
    for T in range(1, Tm + 1):
        for ring in (20, 48):
            stuck, n_gu, n_down = walk(H, F, K, T, Tm, wide, 148, ring)
            assert stuck == 0, (T, ring, stuck)
            assert n_gu == 2 * T * K * F * (H // 256) // 32 and n_down == T * K * H * (F // 256) // 32
