"""The grid pass in one launch (small scenes) gives the oracle's grid bit for bit at the edges of its
range (one particle, a full and a ragged last warp, the largest count and one more; few cells, a partial
tile, several tiles a block, one cell more than its limit), for scenes of a batch and crowded cells."""
import numpy as np
import pytest

H = 0.0457


def check(sphlib, oracle_mod, box, counts, prec, seed, crowd=False):
    rng = np.random.default_rng(seed)
    pos = []
    for n in counts:
        p = (rng.random((n, 3)) - 0.5) * np.array(box) * 1.1
        if crowd:
            p[: n // 2] = p[:1] + rng.random((n // 2, 3)) * 0.4 * H
        pos.append(p.astype(np.float32))
    ctx = sphlib.SphContext([box] * len(counts), counts, precision=prec)
    ctx.upload(np.concatenate(pos), None, counts)
    for _ in range(2):
        cur = ctx.download()["pos"].astype(np.float32)
        ctx.pass_grid()
        cell, cnt, order = ctx.grid()
        a = c0 = 0
        for n in counts:
            if n:
                o = oracle_mod.Oracle(box, oracle_mod.CANON, threads=1)
                o.add(cur[a:a + n])
                o.update_grid()
                ocell, ocnt, oorder = o.grid()
                assert np.array_equal(cell[a:a + n], ocell.astype(np.uint32))
                assert np.array_equal(cnt[c0:c0 + ocnt.size], ocnt.astype(np.uint32))
                assert np.array_equal(order[a:a + n], oorder.astype(np.uint32))
            a += n
            c0 += cnt.size // len(counts)
        if prec == sphlib.SPH_F64:
            break  # (its moved positions are not floats)
        ctx.pass_density()
        ctx.pass_forces()
    ctx.close()


@pytest.mark.gpu
@pytest.mark.parametrize("cells,counts", [((1, 1, 1), [1]), ((3, 5, 2), [33]), ((20, 20, 10), [1000, 0, 31]),
                                          ((13, 17, 29), [8191]), ((32, 32, 64), [8192]), ((32, 32, 64), [8193]),
                                          ((31, 37, 57), [4097]), ((31, 37, 58), [4097])])
@pytest.mark.parametrize("prec", ["plain", "f64", "mixed"])
def test_grid_of_small_scenes(sphlib, oracle_mod, cells, counts, prec):
    box = tuple(float(np.float32((c - 0.5) * H)) for c in cells)
    form = {"plain": sphlib.SPH_PLAIN_F32, "f64": sphlib.SPH_F64, "mixed": sphlib.SPH_MIXED}[prec]
    check(sphlib, oracle_mod, box, counts, form, 31)
    check(sphlib, oracle_mod, box, counts, form, 32, crowd=True)
