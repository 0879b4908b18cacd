"""sph_get_grid of a batch right after particles were appended to a scene before others, on both cell multiples: the
reference's grid of the positions that a download gives, and the same when asked again."""
import numpy as np
import pytest

H = np.float32(0.0457)


@pytest.mark.gpu
@pytest.mark.parametrize("form", ["SPH_PLAIN_F32", "SPH_MIXED"])
@pytest.mark.parametrize("multiple", [1, 2])
def test_grid_of_a_batch_after_appending(sphlib, form, multiple):
    rng = np.random.default_rng(11)
    sizes = [77, 1, 7709]
    boxes = [(0.16, 0.2, 0.16), (0.1, 0.1, 0.1), (0.5, 0.7, 0.5)]
    parts = [((rng.random((n, 3)) - 0.5) * np.array(b)).astype(np.float32) for n, b in zip(sizes, boxes)]
    ctx = sphlib.SphContext(boxes, [n + 50 for n in sizes], precision=getattr(sphlib, form))
    if multiple == 2:
        ctx.set_cell_multiple(2)
    ctx.upload(np.concatenate(parts), None, sizes)
    for scene in (0, 1, 0):
        ctx.append(scene, ((rng.random((5, 3)) - 0.5) * 0.09).astype(np.float32))
        ctx.pass_grid()
        grids = [ctx.grid(), ctx.grid()]
        pos, counts, at, base = ctx.download()["pos"], ctx.counts(), 0, 0
        for s, box in enumerate(boxes):
            res = ctx.resolution(s)
            n, nc = int(counts[s]), int(np.prod(res))
            half = np.array([np.float32(b) / np.float32(2) for b in box], np.float64)
            q = np.floor((pos[at:at + n].astype(np.float64) + half) / np.float64(H)).astype(np.int64)
            q = np.clip(q, 0, np.array(res) - 1)
            want = q[:, 0] + res[0] * (q[:, 1] + res[1] * q[:, 2])
            for cell, cnt, order in grids:
                assert np.array_equal(cell[at:at + n], want), (scene, s)
                assert np.array_equal(cnt[base:base + nc], np.bincount(want, minlength=nc))
                assert np.array_equal(order[at:at + n], np.argsort(want, kind="stable"))
            at, base = at + n, base + nc
        ctx.pass_density()
        ctx.pass_forces()
    ctx.close()
