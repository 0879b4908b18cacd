"""The allocation-free grid build where cells are crowded: the lists of crowded cells (ordered by warps, by blocks
and in parts), few cells with many particles, and the sizes where the ordering changes; and the reference
grid of a context on cells of h/2, which takes the same route. Bit for bit numpy's stable order."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
H = np.float32(0.0457)


def build(sphlib, torch, xyz, box):
    res = [int(np.ceil(np.float32(b) / H)) for b in box]
    n = xyz.shape[0]
    i32 = dict(dtype=torch.int32, device="cuda")
    out = [torch.empty(m, **i32) for m in (n, int(np.prod(res)) + 1, n)]
    ptr = [ctypes.c_void_p(t.data_ptr()) for t in out]
    a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
    a.record()
    rc = sphlib.load().sph_grid_build_noalloc(ctypes.c_void_p(xyz.data_ptr()), n, (ctypes.c_float * 3)(*box), float(H),
                                              *ptr, ctypes.c_void_p(torch.cuda.current_stream().cuda_stream or None))
    b.record()
    assert rc == sphlib.SPH_OK
    torch.cuda.synchronize()
    return res, [t.cpu().numpy() for t in out], a.elapsed_time(b)


def want_cells(pos, box, res):
    half = np.array([np.float32(b) / np.float32(2) for b in box], np.float64)
    q = np.clip(np.floor((pos.astype(np.float64) + half) / np.float64(H)).astype(np.int64), 0, np.array(res) - 1)
    return q[:, 0] + res[0] * (q[:, 1] + res[1] * q[:, 2])


def cell_box(res):
    return tuple(float(np.float32(r * float(H) * 0.999)) for r in res)


@pytest.mark.parametrize("n,res", [(3000, (1, 1, 1)), (65536, (1, 2, 1)), (65536, (9, 8, 7)), (65537, (1, 1, 1)),
                                   (65537, (5, 5, 5)), (66000, (12, 11, 9)), (200003, (4, 4, 4)), (200003, (13, 12, 10)),
                                   (524288, (40, 45, 50)), (524289, (40, 45, 50)), (524289, (43, 45, 45)),
                                   (524294, (41, 43, 50)), (1 << 20, (6, 6, 6)), (1 << 20, (23, 21, 22))])
def test_crowded_order(sphlib, n, res):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(n + res[0])
    box = cell_box(res)
    pos = (rng.random((n, 3)) - 0.5) * np.array(box)
    if res[0] >= 40:  # cells at the edges of the lists: by threads, by warps, by blocks, in parts
        a = 0
        for k, occ in enumerate((32, 33, 128, 129, 511, 512, 513, 1024, 1025, 5000)):
            mid = (np.array([3 * k + 2, 5, 7]) + 0.25 + 0.5 * rng.random((occ, 3))) * float(H) - np.array(box) / 2
            pos[a:a + occ] = mid
            a += occ
        pos = pos[rng.permutation(n)]
    pos = pos.astype(np.float32)
    xyz = torch.from_numpy(pos).cuda()
    for _ in range(2):
        got_res, (cell, start, order), _ = build(sphlib, torch, xyz, box)
    assert got_res == list(res)
    want = want_cells(pos, box, res)
    assert np.array_equal(cell, want)
    assert np.array_equal(order, np.argsort(want, kind="stable"))
    assert np.array_equal(start, np.concatenate([[0], np.cumsum(np.bincount(want, minlength=int(np.prod(res))))]))


@pytest.mark.parametrize("n,res,ms", [(70000, (1, 1, 1), 20.0), (200000, (12, 13, 13), 0.4), (200000, (4, 4, 4), 0.8),
                                      (1000000, (32, 31, 31), 0.8)])
def test_time_of_crowded_builds(sphlib, n, res, ms):
    """A few cells, or many cells of 33 to 100 particles: the work is spread over the whole GPU. (Limits: several times
    0.43, 0.04, 0.11 and 0.07 ms; on a grid sized by the cells, every block walking the whole list, these take
    480, 1.8, 2.2 and 4.8 ms.)"""
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(3)
    box = cell_box(res)
    xyz = torch.from_numpy(((rng.random((n, 3)) - 0.5) * np.array(box)).astype(np.float32)).cuda()
    best = min(build(sphlib, torch, xyz, box)[2] for _ in range(6))
    assert best < ms


@pytest.mark.parametrize("sizes", [(1501,), (70001, 3, 66003)])
def test_reference_grid_of_half_cells(sphlib, sizes):
    """sph_get_grid on cells of h/2: crowded cells, scenes of odd sizes."""
    rng = np.random.default_rng(7)
    box = (0.5, 0.4, 0.45)
    res = [int(np.ceil(np.float32(b) / H)) for b in box]
    pos = [((rng.random((n, 3)) - 0.5) * np.array(box)).astype(np.float32) for n in sizes]
    for p in pos:
        p[: len(p) // 3] *= np.float32(0.1)
    ctx = sphlib.SphContext([box] * len(sizes), sizes)
    ctx.set_cell_multiple(2)
    ctx.upload(np.concatenate(pos), None, sizes)
    ctx.pass_grid()
    cell, counts, order = ctx.grid()
    ctx.close()
    at, nc = 0, int(np.prod(res))
    for s, p in enumerate(pos):
        want = want_cells(p, box, res)
        assert np.array_equal(cell[at:at + len(p)], want)
        assert np.array_equal(counts[s * nc:(s + 1) * nc], np.bincount(want, minlength=nc))
        assert np.array_equal(order[at:at + len(p)], np.argsort(want, kind="stable"))
        at += len(p)


def test_ids_beyond_the_float_range(sphlib):
    """Ids from 2^24 on are compared as integers: neighbouring ones round to one float."""
    n = (1 << 24) + 700
    box = (1.4, 1.4, 1.4)
    res = [int(np.ceil(np.float32(b) / H)) for b in box]
    rng = np.random.default_rng(9)
    pos = ((rng.random((n, 3), np.float32) - np.float32(0.5)) * np.float32(1.39)).astype(np.float32)
    pos[-700:] = np.float32(0.001)
    ctx = sphlib.SphContext(box, n)
    ctx.set_cell_multiple(2)
    ctx.upload(pos)
    ctx.pass_grid()
    cell, counts, order = ctx.grid()
    ctx.close()
    want = want_cells(pos, box, res)
    assert np.array_equal(cell, want)
    assert np.array_equal(counts, np.bincount(want, minlength=int(np.prod(res))))
    assert np.array_equal(order, np.argsort(want, kind="stable"))
