"""The allocation-free grid build's two orderings (by particles up to 65,536, by cells beyond): bit for bit
numpy's stable order, for scattered particles, cells of 8, 9, 32, 33 and 4,096 particles and more."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
H = np.float32(0.0457)


@pytest.mark.parametrize("n,kind", [(65535, "scattered"), (65536, "crowded"), (65537, "scattered"), (65537, "crowded"),
                                    (200003, "crowded"), (1048576, "scattered"), (1048576, "one_cell")])
def test_order(sphlib, n, kind):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(n)
    box = (2.0, 1.5, 1.1)
    pos = (rng.random((n, 3)) - 0.5) * np.array(box) * 1.02
    if kind == "crowded":
        a = 0
        for k, occ in enumerate((8, 9, 31, 32, 33, 128, 129, 4095, 4096, 4097, 9000)):
            pos[a:a + occ] = (np.array([k + 2, 5, 7]) + 0.25 + 0.5 * rng.random((occ, 3))) * float(H) - np.array(box) / 2
            a += occ
        pos = pos[rng.permutation(n)]
    elif kind == "one_cell":
        pos[: n // 8] = 0.001
    xyz = torch.from_numpy(pos.astype(np.float32)).cuda()
    res = [int(np.ceil(np.float32(b) / H)) for b in box]
    i32 = dict(dtype=torch.int32, device="cuda")
    cell, start, order = (torch.empty(m, **i32) for m in (n, int(np.prod(res)) + 1, n))
    for _ in range(2):
        rc = sphlib.load().sph_grid_build_noalloc(
            ctypes.c_void_p(xyz.data_ptr()), n, (ctypes.c_float * 3)(*box), float(H), ctypes.c_void_p(cell.data_ptr()),
            ctypes.c_void_p(start.data_ptr()), ctypes.c_void_p(order.data_ptr()),
            ctypes.c_void_p(torch.cuda.current_stream().cuda_stream or None))
        assert rc == sphlib.SPH_OK
    torch.cuda.synchronize()
    half = np.array([np.float32(b) / np.float32(2) for b in box], np.float64)
    q = np.floor((xyz.cpu().numpy().astype(np.float64) + half) / np.float64(H)).astype(np.int64)
    q = np.clip(q, 0, np.array(res) - 1)
    want = q[:, 0] + res[0] * (q[:, 1] + res[1] * q[:, 2])
    assert np.array_equal(cell.cpu().numpy(), want)
    assert np.array_equal(order.cpu().numpy(), np.argsort(want, kind="stable"))
    assert np.array_equal(start.cpu().numpy(), np.concatenate([[0], np.cumsum(np.bincount(want, minlength=np.prod(res)))]))
