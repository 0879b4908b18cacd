"""Downloads into pageable, page-locked and device memory, alone and mixed in one call, of scenes small enough for the
one-copy route and beyond it. Device arrays are targets of plain device copies (in a child process: the host must not
touch them)."""
import ctypes
import os
import subprocess
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = r"""
import ctypes, itertools, sys
import numpy as np
sys.path.insert(0, sys.argv[1] + "/gmu-water-simulation_gb300")
import sphcuda, torch
L = sphcuda.load()
KEYS = ("pos", "vel", "rho", "p", "acc")
for form in (sphcuda.SPH_PLAIN_F32, sphcuda.SPH_MIXED, sphcuda.SPH_F64):
    for n in (1, 700, 60001):
        pos = ((np.random.default_rng(n).random((n, 3)) - 0.5) * 0.9).astype(np.float32)
        ctx = sphcuda.SphContext((1.0, 1.0, 1.0), n, precision=form, flags=sphcuda.SPH_FLAG_RECORD_ACC)
        ctx.upload(pos)
        ctx.step(1)
        want = ctx.download(acc=True)
        fn = L.sph_download_f64 if form == sphcuda.SPH_F64 else L.sph_download
        for places in (("d",) * 5, ("h",) * 5, ("p",) * 5, ("d", "p", "h", "d", "h"), ("p", "h", "p", None, None),
                       (None, None, "h", "d", None), (None, "p", None, None, "d")):
            out = {}
            for k, where in zip(KEYS, places):
                t = torch.zeros(want[k].shape, dtype=torch.from_numpy(want[k]).dtype)
                out[k] = None if where is None else t.cuda() if where == "d" else t.pin_memory() if where == "p" else t
            torch.cuda.synchronize()
            rc = fn(ctx.h, *[None if out[k] is None else ctypes.c_void_p(out[k].data_ptr()) for k in KEYS])
            assert rc == 0, (form, n, places, rc)
            for k in KEYS:
                if out[k] is not None:
                    assert np.array_equal(out[k].cpu().numpy(), want[k]), (form, n, places, k)
        ctx.close()
print("all targets")
"""


@pytest.mark.gpu
def test_download_into_any_memory(sphlib):
    pytest.importorskip("torch")
    r = subprocess.run([sys.executable, "-c", CHILD, ROOT], capture_output=True, text=True, timeout=600)
    assert r.returncode == 0 and "all targets" in r.stdout, (r.returncode, r.stderr[-2000:])


@pytest.mark.gpu
def test_time_into_page_locked_memory(sphlib):
    """Four arrays of 7,000 particles in FP64 come by copies of their own. (24 us, 45 through the buffer; the pageable
    download of the same arrays, 45 us, is the yardstick.)"""
    torch = pytest.importorskip("torch")
    import time
    n = 7000
    pos = ((np.random.default_rng(n).random((n, 3)) - 0.5) * 0.9).astype(np.float32)
    ctx = sphlib.SphContext((1.0, 1.0, 1.0), n, precision=sphlib.SPH_F64)
    ctx.upload(pos)
    ctx.step(1)
    took = {}
    for pin in (False, True):
        a = [torch.empty(s, dtype=torch.float64, pin_memory=pin) for s in ((n, 3), (n, 3), (n,), (n,))]
        args = [ctypes.c_void_p(t.data_ptr()) for t in a]
        times = []
        for _ in range(60):
            t0 = time.perf_counter()
            assert sphlib.load().sph_download_f64(ctx.h, *args, None) == 0
            times.append(time.perf_counter() - t0)
        took[pin] = np.median(times[10:])
    ctx.close()
    assert took[True] < 0.8 * took[False]
