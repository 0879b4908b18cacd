"""The checked library over the kernels that scenes beyond the group forms and beyond the one-launch grid pass take, on
both cell multiples, and over the allocation-free grid build's orderings: no check fails, and the bits are
those of the production library. (tests/test_checked_build.py has the small scenes.)"""
import json
import os
import re
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

CHILD = r"""
import ctypes, hashlib, json, sys
import numpy as np
sys.path.insert(0, sys.argv[1]); sys.path.insert(0, sys.argv[1] + "/gmu-water-simulation_gb300")
sys.path.insert(0, sys.argv[1] + "/tests")
import sphcuda, torch
from test_group_form import scene
checked = sys.argv[2] == "1"
G = (0.0, -9.81, 0.0)
out, flags = {}, {}

def note(name, ctx, arrays):
    out[name] = hashlib.sha256(b"".join(np.ascontiguousarray(a).tobytes() for a in arrays)).hexdigest()
    if checked:
        flags[name] = ctx.debug_check()

def steps(name, boxes, sizes, pos, vel, form, multiple, variant, emit=0, obstacles=None):
    caps = list(sizes)
    caps[0] += emit
    ctx = sphcuda.SphContext(boxes, caps, precision=form, gravity=G, flags=sphcuda.SPH_FLAG_RECORD_ACC, obstacles=obstacles)
    if multiple == 2:
        ctx.set_cell_multiple(2)
    if variant is not None:
        ctx.set_variant(0, variant)
    ctx.upload(pos, vel, sizes)
    ctx.step(2)
    if emit:
        ctx.emit_fountain(0, 5, 0, emit, (0.0, -0.2, 0.0), 0.03, 0.5, 0.05)
    ctx.pass_grid()
    cell, counts, order = ctx.grid()
    ctx.pass_density()
    ctx.pass_forces()
    d = ctx.download(acc=True)
    s = ctx.splat(0, 1, 64, 48)
    note(name, ctx, [d["pos"], d["vel"], d["rho"], d["p"], d["acc"], cell, counts, order, *s])
    ctx.close()

P, M, F = sphcuda.SPH_PLAIN_F32, sphcuda.SPH_MIXED, sphcuda.SPH_F64
for n, kind in ((20003, "lattice"), (33001, "clump"), (40003, "lattice")):
    box, pos, vel = scene(n, kind, 3)
    for form, multiples, variants in ((P, (1, 2), (None, 4, 5, 7, 10)), (M, (1, 2), (0, 1, 2, 3)), (F, (1,), (None, 4, 7))):
        for m in multiples:
            for v in variants:
                if m == 2 and form == P and v in (4, 5):
                    continue
                steps(f"{n} {kind} {form} m{m} v{v}", box, [n], pos, vel, form, m, v, emit=0 if m == 2 else 500)
box, pos, vel = scene(8192, "clump", 4)
for form in (P, M, F):
    steps(f"8192 {form}", box, [8192], pos, vel, form, 1, None)
sizes = [9001, 1, 30011, 4099]
parts = [scene(k, "lattice", 5) for k in sizes]
obstacles = [np.array([[-0.05, -0.1, -0.05, 0.05, 0.0, 0.05]], np.float32) if k > 1 else None for k in sizes]
for form, m in ((P, 1), (P, 2), (M, 1), (M, 2), (F, 1)):
    steps(f"batch {form} m{m}", [p[0] for p in parts], sizes, np.concatenate([p[1] for p in parts]),
          np.concatenate([p[2] for p in parts]), form, m, None, obstacles=obstacles)
box, pos, vel = scene(530003, "lattice", 6)
steps("530003", box, [530003], pos, vel, P, 1, None)
box, pos, vel = scene((1 << 21) + 1, "lattice", 6)
steps("2097153 m2", box, [pos.shape[0]], pos, vel, P, 2, None)

H = np.float32(0.0457)
rng = np.random.default_rng(5)
for n, res in ((65000, (30, 31, 33)), (70001, (30, 31, 33)), (70001, (4, 5, 3)), (66000, (1, 1, 1)), (530003, (60, 61, 62)),
               (530003, (20, 21, 22)), (1 << 20, (101, 101, 102))):
    box = tuple(float(np.float32(r * float(H) * 0.999)) for r in res)
    pos = (rng.random((n, 3)) - 0.5) * np.array(box)
    pos[: n // 50] *= 0.05
    xyz = torch.from_numpy(pos.astype(np.float32)).cuda()
    i32 = dict(dtype=torch.int32, device="cuda")
    got = [torch.empty(k, **i32) for k in (n, int(np.prod(res)) + 1, n)]
    rc = sphcuda.load().sph_grid_build_noalloc(ctypes.c_void_p(xyz.data_ptr()), n, (ctypes.c_float * 3)(*box), float(H),
                                               *[ctypes.c_void_p(t.data_ptr()) for t in got], None)
    torch.cuda.synchronize()
    assert rc == 0
    ctx = sphcuda.SphContext((0.4, 0.4, 0.4), 10)  # (its check collects the build's)
    note(f"noalloc {n} {res}", ctx, [t.cpu().numpy() for t in got])
    ctx.close()
print(json.dumps({"flags": flags, "out": out}))
"""


def child(lib, checked):
    env = dict(os.environ, SPH_LIBRARY=lib)
    r = subprocess.run([sys.executable, "-c", CHILD, ROOT, str(int(checked))], capture_output=True, text=True, env=env,
                       timeout=900)
    assert r.returncode == 0, r.stderr[-3000:]
    return json.loads(r.stdout.strip().splitlines()[-1])


@pytest.mark.gpu
def test_large_scenes_are_clean_and_identical(sphlib):
    pytest.importorskip("torch")
    checked = child(sphlib.LIB_CHECKED_PATH, True)
    plain = child(os.path.join(os.path.dirname(sphlib.LIB_CHECKED_PATH), "libsph_gb300.so"), False)
    assert not {k: v for k, v in checked["flags"].items() if v}
    assert checked["out"] == plain["out"]


def test_every_array_has_a_guard_region(sphlib):
    """The checked library's contexts need 256 bytes more for each array of the pool."""
    code = ("import sys, ctypes; sys.path.insert(0, sys.argv[1] + '/gmu-water-simulation_gb300'); import sphcuda as s\n"
            "p = s.default_params(); p.precision = s.SPH_MIXED; d = s.sph_scene_desc(); d.max_particles = 1000\n"
            "for a in range(3): d.box[a] = 1.0\n"
            "b = ctypes.c_uint64(); assert s.load().sph_memory_required(ctypes.byref(p), 1, ctypes.byref(d), ctypes.byref(b)) == 0\n"
            "print(b.value)")
    need = []
    for lib in (sphlib.LIB_CHECKED_PATH, os.path.join(os.path.dirname(sphlib.LIB_CHECKED_PATH), "libsph_gb300.so")):
        r = subprocess.run([sys.executable, "-c", code, ROOT], capture_output=True, text=True,
                           env=dict(os.environ, SPH_LIBRARY=lib))
        assert r.returncode == 0, r.stderr
        need.append(int(r.stdout))
    header = open(os.path.join(ROOT, "gmu-water-simulation_gb300", "csrc", "sph_internal.h")).read()
    body = re.sub(r"//[^\n]*", "", header[header.index("struct DevBufs {"):])
    body = body[:body.index("};")]
    arrays = set(re.findall(r"\*\s*(\w+)", body)) - {"big"}  # (big: the allocation-free build's own memory)
    assert (need[0] - need[1]) == 256 * len(arrays)
