"""The graph of whole steps outlives an upload: runs after further uploads (the same count, another
count, after a change of variant, cell multiple or gravity) equal runs of a fresh context."""
import numpy as np
import pytest

from test_group_form import G981, scene


@pytest.mark.gpu
@pytest.mark.parametrize("prec", ["plain", "mixed", "f64"])
def test_steps_after_another_upload(sphlib, prec):
    form = {"plain": sphlib.SPH_PLAIN_F32, "mixed": sphlib.SPH_MIXED, "f64": sphlib.SPH_F64}[prec]
    box, pos, vel = scene(2003, "lattice", 21)
    other = scene(2003, "lattice", 22)
    changes = [lambda c: None, lambda c: c.set_gravity((1.0, -3.0, 0.5)),
               lambda c: c.set_variant(0, 1 if prec == "mixed" else 4)]
    if prec != "f64":
        changes.append(lambda c: c.set_cell_multiple(2))
    kept = sphlib.SphContext(box, 2003, precision=form, gravity=G981)
    kept.upload(pos, vel)
    kept.step(16)
    n = [2003, 2003, 1501, 2003]
    for k, change in enumerate(changes):
        fresh = sphlib.SphContext(box, 2003, precision=form, gravity=G981)
        for c in (kept, fresh):
            for ch in changes[:k + 1] if c is fresh else [change]:
                ch(c)
            c.upload(other[1][:n[k]], other[2][:n[k]])
            c.step(19)
        a, b = kept.download(), fresh.download()
        fresh.close()
        for key in a:
            assert np.array_equal(a[key], b[key]), (k, key)
    kept.close()
