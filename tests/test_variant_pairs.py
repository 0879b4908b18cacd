"""A force variant set between the density and the force pass: whatever the density pass of the variant before has
left (nothing, masks, masks and records), the force pass gives the bits of any variant."""
import itertools

import numpy as np
import pytest

from test_group_form import G981, run, scene


@pytest.mark.gpu
@pytest.mark.parametrize("form", ["SPH_PLAIN_F32", "SPH_F64"])
@pytest.mark.parametrize("n", [2003, 33001])
def test_every_pair(sphlib, form, n):
    if form == "SPH_F64" and n > 32768:
        n = 16387
    box, pos, vel = scene(n, "lattice", 6)
    ref = run(sphlib, box, pos, vel, 0, getattr(sphlib, form), steps=2)
    other = scene(n, "lattice", 7)[1]  # another state's masks and records lie in the buffers
    pairs = [((d, a), f) for d, a in ((0, 0), (2, 1), (4, 2)) for f in (3, 4, 6, 7, 9, 10, 11)]
    pairs += [((0, a), f) for a, f in itertools.product((3, 4, 6, 7, 11), (0, 2, 3, 4, 5, 7, 10))]
    ctx = sphlib.SphContext(box, n, gravity=G981, flags=sphlib.SPH_FLAG_RECORD_ACC, precision=getattr(sphlib, form))
    for dense, forces in pairs:
        ctx.set_variant(0, 10)
        ctx.upload(other, vel)
        ctx.step(1)
        ctx.upload(pos, vel)
        for _ in range(2):
            ctx.set_variant(*dense)
            ctx.pass_grid()
            ctx.pass_density()
            ctx.set_variant(0, forces)
            ctx.pass_forces()
        got = ctx.download(acc=True)
        for k in ref:
            assert np.array_equal(got[k], ref[k]), (dense, forces, k)
    ctx.close()
