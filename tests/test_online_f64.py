"""Online tuning of the FP64 form tries no variant but the group form: the mask forms never win there, and a trial step
of theirs takes several times as long. A variant set by the caller before is left at the first trial."""
import numpy as np
import pytest

from test_group_form import G981, scene


@pytest.mark.gpu
def test_f64_online_tuning_stays_on_the_group_form(sphlib):
    box, pos, vel = scene(1501, "lattice", 3)
    out = []
    for online in (False, True):
        ctx = sphlib.SphContext(box, pos.shape[0], gravity=G981, precision=sphlib.SPH_F64)
        if online:
            ctx.set_variant(0, 10)
            ctx.set_online_tuning(4)
        ctx.upload(pos, vel)
        for k in range(14):
            ctx.step(1)
            assert ctx.variant()[1] == 3, k
        ctx.step(26)
        out.append(ctx.download())
        ctx.close()
    for k in out[0]:
        assert np.array_equal(out[0][k], out[1][k]), k
