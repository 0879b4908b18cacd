"""A particle with a NaN coordinate has no neighbours, not even itself: its density is +0 in every variant, and
every density has the same bits in all of them on one cell size."""
import numpy as np
import pytest

from test_group_form import G981, scene


@pytest.mark.gpu
@pytest.mark.parametrize("form,n", [("SPH_PLAIN_F32", 1501), ("SPH_PLAIN_F32", 33001), ("SPH_F64", 1501), ("SPH_MIXED", 1501)])
def test_density_of_nan_particles_is_plus_zero(sphlib, form, n):
    box, pos, vel = scene(n, "lattice", 8)
    pos[7] = np.nan
    pos[700, 1] = np.nan
    ref = None
    variants = {"SPH_PLAIN_F32": [(1, 0), (1, None), (1, 4), (1, 7), (2, 7), (2, 10)],
                "SPH_F64": [(1, 0), (1, None), (1, 4), (1, 7)], "SPH_MIXED": [(1, 0), (1, 1), (2, 0)]}[form]
    for m, v in variants:
        ctx = sphlib.SphContext(box, n, precision=getattr(sphlib, form), gravity=G981)
        if m == 2:
            ctx.set_cell_multiple(2)
        if v is not None:
            ctx.set_variant(0, v)
        ctx.upload(pos, vel)
        ctx.pass_grid()
        ctx.pass_density()
        rho = ctx.download()["rho"]
        ctx.close()
        if form != "SPH_MIXED":
            assert np.array_equal(rho[[7, 700]], [0, 0]) and not np.signbit(rho[[7, 700]]).any(), (m, v)
        if m == 1:
            ref = rho if ref is None else ref
            assert rho.tobytes() == ref.tobytes(), (m, v)
