"""The FP64 group form's first test in FP32 at smoothing lengths whose square is denormal in float, or zero: the bits of
the mask form, which tests in FP64 alone."""
import numpy as np
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("h", [0.0457, 1e-18, 4e-20, 1e-20, 1e-21, 1e-22, 1e-24])
def test_group_form_equals_mask_form(sphlib, h):
    rng = np.random.default_rng(5)
    n, a = 1500, 5.0 * h
    pos = (rng.random((n, 3)) - 0.5) * a
    d = rng.normal(size=(n // 2, 3))
    d /= np.linalg.norm(d, axis=1)[:, None]
    pos[n // 2:] = pos[:n // 2] + d * h * (1 + 1e-7 * rng.normal(size=(n // 2, 1)))  # pairs about h apart
    pos = pos.astype(np.float32)
    p = sphlib.default_params()
    p.h = h
    out = []
    for variant in (None, 4):
        ctx = sphlib.SphContext((8 * h,) * 3, n, precision=sphlib.SPH_F64, flags=sphlib.SPH_FLAG_RECORD_ACC, params=p)
        if variant is not None:
            ctx.set_variant(0, variant)
        ctx.upload(pos)
        ctx.pass_grid()
        ctx.pass_density()
        rho = ctx.download()["rho"]
        ctx.pass_forces()
        out.append({"rho": rho, "acc": ctx.download(acc=True)["acc"]})
        ctx.close()
    for k in out[0]:
        assert np.isfinite(out[1][k]).all()
        assert np.array_equal(out[0][k], out[1][k]), (h, k, int((out[0][k] != out[1][k]).sum()))
