"""Uploads from pinned host memory, read by a bounded number of blocks that loop over the particles, give
the bits of uploads from pageable memory, copied first and read by one thread a particle."""
import numpy as np
import pytest
import torch

from test_group_form import G981, scene

PER_PASS = 96 * 256  # particles that the bounded ingest takes at a time


def final(sphlib, box, sizes, upload, **kw):
    ctx = sphlib.SphContext([box] * len(sizes), list(sizes), gravity=G981, **kw)
    upload(ctx)
    ctx.step(1)
    out = ctx.download()
    ctx.close()
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("with_vel", [False, True])
@pytest.mark.parametrize("n", [1, 33, PER_PASS - 1, PER_PASS, PER_PASS + 1, 3 * PER_PASS + 77])
def test_pinned_upload_equals_pageable(sphlib, n, with_vel):
    box, pos, vel = scene(n, "clump", 21)
    sizes = np.array([n] if n < 40 else [n // 3, 5, n - n // 3 - 5], np.uint32)
    p, v = torch.from_numpy(pos).pin_memory(), torch.from_numpy(vel).pin_memory()
    for form in (sphlib.SPH_PLAIN_F32, sphlib.SPH_MIXED, sphlib.SPH_F64):
        ref = final(sphlib, box, sizes, lambda c: c.upload(pos, vel if with_vel else None, sizes), precision=form)
        got = final(sphlib, box, sizes,
                    lambda c: c.upload_raw(p.data_ptr(), v.data_ptr() if with_vel else None, sizes), precision=form)
        for k in ref:
            assert np.array_equal(got[k], ref[k]), (n, form, k)
