"""Plain scenes beyond the group form: the default variant's density pass from quads of positions and
its record force kernels give the bits of the one-load density pass and the mask kernels (variant 4)
and of the first form (variant 0)."""
import numpy as np
import pytest

from test_group_form import G981, run, scene


@pytest.mark.gpu
@pytest.mark.parametrize("n,kind", [(32769, "lattice"), (40003, "clump"), (524287, "lattice"), (524288, "lattice"),
                                    (524290, "clump")])
def test_default_variant_equals_mask_variant(sphlib, n, kind):
    box, pos, vel = scene(n, kind, 11)
    got = run(sphlib, box, pos, vel, None, steps=2)
    for variant in (4,) if n > 100000 else (0, 4, 7, 10):
        ref = run(sphlib, box, pos, vel, variant, steps=2)
        for k in ref:
            assert np.array_equal(got[k], ref[k]), (n, kind, variant, k)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 1003])
def test_record_variants_on_small_ragged_scenes(sphlib, n):
    """Quads at the ends of the particles and rows of fewer candidates than a quad; a narrow box, whose
    rows follow one another in memory within h; a batch, whose scenes do."""
    for kind in ("lattice", "clump"):
        box, pos, vel = scene(n, kind, 12)
        box = (0.03, box[1], box[2])
        pos[:, 0] *= 0.1
        runs = []
        for variant in (0, 7, 10):
            ctx = sphlib.SphContext([box] * 3, [n, 2, n], gravity=G981, flags=sphlib.SPH_FLAG_RECORD_ACC)
            ctx.set_variant(0, variant)
            ctx.upload(np.concatenate([pos, pos[:1], pos[:1] + np.float32(0.001), pos]), None, [n, 2, n])
            ctx.step(3)
            runs.append(ctx.download(acc=True))
            ctx.close()
        for r in runs[1:]:
            for k in runs[0]:
                assert np.array_equal(runs[0][k], r[k]), (n, kind, k)


@pytest.mark.gpu
def test_exact_lattice(sphlib):
    """An unjittered lattice: pairs exactly h apart, at the edge of rows and of the neighbour test."""
    m = 34
    g = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3)
    s = np.float32(np.float32(0.0457) / np.float32(2))
    box = (float(m * s),) * 3
    pos = (g.astype(np.float32) * s - np.float32(box[0] / 2)).astype(np.float32)
    vel = np.zeros_like(pos)
    got = run(sphlib, box, pos, vel, None, steps=2)
    for variant in (0, 4):
        ref = run(sphlib, box, pos, vel, variant, steps=2)
        for k in ref:
            assert np.array_equal(got[k], ref[k]), (variant, k)


@pytest.mark.gpu
def test_download_between_the_passes(sphlib):
    """A download after the grid pass overwrites the staging memory that holds the quads: the density
    pass then takes the form that needs none."""
    box, pos, vel = scene(33001, "lattice", 13)
    out = []
    for look in (False, True):
        ctx = sphlib.SphContext(box, pos.shape[0], gravity=G981, flags=sphlib.SPH_FLAG_RECORD_ACC)
        ctx.upload(pos, vel)
        for _ in range(2):
            ctx.pass_grid()
            if look:
                ctx.download()
                ctx.grid()
            ctx.pass_density()
            if look:
                ctx.download()
            ctx.pass_forces()
        out.append(ctx.download(acc=True))
        ctx.close()
    for k in out[0]:
        assert np.array_equal(out[0][k], out[1][k]), k


@pytest.mark.gpu
def test_half_cells_density_of_large_scenes(sphlib):
    """Cells of h/2: a scene in a batch of 2^21 particles (density at 32 registers) has the bits that it has
    alone, one particle short of that."""
    n = (1 << 21) - 1
    box, pos, vel = scene(n, "lattice", 13)
    out = []
    for sizes in ([n], [n, 1]):
        ctx = sphlib.SphContext([box] * len(sizes), sizes, gravity=G981)
        ctx.set_cell_multiple(2)
        ctx.set_variant(0, 10)
        extra = sum(sizes) - n
        ctx.upload(np.concatenate([pos, pos[:extra]]), np.concatenate([vel, vel[:extra]]), sizes)
        ctx.step(1)
        out.append(ctx.download())
        ctx.close()
    for k in out[0]:
        assert np.array_equal(out[0][k], out[1][k][:n]), k
