"""The group forms of the neighbour passes (several lanes a particle, for small scenes) give the bits
of the forms with one thread a particle: at the particle counts where the launch rule changes form,
with ragged last warps, and where rows run past the recorded mask words and lists are worked off early.
The one-thread forms are variants 0 (pair terms in the candidate loop) and 4 (masks)."""
import numpy as np
import pytest

G981 = (0.0, -9.81, 0.0)


def scene(n, kind, seed=0):
    rng = np.random.default_rng(seed)
    if kind == "clump":  # ~100 particles a cell: rows of ~300 candidates, neighbours past a list's length
        a = 0.0457 * max(1.0, (n / 100) ** (1 / 3))
        box = (2.5 * a, 3.0 * a, 2.0 * a)
        pos = (rng.random((n, 3)) - 0.5) * a
    else:  # a jittered lattice in motion, some of it outside the walls
        m = int(np.ceil(n ** (1 / 3)))
        box = (0.5 * 0.0457 * (m + 2),) * 3
        k = np.arange(n)
        ijk = np.stack([k % m, (k // m) % m, k // (m * m)], 1)
        pos = (ijk + 0.6 * rng.random((n, 3))) * (0.5 * 0.0457) - box[0] / 2 - 0.004
    return box, pos.astype(np.float32), rng.normal(0, 0.4, (n, 3)).astype(np.float32)


def run(sphlib, box, pos, vel, variant, form=None, steps=3):
    ctx = sphlib.SphContext(box, pos.shape[0], gravity=G981, flags=sphlib.SPH_FLAG_RECORD_ACC,
                            precision=sphlib.SPH_PLAIN_F32 if form is None else form)
    if variant is not None:
        ctx.set_variant(0, variant)
    ctx.upload(pos, vel)
    ctx.step(steps)
    out = ctx.download(acc=True)
    ctx.close()
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("n,kind", [(1, "lattice"), (2, "clump"), (33, "lattice"), (1009, "clump"), (10239, "lattice"),
                                    (10240, "lattice"), (10241, "clump"), (32767, "lattice"), (32768, "clump"),
                                    (32769, "lattice")])
def test_plain_group_form_equals_one_thread_forms(sphlib, n, kind):
    box, pos, vel = scene(n, kind)
    got = run(sphlib, box, pos, vel, None)
    for variant in (0, 4):
        ref = run(sphlib, box, pos, vel, variant)
        for k in ref:
            assert np.array_equal(got[k], ref[k]), (n, kind, variant, k)


@pytest.mark.gpu
@pytest.mark.parametrize("n,kind", [(1, "lattice"), (35, "clump"), (1501, "clump"), (16383, "lattice"),
                                    (16384, "lattice"), (16385, "lattice")])
def test_f64_group_form_equals_one_thread_forms(sphlib, n, kind):
    """Also pairs close to r = h, where the float test passes them on to the exact one: the clump's
    many pairs, and a pair of particles moved to within a few float ulps of h."""
    box, pos, vel = scene(n, kind, 2)
    if n > 2:
        pos[1] = pos[0] + np.array([0.0457, 0, 0], np.float32)
        pos[2] = np.nextafter(pos[1], np.float32(-1), dtype=np.float32)
    got = run(sphlib, box, pos, vel, None, sphlib.SPH_F64)
    for variant in (0, 4):
        ref = run(sphlib, box, pos, vel, variant, sphlib.SPH_F64)
        for k in ref:
            assert np.array_equal(got[k], ref[k]), (n, kind, variant, k)


@pytest.mark.gpu
@pytest.mark.parametrize("n,kind", [(1, "lattice"), (35, "clump"), (1501, "clump"), (10240, "clump"),
                                    (10241, "lattice"), (32768, "lattice"), (32769, "clump")])
def test_mixed_group_form_equals_one_thread_form(sphlib, n, kind):
    """The mixed form's density sums are compensated word by word: the group form must keep each word's
    sum and their order. A context of two scenes that together exceed the group form's range runs the
    one-thread kernels on the same particles."""
    box, pos, vel = scene(n, kind, 7)
    got = run(sphlib, box, pos, vel, None, sphlib.SPH_MIXED)
    filler, fpos, fvel = scene(33000, "lattice", 8)
    ctx = sphlib.SphContext([box, filler], [n, 33000], gravity=G981, flags=sphlib.SPH_FLAG_RECORD_ACC,
                            precision=sphlib.SPH_MIXED)
    ctx.upload(np.concatenate([pos, fpos]), np.concatenate([vel, fvel]), [n, 33000])
    ctx.step(3)
    ref = ctx.download(acc=True)
    ctx.close()
    for k in got:
        assert np.array_equal(got[k], ref[k][:n]), (n, kind, k)


@pytest.mark.gpu
def test_f64_far_coordinates(sphlib):
    """Coordinates whose float rounding is larger than h, beyond the float range of squares, and
    infinite: the float test decides nothing there and the exact one gives the mask form's bits."""
    box, pos, vel = scene(300, "clump", 3)
    pos[:20] = np.float32(3.0e7) + np.arange(60, dtype=np.float32).reshape(20, 3)
    pos[20:24] = np.float32(2.5e30)
    pos[24, 1] = np.inf
    got = run(sphlib, box, pos, vel, None, sphlib.SPH_F64, steps=2)
    ref = run(sphlib, box, pos, vel, 4, sphlib.SPH_F64, steps=2)
    for k in ref:
        assert np.array_equal(got[k], ref[k], equal_nan=True), k


@pytest.mark.gpu
def test_variant_changed_between_the_passes(sphlib):
    """A density pass that wrote masks and no records (variants 4 to 6) is followed by a force pass of
    any mask-driven variant: the same bits."""
    box, pos, vel = scene(3001, "lattice", 4)
    ref = run(sphlib, box, pos, vel, 4, steps=1)
    for dense, forces in ((4, 3), (6, 3), (5, 10), (3, 4), (3, 7), (10, 3)):
        ctx = sphlib.SphContext(box, pos.shape[0], gravity=G981, flags=sphlib.SPH_FLAG_RECORD_ACC)
        ctx.upload(pos, vel)
        ctx.set_variant(0, dense)
        ctx.pass_grid()
        ctx.pass_density()
        ctx.set_variant(0, forces)
        ctx.pass_forces()
        got = ctx.download(acc=True)
        ctx.close()
        for k in ref:
            assert np.array_equal(got[k], ref[k]), (dense, forces, k)


@pytest.mark.gpu
def test_f64_variant_changed_between_the_passes(sphlib):
    """The FP64 density pass of variant 3 writes neither masks nor records."""
    box, pos, vel = scene(2003, "lattice", 5)
    ref = run(sphlib, box, pos, vel, 4, sphlib.SPH_F64, steps=1)
    for dense, forces in ((3, 4), (3, 10), (4, 3), (4, 9), (10, 3)):
        ctx = sphlib.SphContext(box, pos.shape[0], gravity=G981, flags=sphlib.SPH_FLAG_RECORD_ACC,
                                precision=sphlib.SPH_F64)
        ctx.upload(pos, vel)
        ctx.set_variant(0, dense)
        ctx.pass_grid()
        ctx.pass_density()
        ctx.set_variant(0, forces)
        ctx.pass_forces()
        got = ctx.download(acc=True)
        ctx.close()
        for k in ref:
            assert np.array_equal(got[k], ref[k]), (dense, forces, k)
