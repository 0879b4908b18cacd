"""The tuning cache: choices of older libraries (keys without a rules version) do not keep small scenes off the group
forms; where those are not the default, and on cells of h/2, they apply as before."""
import pytest


@pytest.mark.gpu
@pytest.mark.parametrize("form,n,line,rules,want", [
    ("SPH_PLAIN_F32", 8000, "0 9 1", "", (3, 1)), ("SPH_PLAIN_F32", 8000, "0 9 1", "|v2", (9, 1)),
    ("SPH_PLAIN_F32", 8000, "0 9", "", (3, 1)), ("SPH_PLAIN_F32", 8000, "0 10 2", "", (10, 2)),
    ("SPH_PLAIN_F32", 32768, "0 7 1", "", (3, 1)), ("SPH_PLAIN_F32", 32769, "0 7 1", "", (7, 1)),
    ("SPH_PLAIN_F32", 40000, "0 11 1", "|v2", (11, 1)), ("SPH_F64", 40000, "0 10 1", "", (3, 1)),
    ("SPH_F64", 40000, "0 10 1", "|v2", (10, 1)), ("SPH_MIXED", 8000, "0 2 1", "", (0, 1)),
    ("SPH_MIXED", 8000, "0 2 1", "|v2", (2, 1)), ("SPH_MIXED", 33000, "0 2 1", "", (2, 1))])
def test_choices_of_older_libraries(sphlib, tmp_path, monkeypatch, form, n, line, rules, want):
    monkeypatch.setenv("SPH_TUNE_CACHE", str(tmp_path / "tune.txt"))
    m = 35
    pos = sphlib.dam_break_scene((m, m, m), (1.0, 1.0, 1.0), 1)[:n]
    ctx = sphlib.SphContext((1.0, 1.0, 1.0), n, precision=getattr(sphlib, form))
    key = f"{ctx.device_name.replace(' ', '_')}|p{getattr(sphlib, form)}|b{n.bit_length() - 1}"
    (tmp_path / "tune.txt").write_text(f"{key}{rules} {line}\n")
    ctx.upload(pos)
    assert (ctx.variant()[1], ctx.cell_multiple()) == want
    ctx.close()
