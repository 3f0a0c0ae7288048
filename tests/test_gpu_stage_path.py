"""trhepd_last_stats says how the stages of the last solve ran, which the launches alone do
not tell (a fused solve, too, has fewer launches than stage products)."""
from __future__ import annotations

import pytest

from test_beam_grid import disc

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from trhepd_opt_b200 import build, native
    build.build()
    c = native.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("beams,precision,stages,length", [
    (disc(23), 0, "fused", 0), (disc(23), 2, "dense", 0), (disc(95), 0, "convolution", 12),
    (disc(95), 2, "convolution", 12), (disc(225), 2, "dense", 0),
    (disc(225), 0, "convolution", 20), (disc(401)[::2], 0, "dense", 0)])
def test_stages(ctx, tmp_path, beams, precision, stages, length):
    from trhepd_opt_b200 import bulkfile, generator, surface
    s = generator.dense(23, seed=1, n_angles=2, region=1.0, dz=0.05)
    s.beams = beams
    s.write(tmp_path)
    bulkfile.write_bulkp(s, tmp_path / "bulkP.b")
    sp = surface.SurfaceProblem(ctx, tmp_path / "bulkP.b", tmp_path / "surf.txt", 0.05, 5)
    rp = sp.resident()
    for _ in range(3):  # direct, captured, replayed
        rp.solve(precision)
        st = ctx.last_stats()
        assert (st["stages"], st["transform_length"]) == (stages, length)
    surface.solve_batch(ctx, [rp, sp.resident()], precision)
    st = ctx.last_stats()
    assert (st["stages"], st["transform_length"]) == ("batch", 0)
