"""Stage products as convolutions over the beam grid, against the oracle: one beam count
per transform length, beams shuffled, sheared, on a rectangular grid and with holes, every
integrator that takes the path, both renormalisation schedules and several problems in one
stacked solve.  Both sides are FP64 in another summation order: 1e-10 of the row maximum,
1e-8 relative on spots >= 1e-6 of it."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import spot_errors
from test_beam_grid import SETS, disc

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from trhepd_opt_b200 import build, native
    build.build()
    c = native.Context(0)
    yield c
    c.close()


def write(d, beams, angles, dz, method=5, seed=1):
    from trhepd_opt_b200 import bulkfile, generator
    s = generator.dense(23, seed=seed, n_angles=angles, region=2.0, dz=dz)
    s.beams = beams
    s.int_method = method
    s.write(d)
    rng = np.random.default_rng(seed)
    bulkfile.write_bulkp(s, d / "bulkP.b", lambda t, g, m: 0.1 / m * (
        rng.standard_normal((m, m)) + 1j * rng.standard_normal((m, m))))
    return s


def check(got, ref):
    abs_err, rel = spot_errors(got, ref)
    assert abs_err <= 1e-10, abs_err
    assert rel <= 1e-8, rel


# one beam count per transform length (9, 10, 12, 15, 16, 20, 25, 27, 32)
@pytest.mark.parametrize("n,angles,dz", [(65, 3, 0.1), (78, 37, 0.1), (113, 2, 0.1), (150, 3, 0.15),
                                         (200, 2, 0.15), (290, 2, 0.2), (400, 1, 0.25),
                                         (521, 2, 0.25), (640, 1, 0.3)])
def test_every_length(ctx, tmp_path, oracle_mod, n, angles, dz):
    from trhepd_opt_b200 import native
    beams = disc(n, seed=n)
    if n == 78:
        beams = [b for b in disc(120, seed=n) if abs(b[0]) <= 4 and -5 <= b[1] <= 4]
    write(tmp_path, beams, angles, dz)
    f2, _ = ctx.surf_run(tmp_path / "bulkP.b", tmp_path / "surf.txt", dz, 5, native.FP64)
    ref, _, _ = oracle_mod.Surface(tmp_path / "bulkP.b", tmp_path / "surf.txt", dz, 5).solve()
    check(f2, ref)


@pytest.mark.parametrize("name", ["disc131-sheared", "disc191-sheared-back", "wide100", "holes300"])
def test_beam_sets(ctx, tmp_path, oracle_mod, name):
    from trhepd_opt_b200 import native
    write(tmp_path, SETS[name], 2, 0.15)
    # the split forms share the path on short transforms
    split = () if name == "holes300" else (native.SPLIT_INT8, native.SPLIT_BF16)
    for precision in (native.FP64, *split):
        f2, _ = ctx.surf_run(tmp_path / "bulkP.b", tmp_path / "surf.txt", 0.15, 5, precision)
        if precision == native.FP64:
            ref, _, _ = oracle_mod.Surface(tmp_path / "bulkP.b", tmp_path / "surf.txt", 0.15,
                                           5).solve()
        check(f2, ref)


@pytest.mark.parametrize("policy", [0, 1])
@pytest.mark.parametrize("method", [4, 6, 7, 8])
def test_integrators(ctx, tmp_path, oracle_mod, method, policy):
    from trhepd_opt_b200 import native
    write(tmp_path, disc(95, seed=8), 3, 0.04, method)
    ctx.set_option(native.OPT_RENORM_POLICY, policy)
    try:
        f2, _ = ctx.surf_run(tmp_path / "bulkP.b", tmp_path / "surf.txt", 0.04, method,
                             native.FP64)
    finally:
        ctx.set_option(native.OPT_RENORM_POLICY, 0)
    ref, _, _ = oracle_mod.Surface(tmp_path / "bulkP.b", tmp_path / "surf.txt", 0.04,
                                   method).solve()
    check(f2, ref)


def test_stacked_problems_and_spectra_stretches(ctx, tmp_path):
    """Stacked candidates equal their own solves, resident solves repeat bit for bit
    (direct, captured, replayed), and a table longer than one stretch of spectra (64 MB)
    gives what short groups of slices give."""
    from trhepd_opt_b200 import native, surface
    ctx.set_option(native.OPT_RENORM_POLICY, 1)
    try:
        probs = []
        for k in range(3):
            d = tmp_path / f"s{k}"
            s = write(d, disc(300, seed=8), 3, 0.03, seed=k)
            sp = surface.SurfaceProblem(ctx, d / "bulkP.b", d / "surf.txt", 0.03, 5)
            probs.append((sp, sp.resident()))
        alone = []
        for sp, rp in probs:
            out = []
            for _ in range(3):
                rp.solve(native.FP64)
                out.append(rp.fetch()[1])
            assert all(np.array_equal(o, out[0]) for o in out)
            alone.append(out[0])
        surface.solve_batch(ctx, [rp for _, rp in probs], native.FP64)
        for (sp, rp), ref in zip(probs, alone):
            assert spot_errors(rp.fetch()[1], ref)[0] <= 1e-12
    finally:
        ctx.set_option(native.OPT_RENORM_POLICY, 0)
    for (sp, rp), ref in zip(probs[:1], alone):
        rp.solve(native.FP64)  # a launch per slice
        assert spot_errors(rp.fetch()[1], ref)[0] <= 1e-10
