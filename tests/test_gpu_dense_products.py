"""The stage products that remain beside the convolutions (digit slices on tcgen05, FP64
tiles), on beam sets without a grid worth transforming: every second beam of a disc, so
several ragged row and column tiles, several angles, one problem and a stacked batch,
against the oracle.  Each test checks from the launches that it is these kernels that ran.
Bars on spots >= 1e-6 of the row maximum: FP64 in another summation order 1e-8 relative;
the split forms their targets, 1e-6 (INT8) and 1e-5 (BF16)."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import spot_errors
from test_beam_grid import disc

pytestmark = pytest.mark.gpu

SPARSE = disc(401)[::2]  # 201 beams on a 23 x 23 grid: 38 % filled
REL = {0: 1e-8, 1: 1e-5, 2: 1e-6}
DZ = 0.02


@pytest.fixture(scope="module")
def ctx():
    from trhepd_opt_b200 import build, native
    build.build()
    c = native.Context(0)
    c.set_option(native.OPT_SPLIT_SLICES, 5)
    yield c
    c.close()


def problem(ctx, d, seed, angles=5, method=5):
    from trhepd_opt_b200 import bulkfile, generator, surface
    d.mkdir(exist_ok=True)
    s = generator.jitter(generator.dense(23, seed=1, n_angles=angles, region=2.0, dz=DZ), 0.1, seed)
    s.beams = SPARSE
    s.int_method = method
    s.write(d)
    rng = np.random.default_rng(seed)
    bulkfile.write_bulkp(s, d / "bulkP.b", lambda t, g, m: 0.1 / m * (
        rng.standard_normal((m, m)) + 1j * rng.standard_normal((m, m))))
    sp = surface.SurfaceProblem(ctx, d / "bulkP.b", d / "surf.txt", DZ, method)
    return sp, sp.resident()


def oracle_curves(oracle_mod, d, method=5):
    return oracle_mod.Surface(d / "bulkP.b", d / "surf.txt", DZ, method).solve()[0]


@pytest.mark.parametrize("method", [4, 5])
def test_alone(ctx, tmp_path, oracle_mod, method):
    sp, rp = problem(ctx, tmp_path, 2, method=method)
    ref = oracle_curves(oracle_mod, tmp_path, method)
    got = {}
    for precision, bar in REL.items():
        rp.solve(precision)
        st = ctx.last_stats()
        # a gather and at least one kernel per product (with the slicing, in the split forms)
        assert st["launches"] >= (3 if precision else 2) * st["stage_products"]
        got[precision] = rp.fetch()[1]
        _, rel = spot_errors(got[precision], ref)
        assert rel <= bar, (precision, rel)
    # three forms, three results: no form stood in for another
    assert not any(np.array_equal(got[a], got[b]) for a, b in ((0, 1), (0, 2), (1, 2)))


@pytest.mark.parametrize("precision", [0, 2], ids=["fp64", "int8"])
def test_stacked(ctx, tmp_path, oracle_mod, precision):
    from trhepd_opt_b200 import surface
    dirs = [tmp_path / f"s{k}" for k in range(3)]
    probs = [problem(ctx, d, 7 + k, angles=3) for k, d in enumerate(dirs)]
    surface.solve_batch(ctx, [rp for _, rp in probs], precision)
    st = ctx.last_stats()
    assert st["launches"] >= (3 if precision else 2) * st["stage_products"]
    for d, (_, rp) in zip(dirs, probs):
        _, rel = spot_errors(rp.fetch()[1], oracle_curves(oracle_mod, d))
        assert rel <= REL[precision], rel


def test_curve_errors(ctx, tmp_path):
    """The per-curve errors of a validated digit solve: those of the two results, none zero."""
    from trhepd_opt_b200 import native
    sp, rp = problem(ctx, tmp_path, 2)
    rp.solve(native.FP64)
    _, f64 = rp.fetch()
    ctx.set_option(native.OPT_VALIDATE, 1)
    try:
        rp.solve(native.SPLIT_INT8)
        err = ctx.last_curve_errors(rp.nangles)
    finally:
        ctx.set_option(native.OPT_VALIDATE, 0)
    _, f8 = rp.fetch()
    d, rowmax = np.abs(f8 - f64), np.abs(f64).max(axis=1)
    rel = np.where(f64 != 0, d / np.where(f64 != 0, np.abs(f64), 1.0), np.where(d > 0, np.inf, 0.0))
    assert (err[:, :2] > 0).all()
    np.testing.assert_allclose(err[:, 0], rel.max(axis=1), rtol=1e-12)
    np.testing.assert_allclose(err[:, 1], d.max(axis=1) / rowmax, rtol=1e-12)
    np.testing.assert_allclose(err[:, 2], rowmax, rtol=1e-15)
