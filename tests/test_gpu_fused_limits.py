"""The fused kernel's limit on table entries: beyond 48 beams one column of them (32 bytes
each) shares its buffer with the pivot rows from 880 entries on, and 2303 fit beside the
state.  Beam sets on both sides, alone and in a batch, against the oracle; what does not fit is
solved all the same.  FP64 on both sides in another summation order: 1e-10 of the row
maximum, 1e-8 relative on spots >= 1e-6 of it."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import spot_errors

pytestmark = pytest.mark.gpu
LIMIT = 2303


@pytest.fixture(scope="module")
def ctx():
    from trhepd_opt_b200 import build, native
    build.build()
    c = native.Context(0)
    yield c
    c.close()


def distinct(n, p=67):
    """n beams on a parabola mod p: every difference of two of them is another one."""
    b = [(i, i * i % p) for i in range(n)]
    h0, k0 = b[n // 2]
    b = [(h - h0, k - k0) for h, k in b]
    return [(0, 0)] + [x for x in b if x != (0, 0)]


def shared(n, extra):
    """`extra` beams of distinct(n) beside the first ones of a line: fewer differences."""
    b = distinct(n)[:extra]
    line = [(h, 0) for k in range(1, 4 * n) for h in (k, -k) if (h, 0) not in b]
    return b + line[:n - extra]


def problem(ctx, d, beams, seed, angles=3, dz=0.02, cell=8):
    from trhepd_opt_b200 import bulkfile, generator, surface
    s = generator.dense(23, seed=seed, n_angles=angles, region=1.0, dz=dz)
    s.beams = beams
    s.nh = s.nk = cell  # the beams reach 33 indices out
    s.write(d)
    rng = np.random.default_rng(seed)
    bulkfile.write_bulkp(s, d / "bulkP.b", lambda t, g, m: 0.1 / m * (
        rng.standard_normal((m, m)) + 1j * rng.standard_normal((m, m))))
    sp = surface.SurfaceProblem(ctx, d / "bulkP.b", d / "surf.txt", dz, 5)
    return sp, sp.resident()


def check(oracle_mod, d, got, dz=0.02):
    ref, _, _ = oracle_mod.Surface(d / "bulkP.b", d / "surf.txt", dz, 5).solve()
    abs_err, rel = spot_errors(got, ref)
    assert abs_err <= 1e-10, abs_err
    assert rel <= 1e-8, rel


@pytest.mark.parametrize("policy", [0, 1])
@pytest.mark.parametrize("beams", [distinct(64), distinct(59), shared(64, 56), distinct(49),
                                   shared(64, 16), shared(64, 17)],
                         ids=["64-distinct", "59-distinct", "64-mixed", "49", "64-873",
                              "64-910"])
def test_alone(ctx, tmp_path, oracle_mod, beams, policy):
    from trhepd_opt_b200 import native
    sp, rp = problem(ctx, tmp_path, beams, 3)
    ctx.set_option(native.OPT_RENORM_POLICY, policy)
    try:
        rp.solve(native.FP64)
    finally:
        ctx.set_option(native.OPT_RENORM_POLICY, 0)
    assert (ctx.last_stats()["launches"] < 40) == (sp.pot.nv <= LIMIT), sp.pot.nv
    check(oracle_mod, tmp_path, rp.fetch()[1])


def test_batch(ctx, tmp_path, oracle_mod):
    """Problems of few and many entries share a launch: the small ones' columns are shorter
    than the pivot rows that share their buffer."""
    from trhepd_opt_b200 import generator, native, surface
    sets = [generator.dense(23, seed=1).beams, distinct(64), shared(64, 30), distinct(59),
            distinct(48)]
    dirs = [tmp_path / f"b{k}" for k in range(len(sets))]
    probs = []
    for k, (d, beams) in enumerate(zip(dirs, sets)):
        d.mkdir()
        probs.append(problem(ctx, d, beams, 5 + k))
    surface.solve_batch(ctx, [rp for _, rp in probs], native.FP64)
    for d, (_, rp) in zip(dirs, probs):
        check(oracle_mod, d, rp.fetch()[1])
