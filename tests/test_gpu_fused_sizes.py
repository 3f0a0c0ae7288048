"""The fused small-beam kernel at the sizes where its shape changes (row tiles of 16, four
beams per column group, 24 / 32 columns per warp pair, P in shared memory beyond 48) and on
beam sets without repeated differences (the most table entries per column: fewer columns
in flight), against the oracle, both renormalisation schedules.  FP64 on both sides in
another summation order: 1e-10 of the row maximum, 1e-8 relative on spots >= 1e-6 of it."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import spot_errors

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from trhepd_opt_b200 import build, native
    build.build()
    c = native.Context(0)
    yield c
    c.close()


def scattered(n):
    """n beams whose pairwise differences are (nearly) all different."""
    rng = np.random.default_rng(n)
    b = {(0, 0)}
    while len(b) < n:
        b.add(tuple(int(v) for v in rng.integers(-9, 10, 2)))
    return [(0, 0)] + sorted(b - {(0, 0)})


def compare(ctx, tmp_path, oracle_mod, n, kind, policy, method, dz, fused=True):
    from trhepd_opt_b200 import bulkfile, generator, native
    s = generator.dense(n, seed=n, n_angles=3, region=2.0, dz=dz)
    if kind == "scattered":
        s.beams = scattered(n)
    s.int_method = method
    s.write(tmp_path)
    rng = np.random.default_rng(n)
    bulkfile.write_bulkp(s, tmp_path / "bulkP.b", lambda t, g, m: 0.1 / m * (
        rng.standard_normal((m, m)) + 1j * rng.standard_normal((m, m))))
    ctx.set_option(native.OPT_RENORM_POLICY, policy)
    try:
        f2, _ = ctx.surf_run(tmp_path / "bulkP.b", tmp_path / "surf.txt", dz, method, native.FP64)
        assert (ctx.last_stats()["launches"] < 40) == fused
    finally:
        ctx.set_option(native.OPT_RENORM_POLICY, 0)
    ref, _, _ = oracle_mod.Surface(tmp_path / "bulkP.b", tmp_path / "surf.txt", dz, method).solve()
    abs_err, rel = spot_errors(f2, ref)
    assert abs_err <= 1e-10, abs_err
    assert rel <= 1e-8, rel


@pytest.mark.parametrize("policy", [0, 1], ids=["gershgorin", "growth"])
@pytest.mark.parametrize("n,kind,fused", [
    (2, "disc", True), (16, "disc", True), (17, "disc", True), (24, "disc", True),
    (25, "disc", True), (32, "disc", True), (33, "disc", True), (48, "disc", True),
    (49, "disc", False), (30, "scattered", True), (48, "scattered", False)])
def test_rk4_sizes(ctx, tmp_path, oracle_mod, n, kind, fused, policy):
    """int_method 7: fused up to 48 beams while two table columns fit beside its arrays."""
    compare(ctx, tmp_path, oracle_mod, n, kind, policy, 7, 0.03, fused)


@pytest.mark.parametrize("policy", [0, 1], ids=["gershgorin", "growth"])
@pytest.mark.parametrize("n,kind", [(2, "disc"), (5, "disc"), (16, "disc"), (17, "disc"),
                                    (24, "disc"), (25, "disc"), (33, "disc"), (48, "disc"),
                                    (49, "disc"), (63, "disc"), (30, "scattered"),
                                    (48, "scattered"), (64, "scattered")])
def test_sizes(ctx, tmp_path, oracle_mod, n, kind, policy):
    compare(ctx, tmp_path, oracle_mod, n, kind, policy, 5, 0.05)
