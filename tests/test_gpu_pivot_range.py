"""Eliminations whose pivots' squares leave the range of a double: a bulk that reflects with
F = -I + 1e-170 C (C a cyclic shift, every beam in one group) makes the boundary transform's
Q 1e-170 and its P 1e170, and with it the first renormalisation's Q.  The curves are as
well determined as any: the oracle's at 1e-50 and 1e-200 agree to 1e-14.  FP64 in another
order on both sides: 1e-10 of the row maximum, 1e-8 relative on spots >= 1e-6 of it."""
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


# the fused kernel, clusters in one launch (stacked path), in blocks
@pytest.mark.parametrize("policy", [0, 1], ids=["gershgorin", "growth"])
@pytest.mark.parametrize("n,fused", [(9, 64), (40, 64), (60, 64), (23, 0), (95, 0), (150, 0)])
def test_pivot_range(ctx, tmp_path, oracle_mod, n, fused, policy):
    from trhepd_opt_b200 import bulkfile, generator, native
    s = generator.dense(n, seed=n, n_angles=2, region=2.0, dz=0.05)
    s.nh = s.nk = 1
    s.write(tmp_path)
    bulkfile.write_bulkp(s, tmp_path / "bulkP.b",
                         lambda t, g, m: -np.eye(m) + 1e-170 * np.roll(np.eye(m), 1, axis=0))
    ctx.set_option(native.OPT_RENORM_POLICY, policy)
    ctx.set_option(native.OPT_FUSED_MAX_N, fused)
    try:
        f2, _ = ctx.surf_run(tmp_path / "bulkP.b", tmp_path / "surf.txt", 0.05, 5, native.FP64)
    finally:
        ctx.set_option(native.OPT_RENORM_POLICY, 0)
        ctx.set_option(native.OPT_FUSED_MAX_N, 64)
    ref, _, _ = oracle_mod.Surface(tmp_path / "bulkP.b", tmp_path / "surf.txt", 0.05, 5).solve()
    abs_err, rel = spot_errors(f2, ref)
    assert abs_err <= 1e-10, abs_err
    assert rel <= 1e-8, rel
