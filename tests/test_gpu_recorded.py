"""Solves that amplify a change of rounding by 1e3 and more (RK4 near its stability limit or
on digit products, the split forms on coarse slices) against recorded curves of the dense
and digit stage products with the row-swapping elimination: another sequence of operations
moves them by the figure in CASES (2-norm of the difference over that of the curves), this
one repeats them.  The bound, 1e-9, is the agreement that results in double precision are
held to from one version to the next.  tests/golden/recorded.npz holds the curves."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import GOLDEN

pytestmark = pytest.mark.gpu

# name: (beams, seed, angles, dz, int_method, precision form, renormalisation policy); what the
# convolutions, the fused RK4 or the cluster elimination give instead
CASES = {
    "rk4-int8-17": (17, 6, 22, 0.127, 7, 2, 1),       # 1.0e-7
    "rk4-int8-76": (76, 5, 6, 0.075, 7, 2, 1),        # 3.3e-7
    "rk4-fp64-47": (47, 5, 9, 0.148, 7, 0, 1),        # 7.7e-8
    "rk4-fp64-91": (91, 5, 7, 0.116, 7, 0, 1),        # 4.1e-7
    "rk4-gs-int8-71": (71, 71, 8, 0.099, 8, 2, 1),    # 6.2e-8
    "sp4-int8-178": (178, 1, 5, 0.488, 5, 2, 1),      # 1.4e-9
    "sp4-int8-271": (271, 1, 4, 0.495, 5, 2, 0),      # 1.3e-9
    "sp6-int8-477": (477, 1, 2, 0.431, 6, 2, 1),      # 1.3e-8
}


def curves(ctx, d, name):
    from trhepd_opt_b200 import bulkfile, generator, native
    n, seed, angles, dz, method, precision, policy = CASES[name]
    s = generator.dense(n, seed=seed, n_angles=angles, region=12.0, dz=dz)
    s.int_method = method
    s.write(d)
    rng = np.random.default_rng(seed)
    bulkfile.write_bulkp(s, d / "bulkP.b", lambda t, g, m: 0.15 / np.sqrt(m) * (
        rng.standard_normal((m, m)) + 1j * rng.standard_normal((m, m))))
    ctx.set_option(native.OPT_RENORM_POLICY, policy)
    return ctx.surf_run(d / "bulkP.b", d / "surf.txt", dz, method, precision)[0]


@pytest.fixture(scope="module")
def ctx():
    from trhepd_opt_b200 import build, native
    build.build()
    c = native.Context(0)
    yield c
    c.close()


@pytest.mark.parametrize("name", sorted(CASES))
def test_recorded(ctx, tmp_path, name):
    ref = np.load(GOLDEN / "recorded.npz")[name]
    off = np.linalg.norm(curves(ctx, tmp_path, name) - ref) / np.linalg.norm(ref)
    print(f"{name}: {off:.2e}")
    assert off <= 1e-9
