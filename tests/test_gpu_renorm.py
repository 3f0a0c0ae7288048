"""The renormalisation (Gershgorin estimate and Gauss-Jordan elimination on clusters)
against the oracle, at the beam counts where its kernels change shape: one partial
sub-panel of 16 columns, the last size of the one-launch form (128) and the first
blocked one, the largest and smallest of each warp height, a last block of one column.
Slices are coarse, so every one is followed by an elimination.  Both sides are FP64 in
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
    c.set_option(native.OPT_FUSED_MAX_N, 0)  # small sizes through the stacked path too
    yield c
    c.close()


@pytest.mark.parametrize("n,angles,dz", [(13, 3, 0.1), (17, 40, 0.1), (96, 3, 0.1), (97, 5, 0.1),
                                         (128, 3, 0.1), (129, 50, 0.2), (193, 2, 0.2),
                                         (256, 2, 0.2), (257, 2, 0.2), (577, 2, 0.3)])
def test_renormalisation_matches_oracle(ctx, tmp_path, oracle_mod, n, angles, dz):
    from trhepd_opt_b200 import bulkfile, generator, native
    s = generator.dense(n, seed=40 + n, n_angles=angles, region=2.0, dz=dz)
    s.write(tmp_path)
    rng = np.random.default_rng(n)
    bulkfile.write_bulkp(s, tmp_path / "bulkP.b", lambda t, g, m: 0.1 / m * (
        rng.standard_normal((m, m)) + 1j * rng.standard_normal((m, m))))
    f2, _ = ctx.surf_run(tmp_path / "bulkP.b", tmp_path / "surf.txt", dz, 5, native.FP64)
    ref, _, _ = oracle_mod.Surface(tmp_path / "bulkP.b", tmp_path / "surf.txt", dz, 5).solve()
    abs_err, rel = spot_errors(f2, ref)
    print(f"N {n}: {abs_err:.2e} of the row maximum, {rel:.2e} relative")
    assert abs_err <= 1e-10, abs_err
    assert rel <= 1e-8, rel
