"""bulk.exe on beam groups of every small size: the one-launch form (groups of up to 8
beams) at its edges (1, 2, 4 and 5 beams: one or two MMA steps; 8: the largest) and the
general form above it, electrons and a shifted unit layer among them, against the oracle.
Records agree within 1e-8 of their maximum plus 64 times the oracle's own sensitivity to a
2^-50 rescale of the potential (the bound of the ill-conditioned cases)."""
from __future__ import annotations

import numpy as np
import pytest

from test_gpu_bulk import records, sensitivity

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    from trhepd_opt_b200 import build, native
    build.build()
    c = native.Context(0)
    yield c
    c.close()


# beams (m, -m) of a 7 x 7 cell: groups of ceil(nb / 7)
@pytest.mark.parametrize("nb,angles", [(5, 1), (13, 3), (27, 2), (35, 9), (55, 2), (61, 2)])
def test_group_sizes(ctx, golden, oracle_mod, tmp_path, nb, angles):
    lines = (golden / "test23" / "bulk.txt").read_text().split("\n")
    out = []
    for line in lines:
        if line.rstrip().endswith(",NB"):
            line = f"{nb}\t\t\t\t\t\t,NB"
        elif "(IH(I),IK(I)" in line:
            b = [(0, 0)] + [(s * m, -s * m) for m in range(1, nb) for s in (1, -1)]
            line = ",".join(f"{h},{k}" for h, k in b[:nb]) + "\t,(IH(I),IK(I)"
        elif "BE,AZI" in line:
            f = line.split(",")
            f[4], f[5], f[6] = "0.5", f"{0.5 + 0.4 * (angles - 1):.2f}", "0.4\t\t\t"
            line = ",".join(f)
        out.append(line)
    bulk_txt = tmp_path / "bulk.txt"
    bulk_txt.write_text("\n".join(out))
    ours = tmp_path / "gpu.b"
    st = ctx.bulk_run(bulk_txt, ours)
    assert st["layers"] >= 20
    ref, pert = sensitivity(oracle_mod, bulk_txt, tmp_path)
    mine = records(ours)
    assert len(mine) == len(ref)
    compared = 0
    for x, y, z in zip(mine, ref, pert):
        if x == y:
            continue
        a, b, c = (np.frombuffer(v, np.complex128) for v in (x, y, z))
        assert np.isfinite(a).all()
        bound = 1e-8 * np.abs(b).max() + 64 * np.abs(c - b)
        assert (np.abs(a - b) <= bound).all(), (nb, float((np.abs(a - b) / bound).max()))
        compared += 1
    assert compared > 0
