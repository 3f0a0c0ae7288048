"""The beam grid behind the convolution stage products (csrc/beam_grid.h), on the CPU: the
header is compiled with g++ and its grid is checked pair by pair against the beam-pair map
it came from, for beam sets of every form the surface solve takes (discs in any order,
sheared, rectangular, holed, fractional-order rods, spans beyond the transforms) and maps
that are not a function of the beam difference."""
from __future__ import annotations

import subprocess
import textwrap

import numpy as np
import pytest

from conftest import ROOT

MAIN = textwrap.dedent("""
    #include "beam_grid.h"
    #include <cstdio>
    int main() {
      int n;
      if (std::scanf("%d", &n) != 1) return 2;
      std::vector<int> ih(n), ik(n), pair((size_t)n * n);
      for (int& v : ih) if (std::scanf("%d", &v) != 1) return 2;
      for (int& v : ik) if (std::scanf("%d", &v) != 1) return 2;
      for (int& v : pair) if (std::scanf("%d", &v) != 1) return 2;
      trhepd::ConvGrid g = trhepd::conv_grid(n, ih.data(), ik.data(), pair.data());
      std::printf("%d %d %d\\n", g.m, g.sx, g.sy);
      if (!g.m) return 0;
      for (const std::vector<int>* v : {&g.cell, &g.entry, &g.twins}) {
        for (int x : *v) std::printf("%d ", x);
        std::printf("\\n");
      }
      for (unsigned x : g.mask) std::printf("%u ", x);
      std::printf("\\n");
    }
""")


@pytest.fixture(scope="module")
def tool(tmp_path_factory):
    d = tmp_path_factory.mktemp("grid")
    (d / "main.cpp").write_text(MAIN)
    subprocess.run(["g++", "-std=c++17", "-O1", "-I", str(ROOT / "trhepd-opt_b200" / "csrc"),
                    str(d / "main.cpp"), "-o", str(d / "grid")], check=True)
    return d / "grid"


def pair_map(beams):
    """surfio's beam-difference index (surfsub.f90:9-41) as the solver's 0-based map."""
    n, index = len(beams), {(0, 0): 0}
    pair = np.zeros((n, n), dtype=int)
    for k in range(n):
        for l in range(k + 1, n):
            d = (beams[l][0] - beams[k][0], beams[l][1] - beams[k][1])
            pair[k, l] = pair[l, k] = index.setdefault(d, len(index))
    return pair


def disc(n, seed=None, shear=0, scale=(1, 1)):
    c = sorted((scale[0] * h * h + scale[1] * k * k, h, k) for h in range(-40, 41)
               for k in range(-40, 41))[:n]
    b = [(h, k + shear * h) for _, h, k in c]
    if seed is not None:
        np.random.default_rng(seed).shuffle(b)
    return [tuple(map(int, x)) for x in b]


def solve(tool, beams, pair):
    n = len(beams)
    text = "\n".join([str(n), " ".join(str(h) for h, _ in beams),
                      " ".join(str(k) for _, k in beams), " ".join(map(str, pair.ravel()))])
    out = subprocess.run([str(tool)], input=text, capture_output=True, text=True, check=True)
    lines = [list(map(int, x.split())) for x in out.stdout.strip().split("\n")]
    return lines


SETS = {"disc66": disc(66), "disc95-shuffled": disc(95, seed=1), "disc131-sheared": disc(131, 2, 2),
        "disc191-sheared-back": disc(191, 3, -1), "wide100": disc(100, 4, scale=(1, 2)),
        "holes300": [b for i, b in enumerate(disc(340, 5)) if i % 9], "disc521": disc(521, 6),
        "disc640": disc(640)}


@pytest.mark.parametrize("name", sorted(SETS))
def test_grid_reproduces_the_pair_map(tool, name):
    beams = SETS[name]
    pair = pair_map(beams)
    (m, sx, sy), cell, entry, twins, mask = solve(tool, beams, pair)
    assert m >= max(sx, sy) and m <= 32
    L, n = 2 * m, len(beams)
    x, y = np.array(cell) & 255, np.array(cell) >> 8
    assert (x < sx).all() and (y < sy).all() and len({*cell}) == n
    assert [sum(1 << v for v in x[y == r]) for r in range(sy)] == mask
    twin = {tuple(twins[i:i + 2]) for i in range(0, len(twins), 2)}
    entry = np.array(entry).reshape(L, L)
    for k in range(n):
        for j in range(n):
            e = entry[(y[j] - y[k]) % L, (x[j] - x[k]) % L]
            if k == j:
                assert e == 1
            elif k < j:   # -conj(u[pair])
                assert e == pair[k, j] + 1
            else:         # -w[pair], or its twin's -conj(u)
                assert e == -(pair[k, j] + 1) or (e - 1, pair[k, j]) in twin


def test_refused(tool):
    beams = disc(95)
    pair = pair_map(beams)
    bad = pair.copy()
    bad[3, 7] = bad[7, 3] = bad[0, 1]  # one pair with another difference's entry
    assert solve(tool, beams, bad)[0][0] == 0
    assert solve(tool, beams[:-1] + [beams[0]], pair)[0][0] == 0          # a beam twice
    assert solve(tool, beams[:-1] + [(40, 0)], pair)[0][0] == 0           # span beyond 32
    rods = [(m, -m) for m in range(-35, 36)]
    assert solve(tool, rods, pair_map(rods))[0][0] == 0                   # one line of beams
    assert solve(tool, disc(64), pair_map(disc(64)))[0][0] == 0           # the fused sizes
    sparse = disc(700)[::8]
    assert solve(tool, sparse, pair_map(sparse))[0][0] == 0               # an almost empty grid
