"""Duplicate pairs by warps: groups that end inside and at a warp's step, and
more pairs than the first pass has room for, against the oracle."""
import numpy as np
import pytest

import gisspa_b200 as G
from gisspa_b200 import formats
from oracle import merge_oracle as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [(1, 2, 31, 32, 33, 34), (65, 1, 1, 96), (260,)])
def test_merge_groups_match_oracle(sizes):
    from gisspa_b200 import build
    build.build_library()
    r = np.random.default_rng(sum(sizes))
    lines = []
    for g, n in enumerate(sizes):
        for _ in range(n):
            # the last group is one cluster: nearly every pair of it is a duplicate
            near = g == len(sizes) - 1
            x, y = (100.0, 100.0) if near else r.integers(100, 160, 2)
            e = (40.0, 50.0, 60.0) if near else r.uniform(5, 60, 3)
            lines.append(formats.format_pick_line(g, "m%d.mrc" % g, 1.5, 0.0, 0.0, float(e[0]) + 0.1 * r.random(),
                                                  float(e[1]), float(e[2]), float(x) + r.integers(0, 3), float(y),
                                                  float(np.round(r.uniform(7, 12), 1))))
    want = M.merge_lines(lines, 20.0, 10.0)
    assert 0 < len(want) < len(lines)
    assert G.merge_lines(lines, 20.0, 10.0) == want
