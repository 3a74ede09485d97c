"""The coloring's kernels (hashes kept per vertex up to eight, computed per entry above)
against the oracle (GPU): every number of hashes around the two layouts, entries around
the kept ones' limit, rows longer than a warp's stage, self loops, isolated vertices,
several rounds, both layouts."""
import numpy as np
import pytest

from oracle import vite_oracle as vo
from test_small_phase import multigraph

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_hash", [1, 3, 4, 5, 8, 9])
@pytest.mark.parametrize("n,m,loops,hub", [(1, 0, 1, 0), (33, 40, 3, 0), (5000, 65520, 9, 0),
                                           (5000, 70000, 9, 900),
                                           (90000, 70000, 0, 0)])
def test_colors_match_oracle(ctx, n, m, loops, hub, n_hash):
    g = multigraph(n, m, 3, False, loops, hub)
    colors, nc = vo.color(g, n_hash, 95)
    for reorder in (False, True):
        dev = ctx.upload(g.rowptr, g.tail, g.weight)
        if reorder:
            ctx.reorder(dev, 1)
        got, got_nc = ctx.color(dev, n_hash, 95)
        assert got_nc == nc
        np.testing.assert_array_equal(got, colors)
