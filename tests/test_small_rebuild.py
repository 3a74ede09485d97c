"""The one-launch rebuild of small graphs (rebuild_small.cuh) against the oracle (GPU), bit
for bit: members per row around 32 (registers, bitmap), segments of entries around a chunk and
1,024 (warp and block tables), a giant community, more distinct keys than the tables take
(ranges of keys, and the general path), entries around the launch forms' limits, both layouts."""
import numpy as np
import pytest

from oracle import vite_oracle as vo
from test_gpu_parity import assert_graph_equal
from test_small_phase import multigraph

pytestmark = pytest.mark.gpu


def communities(n, kind, seed):
    """Labels in [0, n): blocks of a size, random ones, one giant among small ones, or all one."""
    rng = np.random.default_rng([seed, n])
    if kind == "one":
        return np.full(n, n // 2, np.int64)
    if kind == "single":
        return rng.permutation(n).astype(np.int64)
    if kind == "giant":
        c = rng.integers(0, n, n)
        c[rng.random(n) < 0.5] = 3 % n
        return c
    if kind == "wide":  # one community of a tenth of the vertices, the others single
        c = rng.permutation(n).astype(np.int64)
        c[rng.random(n) < 0.1] = c[0]
        return c
    if kind.startswith("random"):
        return rng.integers(0, min(n, int(kind[6:])), n) * (n // min(n, int(kind[6:])))
    return rng.permutation(n)[np.arange(n) // int(kind)].astype(np.int64)


CASES = [(1, 0, 2, "one"), (2, 5, 0, "single"), (97, 300, 3, "31"), (97, 300, 3, "32"),
         (990, 4000, 9, "33"), (990, 4000, 9, "random20"), (3000, 15000, 5, "single"),
         (5000, 40000, 0, "random40"), (5000, 40000, 20, "giant"), (20000, 60000, 0, "7"),
         (30000, 300000, 0, "random300"), (40000, 200000, 0, "one"), (9000, 400000, 0, "random4"),
         (16000, 8190, 1, "single"), (16000, 8194, 1, "5"), (30000, 400000, 0, "giant"),
         (30000, 300000, 0, "wide"), (60000, 60000, 0, "wide"), (131072, 140000, 0, "3"), (131073, 140000, 0, "3"), (20000, 1 << 20, 0, "random900"),
         (20000, (1 << 20) + 9000, 0, "random900")]


@pytest.mark.parametrize("real", [False, True])
@pytest.mark.parametrize("n,m,loops,kind", CASES)
def test_small_rebuild_matches_oracle(ctx, n, m, loops, kind, real):
    g = multigraph(n, m, 11, real, loops)
    cv = communities(n, kind, 13)
    ref = vo.rebuild(g, cv)
    for reorder in (False, True):
        dev = ctx.upload(g.rowptr, g.tail, g.weight)
        if not real:
            ctx.vertex_degree(dev)  # the weights are known to be integral from here on
        if reorder:
            ctx.reorder(dev, 1)
        ctx.rebuild(dev, cv)
        assert_graph_equal(dev.download(), ref)
