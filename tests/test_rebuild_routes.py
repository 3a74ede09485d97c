"""Which rebuilds of small graphs run in one launch (GPU): those whose longest segment one block
reads in little time. The numbers of launches, on both sides of the lines, and the oracle's bits."""
import numpy as np
import pytest

from oracle import vite_oracle as vo
from test_general_path import launches_of
from test_gpu_parity import assert_graph_equal
from test_small_phase import multigraph

pytestmark = pytest.mark.gpu


def one_long(n, members, others):
    """One community of `members` vertices and `others` (or single) ones, at random places."""
    rng = np.random.default_rng([n, members, others])
    cv = 1 + (np.arange(n) % others)
    cv[:members] = 0
    return rng.permutation(n)[cv][rng.permutation(n)]


# (vertices, pairs, members, others, real, one launch): entries of the long segment about
# 2 * pairs * members / vertices, its reads one up to 4,096 communities
@pytest.mark.parametrize("n,m,members,others,real,one", [
    (10000, 60000, 2500, 1000, True, True), (10000, 60000, 3000, 1000, True, False),
    (10000, 60000, 8000, 1000, True, False), (6000, 250000, 4800, 50, True, False),
    (10000, 200000, 3000, 1000, False, True), (10000, 200000, 3500, 1000, False, False),
    (12000, 48000, 1950, 9000, False, True), (12000, 48000, 2200, 9000, False, False),
    (20000, 60000, 4000, 15000, True, False)])
def test_long_segments(ctx, n, m, members, others, real, one):
    g = multigraph(n, m, 23, real)
    cv = one_long(n, members, others)
    dev = ctx.upload(g.rowptr, g.tail, g.weight)
    if not real:
        ctx.vertex_degree(dev)  # the weights are known to be integral from here on
    _, launches = launches_of(ctx, lambda: ctx.rebuild(dev, cv))
    assert (launches <= 10) == one
    assert_graph_equal(dev.download(), vo.rebuild(g, cv))


@pytest.mark.parametrize("members,sorted_path", [(7000, False), (15000, True)])
def test_long_segment_of_real_weights_is_sorted(ctx, members, sorted_path):
    """Above the one-launch size: 28,000 and 60,000 entries, integral ones in a block's table."""
    n = 140000
    cv = one_long(n, members, 2000)
    count = {}
    for real in (False, True):
        g = multigraph(n, 280000, 29, real)
        dev = ctx.upload(g.rowptr, g.tail, g.weight)
        if not real:
            ctx.vertex_degree(dev)
        _, count[real] = launches_of(ctx, lambda: ctx.rebuild(dev, cv))
        assert_graph_equal(dev.download(), vo.rebuild(g, cv))
        dev.free()
    assert (count[True] > count[False] + 10) == sorted_path


@pytest.mark.parametrize("n,m,one", [(3000, 40000, True), (140000, 300000, False)])
def test_negative_zeros_stay(ctx, n, m, one):
    """Integral weights that are -0.0: a sum of nothing else is -0.0, in a block's table too."""
    g = multigraph(n, m, 5, False)
    w = np.where(g.tail % 7 == 0, 2.0, np.where(g.tail % 3 == 0, 0.0, -0.0))
    g = vo.Graph(g.rowptr, g.tail, w)
    cv = one_long(n, n // 20, 1500)
    dev = ctx.upload(g.rowptr, g.tail, g.weight)
    ctx.vertex_degree(dev)
    _, launches = launches_of(ctx, lambda: ctx.rebuild(dev, cv))
    assert (launches <= 10) == one
    ref = vo.rebuild(g, cv)
    assert np.signbit(ref.weight).any() and np.diff(ref.rowptr).max() > 256
    assert_graph_equal(dev.download(), ref)


def test_integral_weights_are_known_after_a_phase(ctx):
    """A phase in one launch does not look whether the weights are integral; the rebuild by launches
    does, and keeps a segment of 60,000 integral entries out of the sorted path."""
    n = 10000
    cv = one_long(n, 5000, 1000)
    count = {}
    for real in (False, True):
        g = multigraph(n, 60000, 37, real)
        dev = ctx.upload(g.rowptr, g.tail, g.weight)
        _, launches = launches_of(ctx, lambda: ctx.louvain_phase(dev))
        assert launches <= 10
        _, count[real] = launches_of(ctx, lambda: ctx.rebuild(dev, cv))
        assert_graph_equal(dev.download(), vo.rebuild(g, cv))
        dev.free()
    assert 10 < count[False] < count[True] - 10
