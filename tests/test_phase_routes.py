"""Which phases of small graphs run in one launch (GPU): those whose longest row one block reads
in little time. The numbers of launches, on both sides of the lines, and the oracle's results."""
import numpy as np
import pytest

from oracle import vite_oracle as vo
from test_general_path import launches_of
from test_small_phase import multigraph

pytestmark = pytest.mark.gpu


def hub_graph(n, pairs, entries):
    """Random unit pairs, and vertex n - 1 joined to the others in turn, `entries` times."""
    rng = np.random.default_rng([n, pairs])
    a = np.concatenate([rng.integers(0, n - 1, pairs), np.full(entries, n - 1)])
    b = np.concatenate([rng.integers(0, n - 1, pairs), np.arange(entries) % (n - 1)])
    keep = a != b
    a, b = a[keep], b[keep]
    return vo._csr_from_list(n, np.concatenate([a, b]), np.concatenate([b, a]), np.ones(2 * len(a)))


@pytest.mark.parametrize("n,pairs,entries,one", [(2000, 5000, 49152, True), (2000, 5000, 49153, False),
                                                 (8193, 20000, 90000, False), (20000, 9000, 8192, True),
                                                 (20000, 9000, 8193, False), (8000, 9000, 20000, True)])
def test_longest_row(ctx, n, pairs, entries, one):
    g = hub_graph(n, pairs, entries)
    dev = ctx.upload(g.rowptr, g.tail, g.weight)
    ref = vo.louvain_phase(g)
    (cv, mod, it), launches = launches_of(ctx, lambda: ctx.louvain_phase(dev))
    assert (launches <= 10) == one
    np.testing.assert_array_equal(cv, ref[0])
    assert (it, float(mod).hex()) == (ref[2], float(ref[1]).hex())


@pytest.mark.parametrize("n", [20000, 140000])
@pytest.mark.parametrize("rebuilt", [False, True])
def test_known_row_is_not_launched_for(n, rebuilt):
    """A row of 8,193 communities, known from the upload or from the rebuild (in one launch or by
    several), costs one launch less than one of 8,192 whose launch gives up at its barriers."""
    import vite_b200

    count, iters = {}, {}
    with vite_b200.Context(0) as c:
        for entries in (8192, 8193):
            c.set_barrier_polls(1 << 23)
            g = hub_graph(n, n // 2, entries)
            dev = c.upload(g.rowptr, g.tail, g.weight)
            if rebuilt:  # every vertex alone: equal pairs become one
                c.rebuild(dev, np.arange(n))
            if entries == 8192:
                c.set_barrier_polls(1)
            (_, _, iters[entries]), count[entries] = launches_of(
                c, lambda: c.louvain_phase(dev, threshold=10.0))
            dev.free()
    assert iters[8192] == iters[8193] == 1  # no gain is enough to go on
    assert count[8193] == count[8192] - 1 and count[8193] > 10


def test_short_phase_has_no_iteration_in_vain(ctx):
    """Below 2^22 entries the loop test moves to the device, with an iteration ahead, only after
    some iterations: a phase of one takes the launches it takes above."""
    count = []
    for pairs in ((1 << 21) - 4000, (1 << 21) + 4000):
        g = multigraph(400000, pairs, 31, False)
        dev = ctx.upload(g.rowptr, g.tail, g.weight)
        (_, _, it), launches = launches_of(ctx, lambda: ctx.louvain_phase(dev, threshold=10.0))
        assert it == 1
        count.append(launches)
        dev.free()
    assert count[0] == count[1]
