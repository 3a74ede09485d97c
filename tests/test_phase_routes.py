"""Which phases of small graphs run in one launch (GPU): those whose longest row one block reads
in little time. The numbers of launches, on both sides of the lines, and the oracle's results."""
import numpy as np
import pytest

from oracle import vite_oracle as vo
from test_general_path import launches_of

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
