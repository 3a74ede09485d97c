"""The one-launch phase of small graphs (phase_small.cuh) against the oracle (GPU): sizes at
the edges of its row classes, sum chunks, launch forms and limits, all early-termination
types, both layouts. Unit weights: communities, iterations and modularity bits equal; real
weights: the same communities, modularity within 1e-9 relative (the community updates'
atomics reorder those sums, as in the reference's own)."""
import numpy as np
import pytest

from oracle import vite_oracle as vo

pytestmark = pytest.mark.gpu

REL_TOL = 1e-9


def multigraph(n, m, seed, real, loops=0, hub=0):
    """m random undirected pairs (repeats kept), `loops` self loops, and vertex n - 1 joined
    to `hub` vertices (each as often as it takes)."""
    rng = np.random.default_rng([seed, n, m])
    a, b = rng.integers(0, n, m), rng.integers(0, n, m)
    if hub:
        a = np.concatenate([a, np.full(hub, n - 1)])
        b = np.concatenate([b, np.arange(hub) % max(n - 1, 1)])
    keep = a != b
    a, b = a[keep], b[keep]
    s = rng.integers(0, n, loops)
    w = rng.random(len(a)) if real else np.ones(len(a))
    ws = rng.random(loops) if real else np.ones(loops)
    return vo._csr_from_list(n, np.concatenate([a, b, s]), np.concatenate([b, a, s]),
                             np.concatenate([w, w, ws]))


def check(ctx, g, real, **kw):
    ref = vo.louvain_phase(g, **kw)
    for reorder in (False, True):
        dev = ctx.upload(g.rowptr, g.tail, g.weight)
        if reorder:
            ctx.reorder(dev, 1)
        cv, mod, it = ctx.louvain_phase(dev, **kw)
        assert it == ref[2]
        np.testing.assert_array_equal(cv, ref[0])
        if real:
            assert abs(mod - ref[1]) <= REL_TOL * abs(ref[1])
        else:
            assert float(mod).hex() == float(ref[1]).hex()


# (vertices, pairs, self loops, hub entries): one vertex; rows of 31..33 entries (thread and
# warp rows), 511..513 (warp and block rows), thousands of entries on fewer and on
# more than 8,192 vertices (block table, general path); 2,048-vertex sum chunks +- 1; entries just
# below and above the cluster's 16,384 and the path's 2^21; a warp per row and a thread per row
SIZES = [(1, 0, 3, 0), (2, 8, 0, 0), (33, 500, 4, 0), (700, 900, 5, 31), (700, 900, 5, 32),
         (700, 900, 0, 33), (700, 300, 9, 511), (700, 300, 9, 513), (1500, 4000, 0, 9000),
         (2047, 4000, 3, 0), (2049, 8180, 0, 0), (2049, 8200, 7, 0), (5000, 9000, 0, 4090),
         (9000, 9000, 0, 8000), (8193, 9000, 0, 8190), (9500, 9000, 0, 9000), (9400, 30000, 0, 0), (40000, 90000, 20, 600), (65537, 100000, 0, 0),
         (30000, (1 << 20) - 2000, 0, 0), (30000, (1 << 20) + 2000, 0, 0)]


@pytest.mark.parametrize("real", [False, True])
@pytest.mark.parametrize("n,m,loops,hub", SIZES)
def test_small_phase_matches_oracle(ctx, n, m, loops, hub, real):
    check(ctx, multigraph(n, m, 3, real, loops, hub), real)


@pytest.mark.parametrize("et", [1, 2, 3, 4])
@pytest.mark.parametrize("n", [600, 20000])
def test_small_phase_early_termination(ctx, n, et):
    check(ctx, vo.rgg(n).unit(), False, et_type=et, et_delta=0.25)


def test_small_phase_negative_weights(ctx):
    """A negative degree turns the candidate pruning off inside the launch."""
    g = multigraph(2000, 9000, 7, False)
    w = g.weight.copy()
    w[(np.repeat(np.arange(g.nv), np.diff(g.rowptr)) + g.tail) % 3 == 0] = -2.0
    check(ctx, vo.Graph(g.rowptr, g.tail, w), False)


@pytest.mark.parametrize("ordering", [1, 2])
@pytest.mark.parametrize("et", [0, 2])
@pytest.mark.parametrize("n,m,hub", [(500, 2000, 0), (3000, 20000, 700), (30000, 100000, 0)])
def test_small_phase_colors(ctx, n, m, hub, et, ordering):
    """A sweep per color, with and without the community update between colors; some
    vertices stay uncolored."""
    g = multigraph(n, m, 9, False, 4, hub)
    colors, nc = vo.color(g, 2)
    kw = dict(et_type=et, et_delta=0.25, ordering=ordering)
    ref = vo.louvain_phase(g, colors=colors, num_color=nc + 1, **kw)
    for reorder in (False, True):
        dev = ctx.upload(g.rowptr, g.tail, g.weight)
        if reorder:
            ctx.reorder(dev, 1)
        assert ctx.color(dev, 2)[1] == nc
        cv, mod, it = ctx.louvain_phase(dev, **kw)
        assert it == ref[2] and float(mod).hex() == float(ref[1]).hex()
        np.testing.assert_array_equal(cv, ref[0])
