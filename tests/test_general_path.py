"""Phases and rebuilds by a launch per step, which the one-launch paths of small graphs leave to
larger ones or to graphs with long rows (GPU), against the oracle: every degree class with several
vertices at its ends, several hubs above 8,192 communities (so that the phase is not taken in one
launch), early termination, colors, other tunings, both loops, segments of every table and of the
sorted path. Unit weights: communities, iterations and modularity bits equal; real weights: the
same communities, modularity within 1e-9 relative (the hubs' and the communities' sums meet
through atomics). Each test looks at the number of launches, so that it fails when its route is
taken over."""
import numpy as np
import pytest

from conftest import multi_hub_csr
from oracle import vite_oracle as vo
from test_gpu_parity import assert_graph_equal
from test_small_phase import multigraph

pytestmark = pytest.mark.gpu

REL_TOL = 1e-9
DEGREES = [15, 16, 17, 31, 32, 33, 127, 128, 129, 511, 512, 513, 1023, 1024, 1025, 4095, 4096, 4097]
OTHER = {"t32": 0, "ws_max": 48, "wt_max": 200, "ct_max": 1024, "tile_grid": 8}


def classes_graph(n, seed, real, hubs=(9000, 9001, 12000)):
    """Two vertices of each of DEGREES and one of each of `hubs`, joined to neighbours of a
    place of theirs on a ring of the other vertices, each joined to its next three, or (one in
    twenty) to any; a few self loops; names at random."""
    rng = np.random.default_rng([seed, n])
    spikes = [d for d in DEGREES for _ in range(2)] + list(hubs)
    k = len(spikes)
    ring = n - k
    a = np.repeat(np.arange(ring), 3)
    b = (a + np.tile([1, 2, 3], ring)) % ring
    far = rng.random(len(b)) < 0.05
    b[far] = rng.integers(0, ring, far.sum())
    a, b = [a[a != b]], [b[a != b]]
    for v, d in enumerate(spikes):
        a.append(np.full(d, ring + v))
        b.append((rng.integers(0, ring) + np.arange(d)) % ring)
    name = rng.permutation(n)
    a, b = name[np.concatenate(a)], name[np.concatenate(b)]
    s = name[rng.integers(0, ring, 40)]
    w = rng.random(len(a)) if real else np.ones(len(a))
    ws = rng.random(len(s)) if real else np.ones(len(s))
    g = vo._csr_from_list(n, np.concatenate([a, b, s]), np.concatenate([b, a, s]),
                          np.concatenate([w, w, ws]))
    length = np.diff(g.rowptr)
    assert all((length == d).sum() >= 2 for d in DEGREES) and all((length == d).any() for d in hubs)
    return g


def some_colors(n, seed):
    """Four colors and, one in ten, none: not a proper coloring, every class in each."""
    return np.random.default_rng([seed, n]).integers(-1, 9, n) // 2


def launches_of(ctx, call):
    ctx.profile(False, reset=True)
    out = call()
    return out, ctx.profile(False, reset=True)[1]


def check_phase(ctx, g, real, colors=None, num_colors=0, **kw):
    ref = vo.louvain_phase(g, colors=colors, num_color=num_colors + 1, **kw)
    for reorder in (False, True):
        dev = ctx.upload(g.rowptr, g.tail, g.weight)
        if reorder:
            ctx.reorder(dev, 1)
        if colors is not None:
            ctx.set_colors(dev, colors, num_colors)
        (cv, mod, it), launches = launches_of(ctx, lambda: ctx.louvain_phase(dev, **kw))
        assert launches > 10, "taken in one launch"
        assert it == ref[2]
        np.testing.assert_array_equal(cv, ref[0])
        if real:
            assert abs(mod - ref[1]) <= REL_TOL * abs(ref[1])
        else:
            assert float(mod).hex() == float(ref[1]).hex()
        dev.free()


@pytest.mark.parametrize("et", [0, 1, 2, 3, 4])
def test_phase_with_hubs(ctx, et):
    check_phase(ctx, classes_graph(30000, 1, False), False, et_type=et, et_delta=0.25)


@pytest.mark.parametrize("et", [0, 2])
def test_phase_with_hubs_real_weights(ctx, et):
    check_phase(ctx, classes_graph(30000, 2, True), True, et_type=et, et_delta=0.25)


@pytest.mark.parametrize("real", [False, True])
@pytest.mark.parametrize("ordering,et", [(0, 0), (0, 2), (1, 0), (1, 2)])
def test_phase_with_hubs_and_short_rows(ctx, ordering, et, real):
    """No rows of middle length: the hubs' kernels are launched before the others'."""
    g = vo.Graph(*multi_hub_csr(40000, 6, 9000, 21, real))
    colors = some_colors(g.nv, 7) if ordering else None
    check_phase(ctx, g, real, colors, 4, et_type=et, et_delta=0.25, ordering=ordering)


@pytest.mark.parametrize("ordering", [1, 2])
@pytest.mark.parametrize("et", [0, 1, 2, 3, 4])
@pytest.mark.parametrize("real", [False, True])
def test_phase_with_hubs_and_colors(ctx, real, et, ordering):
    g = classes_graph(30000, 3, real)
    check_phase(ctx, g, real, some_colors(g.nv, 4), 4, et_type=et, et_delta=0.25, ordering=ordering)


@pytest.mark.parametrize("tuning", [OTHER,
                                    {"t32": 1, "ws_max": 32, "wt_max": 32, "ct_max": 32},
                                    {"t32": 0, "ws_max": 128, "wt_max": 512, "ct_max": 4096},
                                    {"t32": 1, "ws_max": 32, "wt_max": 512, "ct_max": 512},
                                    {"t32": 0, "ws_max": 32, "wt_max": 32, "ct_max": 2048,
                                     "tile_grid": 1}])
@pytest.mark.parametrize("ordering", [0, 1])
def test_phase_with_other_tunings(tuning, ordering):
    import vite_b200

    g = classes_graph(30000, 4, False)
    colors = some_colors(g.nv, 5) if ordering else None
    with vite_b200.Context(0) as c:
        c.tuning = tuning
        check_phase(c, g, False, colors, 4, ordering=ordering, et_type=2 if ordering else 0,
                    et_delta=0.25)


def test_autotuned_phase():
    import vite_b200

    g = classes_graph(30000, 5, False)
    with vite_b200.Context(0) as c:
        c.autotune([c.upload(g.rowptr, g.tail, g.weight)], sweeps=1)
        check_phase(c, g, False)


def lattice(n, pairs, seed):
    """A ring of n vertices with `pairs` unit pairs in all: each vertex to some of its next 40,
    one pair in twenty to any vertex; names at random."""
    rng = np.random.default_rng([seed, n, pairs])
    a = rng.integers(0, n, pairs)
    b = (a + rng.integers(1, 41, pairs)) % n
    far = rng.random(pairs) < 0.05
    b[far] = rng.integers(0, n, far.sum())
    name = rng.permutation(n)
    a, b = name[a], name[b]
    a, b = a[a != b], b[a != b]
    return vo._csr_from_list(n, np.concatenate([a, b]), np.concatenate([b, a]), np.ones(2 * len(a)))


# plain: the loop test on the device up to 2^22 entries, on the host above; with early
# termination on the host
@pytest.mark.parametrize("pairs", [(1 << 20) + 4000, (1 << 21) - 4000, (1 << 21) + 4000])
@pytest.mark.parametrize("et", [0, 1, 2, 3, 4])
def test_phase_of_many_entries(ctx, pairs, et):
    check_phase(ctx, lattice(150000, pairs, 3), False, et_type=et, et_delta=0.25)


@pytest.mark.parametrize("flags", [["-c", "8", "-t", "2", "-a", "0.25"], ["-c", "8"], ["-d", "8"],
                                   ["-t", "4", "-a", "0.5"], ["-i", "-t", "3"], []])
def test_run_with_hubs(ctx, flags):
    g = classes_graph(30000, 6, False)
    kw = vo.flags_to_kwargs(flags)
    ref = vo.run(g, **kw)
    res = ctx.run(ctx.upload(g.rowptr, g.tail, g.weight), **kw)
    assert [s["nv"] for s in res.stats] == list(ref.level_nv)
    assert [s["iters"] for s in res.stats] == list(ref.level_iters)
    assert [float(s["modularity"]).hex() for s in res.stats] == [float(m).hex() for m in ref.level_mod]


def segments(others, seed):
    """A graph of 140,000 vertices (seven entries each on average) and communities of 30,000
    vertices (more entries than a block takes, runs of 128 to 40,000 entries of one key), 12,000
    (the large block table, or the sorted path when `others` is above its 4,096 keys), 4,000,
    1,000, 500, 200, 60, 20, 4 and `others` more."""
    rng = np.random.default_rng([seed, others])
    n = 140000
    sizes = [30000, 12000, 4000, 1000, 500, 200, 60, 20, 4]
    cv = np.concatenate([np.repeat(np.arange(len(sizes)), sizes),
                         len(sizes) + rng.integers(0, others, n - sum(sizes))])
    return n, rng.permutation(n)[cv][rng.permutation(n)]


@pytest.mark.parametrize("real", [False, True])
@pytest.mark.parametrize("others", [30, 900, 3900, 9000, 94000])
def test_rebuild_segments(ctx, others, real):
    n, cv = segments(others, 17)
    g = multigraph(n, 490000, 7, real, 50)
    ref = vo.rebuild(g, cv)
    for reorder in (False, True):
        dev = ctx.upload(g.rowptr, g.tail, g.weight)
        if not real:
            ctx.vertex_degree(dev)  # the weights are known to be integral from here on
        if reorder:
            ctx.reorder(dev, 1)
        _, launches = launches_of(ctx, lambda: ctx.rebuild(dev, cv))
        assert launches > 10, "taken in one launch"
        assert_graph_equal(dev.download(), ref)
        dev.free()
