"""Runs under a memory budget (GPU): where the paths that trade memory for time have no room
the leaner ones give the same results, and a budget too small for those is VG_ERR_OOM."""
import numpy as np
import pytest

from test_small_phase import multigraph

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("options", [{}, {"coloring": True}, {"vertex_order": True}])
def test_same_results_under_any_budget(options):
    import vite_b200
    g = multigraph(60_000, 240_000, 21, False, 10, 300)
    with vite_b200.Context(0) as c:
        dev = c.upload(g.rowptr, g.tail, g.weight)
        ref = c.run(dev, want_comm=True, **options)
    ran = 0
    for kib in range(9_000, 40_000, 1_500):
        with vite_b200.Context(0, mem_budget=kib << 10) as c:
            try:
                dev = c.upload(g.rowptr, g.tail, g.weight)
                got = c.run(dev, want_comm=True, **options)
            except vite_b200.VgError as e:
                assert e.status == vite_b200.VG_ERR_OOM
                assert ran == 0, "a larger budget failed where a smaller one was enough"
                continue
            ran += 1
            assert [s["iters"] for s in got.stats] == [s["iters"] for s in ref.stats]
            assert [s["modularity"] for s in got.stats] == [s["modularity"] for s in ref.stats]
            np.testing.assert_array_equal(got.comm, ref.comm)
    assert ran > 5
