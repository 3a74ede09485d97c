"""Waits of the one-launch steps that run out (GPU): the blocks give up and return by
themselves, the launch per step takes over with the same results, and the context is as good as
before."""
import numpy as np
import pytest

from oracle import vite_oracle as vo
from test_general_path import launches_of
from test_gpu_parity import assert_graph_equal

pytestmark = pytest.mark.gpu


def test_wait_that_runs_out_is_made_up_for():
    import vite_b200

    g = vo.rgg(20000).unit()  # more than 2^14 entries: blocks on every SM
    ref = vo.louvain_phase(g)
    coarse = vo.rebuild(g, ref[0])
    colors, nc = vo.color(g, 2)
    ref_colors = vo.louvain_phase(g, ordering=1, et_type=2, et_delta=0.25, colors=colors,
                                  num_color=nc + 1)
    with vite_b200.Context(0) as c:
        with pytest.raises(vite_b200.VgError) as e:
            c.set_barrier_polls(0)
        assert e.value.status == vite_b200.VG_ERR_ARG
        for polls, one_launch in ((1, False), (1 << 23, True), (1, False)):
            c.set_barrier_polls(polls)
            dev = c.upload(g.rowptr, g.tail, g.weight)
            c.set_colors(dev, colors, nc)
            (cv, mod, it), n = launches_of(
                c, lambda: c.louvain_phase(dev, ordering=1, et_type=2, et_delta=0.25))
            assert (n <= 10) == one_launch
            np.testing.assert_array_equal(cv, ref_colors[0])
            assert (it, float(mod).hex()) == (ref_colors[2], float(ref_colors[1]).hex())
            (cv, mod, it), n = launches_of(c, lambda: c.louvain_phase(dev))
            assert (n <= 10) == one_launch
            np.testing.assert_array_equal(cv, ref[0])
            assert (it, float(mod).hex()) == (ref[2], float(ref[1]).hex())
            _, n = launches_of(c, lambda: c.rebuild(dev))
            assert (n <= 10) == one_launch
            assert_graph_equal(dev.download(), coarse)


@pytest.mark.parametrize("n", [900, 20000])  # a cluster, and blocks on every SM
def test_launch_of_a_phase_ends_after_its_iterations(n):
    """A phase that never gains too little to stop (a threshold of zero at a fixed point) must not
    be a launch that never ends. Here the limit is below and at a phase's iterations."""
    import vite_b200

    g = vo.rgg(n).unit()
    ref = vo.louvain_phase(g)
    assert ref[2] > 4
    with vite_b200.Context(0) as c:
        with pytest.raises(vite_b200.VgError) as e:
            c.set_phase_iterations(0)
        assert e.value.status == vite_b200.VG_ERR_ARG
        dev = c.upload(g.rowptr, g.tail, g.weight)
        for limit, one_launch in ((1, False), (ref[2] - 1, False), (ref[2], True), (1 << 14, True)):
            c.set_phase_iterations(limit)
            (cv, mod, it), launches = launches_of(c, lambda: c.louvain_phase(dev))
            assert (launches <= 10) == one_launch
            np.testing.assert_array_equal(cv, ref[0])
            assert (it, float(mod).hex()) == (ref[2], float(ref[1]).hex())
