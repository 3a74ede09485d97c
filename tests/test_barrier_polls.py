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
