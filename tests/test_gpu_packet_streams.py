"""The packets' gather and the gather per query beside it (an iteration of 80,000 camera queries and more): on a
caller's stream, in a captured graph, and in two contexts at once.  The values per query do not depend on
which of the two gathers runs when, so they are equal bit for bit."""
import numpy as np
import pytest

import golden_io as G
from smallupbp_b200 import engine
from smallupbp_b200 import workload as W


def results(st):
    pb2d, bb1d = st.segment_results()
    return dict(pb2d=pb2d, bb1d=bb1d, pp3d=st.point_results(), **st.query_stats()), st.image()


def same(got, want):
    for k in want[0]:
        np.testing.assert_array_equal(got[0][k], want[0][k], err_msg=k)
    assert G.image_rel_l2(got[1], want[1]) < 1e-6


@pytest.mark.gpu
@pytest.mark.parametrize("mode", [engine.MODE_PLAIN, engine.MODE_MIXED], ids=["plain", "mixed"])
def test_packets_on_a_callers_stream_in_a_graph_and_in_two_contexts(mode):
    import torch

    w = W.generate(W.cube_scene("a", 419, 317, 3000, 6, 0.01), 0)
    assert len(w["sq_flags"]) >= 100000
    with engine.EstimatorStage(0, mode) as st:
        st.run(w)
        want = results(st)
    streams = [torch.cuda.Stream() for _ in range(2)]
    stages = [engine.EstimatorStage(0, mode) for _ in streams]
    try:
        for st, s in zip(stages, streams):
            st.set_stream(s.cuda_stream)
            st.run(w)
        for st in stages:
            same(results(st), want)
        for st in stages:  # in turn, nothing waited for in between
            st.clear_image()
            st.evaluate()
        for st in stages:
            same(results(st), want)
        for st in stages:
            st.capture_graph()
        for _ in range(2):
            for st in stages:
                st.clear_image()
                st.launch_graph()
            for st in stages:
                same(results(st), want)
    finally:
        for st in stages:
            st.close()
