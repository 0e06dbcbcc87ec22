"""Operators captured into a CUDA graph on the context's stream: the replays
read the links the lattice holds when they run, also after the library has
freed or replaced the copies it makes for speed.

Tolerance: the operators' 1e-13."""
import numpy as np
import pytest

from oracle import rel_l2

pytestmark = pytest.mark.gpu
DIMS = (4, 4, 4, 8)
MASS = 0.1


def test_captured_operator_outlives_the_fixed_point_links(wd, oracle):
    import torch

    gauges = [wd.gen_gauge(DIMS, seed=71), wd.gen_gauge(DIMS, seed=72)]
    gauges.append([np.ascontiguousarray(3.0 * g) for g in gauges[1]])  # links the copy cannot hold
    src = wd.gen_source(DIMS, seed=71)
    with wd.Context(0) as ctx:
        lat = ctx.lattice(DIMS, gauges[2])
        b, x, y = lat.field(src), lat.field(), lat.field()

        def calls():
            lat.dslash_full(b, x, MASS, 0)
            lat.dslash_offd(x, y, 1, 0)

        calls()  # loads the FP64-pipe kernels
        lat.update(gauges[0])
        calls()
        stream = torch.cuda.ExternalStream(ctx.stream)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
            calls()

        def replayed():
            x.zero()
            y.zero()
            with torch.cuda.stream(stream):
                graph.replay()
            return y.download()

        def want(g):
            return oracle.dslash_offd(oracle.dslash_full(src, g, DIMS, MASS, 0), g, DIMS, 1, 0)

        assert rel_l2(replayed(), want(gauges[0])) < 1e-13
        ctx.exhaust_memory_after(0)
        extra = lat.field()  # takes the fixed-point links back
        assert rel_l2(replayed(), want(gauges[0])) < 1e-13
        for g in (gauges[1], gauges[2], gauges[0]):
            lat.update(g)
            assert rel_l2(replayed(), want(g)) < 1e-13
        del graph
        for o in (extra, b, x, y, lat):
            o.close()
