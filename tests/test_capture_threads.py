"""Giving a shape set back while another thread captures a stream leaves the capture whole."""
import threading

import numpy as np
import pytest

import curvami_gb300 as cg
from curvami_gb300 import synth

pytestmark = pytest.mark.gpu


def test_destroy_beside_capture():
    import torch

    import __graft_entry__ as ge

    ge.build()
    ctx = cg.Context(0)
    xy = synth.grid_nodes(21, 21, 0.5, 0.05, np.random.default_rng(1))
    ctx.set_nodes(xy)
    sets = [cg.shape_functions(ctx, xy[60:200] + 0.1, 1.6, 2, [])]
    a = torch.zeros(8, device="cuda")
    torch.cuda.synchronize()
    graph, stream = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.graph(graph, stream=stream, capture_error_mode="thread_local"):
        a.add_(1.0)
        t = threading.Thread(target=sets.clear)
        t.start()
        t.join()
        a.add_(1.0)
    graph.replay()
    torch.cuda.synchronize()
    assert bool((a == 2.0).all())
    assert cg.shape_functions(ctx, xy[60:200] + 0.1, 1.6, 2, []).nnz > 0
