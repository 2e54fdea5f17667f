"""A batch's films in pinned, new and odd-aligned host memory."""
import numpy as np
import pytest
import torch

from crystalgraphics_b200 import backend as B
from crystalgraphics_b200 import scenes

pytestmark = pytest.mark.gpu

# the same samples: only the order of a sample's float additions differs (a few
# dozen terms of one sign, 2^-24 of the sum each)
RTOL = 64 * 2.0 ** -24


@pytest.mark.parametrize("graph", [0, 1])
def test_destinations(graph):
    s = scenes.cornell(32, 32)
    B.EnvInit(B.PathTraceConf(render_width=8, render_height=8, trace_depth=3))
    B.SetTuning(use_graph=graph)
    g = B.LoadScene(s)
    sizes = [(91, 47), (64, 65), (1, 1), (640, 360)]
    views = B.make_views([((0.0, -3.4, 1.0), (0.0, 1.0, 0.0), w, h, 2, 5 + k)
                          for k, (w, h) in enumerate(sizes)])
    n = 3 * sum(w * h for w, h in sizes)
    ref = np.concatenate([f.ravel() for f in B.batch_render(g, views)])
    assert ref.size == n and ref.mean() > 0
    pinned = torch.zeros(n + 2, dtype=torch.float32, pin_memory=True).numpy()
    for buf in (pinned[:n], pinned[1:n + 1], np.empty(n, np.float32), np.zeros(n + 1, np.float32)[1:]):
        guard = pinned[n + 1]
        B._check(B.lib.cg_batch_render(g.handle, views, len(sizes), buf.ctypes.data, None))
        scale = np.maximum(ref, ref.mean())
        assert float((np.abs(buf.astype(np.float64) - ref) / scale).max()) <= RTOL
        assert pinned[n + 1] == guard
    g.close()
    B.EnvTerm()
