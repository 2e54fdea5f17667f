"""View()'s captured graphs: one per scene, a bounded number of scenes, dropped
with their scene.  Frames are those of direct launches."""
import numpy as np
import pytest

from crystalgraphics_b200 import backend as B
from crystalgraphics_b200 import scenes

pytestmark = pytest.mark.gpu

# the same kernels on the same samples: only the order of a sample's float
# additions differs (a few dozen terms of one sign, 2^-24 of the sum each)
RTOL = 64 * 2.0 ** -24


def close(a, b):
    scale = np.maximum(np.abs(b), np.abs(b).mean())
    return float((np.abs(a.astype(np.float64) - b) / scale).max())


@pytest.mark.parametrize("count", [1, 2, 8, 9])
def test_scenes_in_turn(count):
    """More rounds than a graph takes to be captured and replayed, up to one
    scene more than the environment keeps graphs for."""
    B.EnvInit(B.PathTraceConf(render_width=40, render_height=24, sample_count=2, trace_depth=4))
    made = [scenes.cornell(40, 24) if k % 2 else scenes.textured_cornell(40, 24) for k in range(count)]
    loaded = [B.LoadScene(s) for s in made]
    cams = [B.Camera((0.02 * k, -3.4, 1.0), (0.0, 1.0, 0.0), (0.6, 0.4)) for k in range(count)]
    other = B.Camera((0.0, -3.3, 1.1), (0.0, 1.0, 0.0), (0.6, 0.4))

    def rounds(n):
        got = []
        for _ in range(n):
            for g, c in zip(loaded, cams):
                B.View(g, c)
                B.View(g, c)  # the second frame of the running mean
                got.append(B.ReadFilm())
                B.View(g, other)
        return got

    B.SetTuning(use_graph=0)
    ref = rounds(1)
    B.SetTuning(use_graph=1)
    for k, film in enumerate(rounds(3)):
        assert close(film, ref[k % count]) <= RTOL
    loaded[0].close()  # its graph goes with it; the others still replay
    if count > 1:
        B.View(loaded[1], cams[1])
        B.View(loaded[1], cams[1])
        assert close(B.ReadFilm(), ref[1]) <= RTOL
    for g in loaded:
        g.close()
    B.EnvTerm()


def test_statistics_start_at_zero_in_every_run():
    """Direct launches, a capture and replays report one run's rays each; a
    frame of one chunk after one of several does not count the other queue set."""
    s = scenes.cornell(64, 48)
    B.EnvInit(B.PathTraceConf(render_width=64, render_height=48, sample_count=4, trace_depth=3))
    g = B.LoadScene(s)
    cam = B.Camera.from_c(s.camera)
    B.SetTuning(queue_capacity=4096)  # several chunks on both pipelines
    many = []
    for _ in range(3):
        B.View(g, cam)
        st = B.LastStats()
        assert st.samples == 64 * 48 * 4 and st.chunks > 1
        many.append(st.extend_rays)
    B.SetTuning(queue_capacity=1 << 20)
    for k in range(3):
        B.ViewSamples(g, cam, 0, 4)  # frame 0's samples each time
        B.SetSeed(0)
        assert B.LastStats().chunks == 1
        assert B.LastStats().extend_rays == many[0]
    g.close()
    B.EnvTerm()


@pytest.mark.parametrize("capacity", [4096, 4097, 1 << 20])
def test_batch_films_read_in_slices(capacity):
    """A batch's films come back packed through the shadow queue: in one run, in
    several, and with a slice ending inside a view."""
    s = scenes.cornell(32, 32)
    B.EnvInit(B.PathTraceConf(render_width=8, render_height=8, trace_depth=3))
    g = B.LoadScene(s)
    sizes = [(64, 64), (1, 1), (91, 47), (33, 2), (64, 65)]
    views = [((0.0, -3.4, 1.0), (0.0, 1.0, 0.0), w, h, 2, 5 + k) for k, (w, h) in enumerate(sizes)]
    B.SetTuning(queue_capacity=capacity)
    for _ in range(2):  # captured, replayed
        films = B.batch_render(g, views)
        for k, (w, h) in enumerate(sizes):
            assert films[k].shape == (h, w, 3)
            alone = B.batch_render(g, views[k:k + 1])[0]
            assert close(films[k], alone) <= RTOL
    g.close()
    B.EnvTerm()
