"""Every run reports its own rays: direct launches, captures and replays, runs on
one queue set after runs on several, and batches."""
import pytest

from crystalgraphics_b200 import backend as B
from crystalgraphics_b200 import scenes

pytestmark = pytest.mark.gpu

W, H, SPP = 64, 48, 16


@pytest.fixture
def room():
    s = scenes.cornell(W, H)
    start(s)
    g = B.LoadScene(s)
    yield s, g
    g.close()
    B.EnvTerm()


def start(s, **tuning):
    B.EnvInit(B.PathTraceConf(render_width=W, render_height=H, sample_count=SPP, trace_depth=3))
    B.SetTuning(queue_capacity=1 << 15, pipelines=2, **tuning)


def rays():
    st = B.LastStats()
    return st.samples, st.extend_rays, st.shadow_rays


def test_captured_and_replayed_frames_count_as_direct_ones(room):
    s, g = room
    cam = B.Camera.from_c(s.camera)

    def frames(use_graph):
        start(s, use_graph=use_graph)
        out = []
        for _ in range(4):  # a running mean: other samples in every frame
            B.View(g, cam)
            assert B.LastStats().chunks > 1
            out.append(rays())
        return out

    direct = frames(0)
    assert len(set(direct)) > 1 and min(min(r) for r in direct) > 0
    assert frames(1) == direct


def test_one_queue_set_after_two(room):
    s, g = room
    cam = B.Camera.from_c(s.camera)

    def share():
        B.ViewSamples(g, cam, 3, 1)
        assert B.LastStats().chunks == 1
        return rays()

    alone = share()
    for graph in (0, 1):
        start(s, use_graph=graph)
        for _ in range(3):
            B.View(g, cam)
            assert B.LastStats().chunks > 1  # both queue sets
            assert share() == alone


def test_batches_count_their_own_rays(room):
    s, g = room
    views = [((0.0, -3.4, 1.0), (0.0, 1.0, 0.0), w, h, 4, 5 + k)
             for k, (w, h) in enumerate([(64, 64), (91, 47), (33, 2)])]

    def batch():
        B.batch_render(g, views)
        return rays()

    start(s, use_graph=0)
    alone = batch()
    assert min(alone) > 0
    start(s, use_graph=1)
    for _ in range(3):  # captured, replayed
        assert batch() == alone
        B.View(g, B.Camera.from_c(s.camera))
