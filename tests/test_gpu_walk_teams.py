"""Idle lanes that help at the end of a launch (walkQueue, kTeam) on many
overlapping instances of deep meshes: helpers take entries of the TLAS and, from
below a return marker, entries of an instance's tree.  Frames are those of one
ray per thread."""
import numpy as np
import pytest

from crystalgraphics_b200 import backend as B
from crystalgraphics_b200 import scenes

pytestmark = pytest.mark.gpu

# the same hits, so only the order of a sample's float additions differs: a few
# dozen terms of one sign, 2^-24 of the sum each
RTOL = 64 * 2.0 ** -24


@pytest.fixture(scope="module")
def crowd():
    """96 instances, 0.5 to 3 in size, of eight meshes inside a cube of side 3."""
    s = scenes.instanced_scene(width=64, height=48, spp=1, depth=6, instances=96, lights=40, seed=9,
                               mesh_scale=1.0, extent=1.5, camera_distance=9.0)
    B.EnvInit(B.PathTraceConf(render_width=8, render_height=8))
    g = B.LoadScene(s)
    # a four-wide node takes the place of at most three binary ones
    assert g.info().blas_node_count >= 3 << 16
    yield s, g
    g.close()


def frame(g, camera, w, h, spp, depth, **tuning):
    B.EnvInit(B.PathTraceConf(render_width=w, render_height=h, sample_count=spp, trace_depth=depth))
    B.SetTuning(**tuning)
    B.View(g, camera)
    return B.ReadFilm()


@pytest.mark.parametrize("size", [(1, 1, 1), (17, 2, 1), (64, 48, 1), (320, 180, 2), (1024, 1023, 1),
                                  (1025, 1024, 1)])
@pytest.mark.parametrize("block", [32, 256])
def test_teams_on_overlapping_instances(crowd, size, block):
    s, g = crowd
    w, h, spp = size
    inside = B.Camera((0.3, -0.4, 0.2), (0.2, 0.9, -0.1), (0.8, 0.6))
    for camera in (B.Camera.from_c(s.camera), inside):
        ref = frame(g, camera, w, h, spp, 6, persistent=False)
        out = frame(g, camera, w, h, spp, 6, persistent=True, extend_block=block)
        scale = np.maximum(np.abs(ref), np.abs(ref).mean())  # zero: no sample met a light
        assert bool((np.abs(out.astype(np.float64) - ref) <= RTOL * scale).all())
