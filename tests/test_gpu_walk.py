"""The closest-hit and shadow walk over four-wide trees (walkQueue): frames whose
ray counts sit at the edges of a warp, a block and the resident grid, on a mesh
and on heavily overlapping instances (stacks deeper than their shared-memory
part), against one ray per thread, and its hits against the oracle's."""
import numpy as np
import pytest

import oracle as O
from crystalgraphics_b200 import backend as B
from crystalgraphics_b200 import scenes
from gpu_common import keyed_compare, primary_tie_mask

pytestmark = pytest.mark.gpu

# The walks return the same hits, so the frames differ by the order of a
# sample's float additions alone: at most a few dozen terms of one sign, each
# addition rounding by 2^-24 of the sum.
RTOL = 64 * 2.0 ** -24


def overlapping():
    return scenes.instanced_scene(width=64, height=48, spp=1, depth=4, instances=96, lights=40, seed=9,
                                  mesh_scale=0.05, extent=1.5, camera_distance=9.0)


SCENES = {"mesh": lambda: scenes.icosphere_scene(subdiv=4), "overlap": overlapping}


@pytest.fixture(scope="module", params=sorted(SCENES))
def loaded(request):
    s = SCENES[request.param]()
    B.EnvInit(B.PathTraceConf(render_width=8, render_height=8))
    g = B.LoadScene(s)
    yield s, g
    g.close()


def frame(g, camera, w, h, spp, depth, **tuning):
    B.EnvInit(B.PathTraceConf(render_width=w, render_height=h, sample_count=spp, trace_depth=depth))
    B.SetTuning(**tuning)
    B.View(g, camera)
    return B.ReadFilm()


@pytest.mark.parametrize("size", [(1, 1, 1), (31, 1, 1), (33, 1, 1), (127, 3, 1), (257, 16, 5),
                                  (613, 251, 1)])
@pytest.mark.parametrize("bits", [32, 8])
def test_walk_matches_one_ray_per_thread(loaded, size, bits):
    s, g = loaded
    cam = B.Camera.from_c(s.camera)
    w, h, spp = size
    ref = frame(g, cam, w, h, spp, 6, persistent=False, box_bits=32)
    for block in (32, 128, 256):
        out = frame(g, cam, w, h, spp, 6, persistent=True, box_bits=bits, extend_block=block)
        scale = np.maximum(np.abs(ref), np.abs(ref).mean())
        assert float((np.abs(out.astype(np.float64) - ref) / scale).max()) <= RTOL


def test_walk_matches_the_oracle(loaded):
    s, g = loaded
    w, h = 67, 45
    conf = B.PathTraceConf(render_width=w, render_height=h, sample_count=2, trace_depth=4)
    out = frame(g, B.Camera.from_c(s.camera), w, h, 2, 4, persistent=True)
    o = O.OracleScene(s)
    ref, _, _ = o.render(conf.to_c(), s.camera, rng=O.RNG_KEYED, prune=True)
    keep = ~primary_tie_mask(o, s.camera, w, h)
    close, rel_mean, _ = keyed_compare(out, ref, keep)
    assert close >= 0.995  # the criterion of the other keyed frames


# ---- teams: the end of a small launch on deep trees ----------------------------------
@pytest.fixture(scope="module", params=["mesh", "coincident"])
def deep(request):
    """A mesh of 327,680 triangles (launches of up to 2^20 samples let idle lanes
    help), once with a second instance of another material in the same place,
    so that two triangles are at every hit's distance."""
    s = scenes.icosphere_scene(subdiv=7)
    if request.param == "coincident":
        twin = s.instances[:1].copy()
        twin["material"] = 1
        s.instances = np.ascontiguousarray(np.concatenate([s.instances, twin]))
    B.EnvInit(B.PathTraceConf(render_width=8, render_height=8))
    g = B.LoadScene(s)
    yield s, g
    g.close()


@pytest.mark.parametrize("size", [(1, 1, 1), (17, 2, 1), (33, 1, 3), (127, 3, 1), (320, 180, 2),
                                  (1024, 1023, 1), (1024, 1024, 1), (1025, 1024, 1)])
def test_teams_match_one_ray_per_thread(deep, size):
    s, g = deep
    w, h, spp = size
    for k, camera in enumerate((B.Camera.from_c(s.camera),
                                B.Camera((0.0, -1.35, 0.9), (0.0, 0.83, -0.55), (0.8, 0.45)))):
        ref = frame(g, camera, w, h, spp, 8, persistent=False)
        out = frame(g, camera, w, h, spp, 8, persistent=True)
        scale = np.maximum(np.abs(ref), np.abs(ref).mean())
        assert float((np.abs(out.astype(np.float64) - ref) / scale).max()) <= RTOL
