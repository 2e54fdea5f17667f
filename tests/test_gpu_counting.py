"""Traversal counters (SetCounting) are those of the one-ray walk: they repeat from
run to run and do not depend on which lanes share a walk."""
import pytest

from crystalgraphics_b200 import backend as B
from crystalgraphics_b200 import scenes

pytestmark = pytest.mark.gpu


def instances(mesh_scale):
    return scenes.instanced_scene(width=64, height=48, spp=1, depth=6, instances=96, lights=40, seed=9,
                                  mesh_scale=mesh_scale, extent=1.5, camera_distance=9.0)


# below and above the tree size from which idle lanes help
SCENES = {"small mesh": lambda: scenes.icosphere_scene(subdiv=4), "deep mesh": lambda: scenes.icosphere_scene(subdiv=7),
          "small instances": lambda: instances(0.05), "deep instances": lambda: instances(1.0)}


@pytest.mark.parametrize("name", sorted(SCENES))
@pytest.mark.parametrize("size", [(33, 1, 3), (160, 90, 2)])
def test_counters_are_those_of_the_one_ray_walk(name, size):
    s = SCENES[name]()
    w, h, spp = size
    B.EnvInit(B.PathTraceConf(render_width=w, render_height=h, sample_count=spp, trace_depth=6))
    g = B.LoadScene(s)
    cam = B.Camera.from_c(s.camera)

    def counts(**tuning):
        B.SetTuning(**tuning)
        B.ViewSamples(g, cam, 0, spp)
        st = B.LastStats()
        return st.extend_rays, st.shadow_rays, st.node_visits, st.tri_tests, st.inst_visits

    B.SetCounting(True)
    ref = counts(persistent=False)
    assert min(ref[2:]) > 0
    for _ in range(2):
        assert counts(persistent=True) == ref
    B.SetCounting(False)
    assert counts(persistent=True) == ref[:2] + (0, 0, 0)
    g.close()
    B.EnvTerm()
