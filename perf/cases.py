"""The work that a user of this framework has it do, as cases that can be timed.

Every case renders through the Python mirror of the public API: View() of a
moving and of a still camera, a rank's share of a frame (ViewSamples), a batch
of views, and a server's requests.  The scenes are the repository's own
(crystalgraphics_b200.scenes): the Cornell room (with and without material
textures), the dispersive icosphere of 1.31M triangles and the instanced scene
of 4096 objects and 10,000 emitters.  A scene's description is an asset that a
program reads once per process; it is loaded (LoadScene) anew for every state.
A state's seed gives the camera poses and the sample seeds.

Films come back as XYZ floats in host memory, as a headless program reads them
(into pinned memory that it keeps, except where the call allocates them).
"""
import math
import random

import numpy as np
import torch

from crystalgraphics_b200 import _abi, scenes
from crystalgraphics_b200 import backend as B

# What a scene is made of: its description, and the triangles of one instance
# and bytes of geometry and light buffers a frame has to read (for work()).
SCENES = {
    "cornell": dict(make=lambda: scenes.cornell(), tris=36, bytes=8e3),
    "textured": dict(make=lambda: scenes.textured_cornell(), tris=36, bytes=4e4),
    "icosphere": dict(make=lambda: scenes.icosphere_scene(), tris=1310786, bytes=1.15e8),
    "instanced": dict(make=lambda: scenes.instanced_scene(), tris=344 * 1024, bytes=4e7),
    "instanced2048": dict(make=lambda: scenes.instanced_scene(instances=2048, lights=2000, seed=5),
                          tris=344 * 1024, bytes=4e7),
}
_descriptions = {}
_env = None  # the conf and sampling options of the environment in place


def _description(name):
    if name not in _descriptions:
        _descriptions[name] = SCENES[name]["make"]()
    return _descriptions[name]


def _environment(case):
    """The process-wide environment that the case renders in (EnvInit only
    where another one is in place)."""
    global _env
    key = (case["width"], case["height"], case["spp"], case["depth"], case["hero"],
           case["roulette"])
    if _env == key:
        return
    B.EnvInit(B.PathTraceConf(render_width=case["width"], render_height=case["height"],
                              sample_count=case["spp"], trace_depth=case["depth"]))
    B.SetSpectral(_abi.CG_SPECTRAL_HERO if case["hero"] else _abi.CG_SPECTRAL_REFERENCE)
    B.SetRoulette(case["roulette"])
    _env = key


def _case(name, scene, width, height, spp, depth, form="view", frames="ab", hero=False, roulette=0,
          first=0, count=0):
    """form: "view" renders one frame per letter of `frames` (a pose each; the
    same letter again refines that pose's running mean), "share" the samples
    [first, first + count) of every pixel, "batch" `count` views in one call
    and "served" `count` requests through a server (their sizes are drawn up
    to width x height x spp)."""
    c = dict(scene=scene, form=form, width=width, height=height, spp=spp, depth=depth,
             frames=frames, hero=hero, roulette=roulette, first=first, count=count)
    return dict(c, name=name) if name else c


def listed():
    return [
        # an interactive preview of a small room: the camera moves, then rests for a frame
        _case("cornell_preview", "cornell", 256, 256, 1, 2, frames="abb"),
        # the same room with four wavelengths per sample and deeper paths
        _case("cornell_hero", "cornell", 640, 480, 4, 5, hero=True),
        # glTF-style material textures, glass and metal, a small still
        _case("textured_still", "textured", 320, 240, 8, 6),
        # a preview of one big mesh at an odd size
        _case("icosphere_preview", "icosphere", 427, 241, 3, 8, frames="abb"),
        # the benchmark frame: one big dispersive mesh, 720p, 16 samples, depth 8
        _case("icosphere_720p", "icosphere", 1280, 720, 16, 8),
        # the same with Russian roulette after the third bounce
        _case("icosphere_roulette", "icosphere", 1280, 720, 16, 8, roulette=3),
        # the same with four wavelengths per sample
        _case("icosphere_hero", "icosphere", 1280, 720, 16, 8, hero=True),
        # one sample per pixel of the two-level scene: navigating a large scene
        _case("instanced_preview", "instanced", 640, 360, 1, 12, frames="abb"),
        # a production frame of the two-level scene at full HD
        _case("instanced_1080p", "instanced", 1920, 1080, 16, 12),
        # one rank's share of a 64-sample frame split over eight GPUs
        _case("instanced_share", "instanced", 1920, 1080, 64, 12, form="share", first=24, count=8),
        # many views of one scene in one call (data sets, light fields)
        _case("batch_24", "instanced", 448, 448, 16, 12, form="batch", count=24),
        # a render service: requests of mixed sizes for two resident scenes
        _case("served_12", "icosphere", 1280, 720, 16, 8, form="served", count=12),
    ]


def draw(rng):
    kind = rng.choice(["view", "view", "view", "share", "batch", "served"])
    log = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))  # noqa: E731
    if kind == "batch":
        return _case(None, rng.choice(["cornell", "icosphere", "instanced"]), log(64, 448), log(64, 448),
                     rng.choice([4, 16]), rng.randint(4, 10), form="batch", count=rng.randint(2, 20))
    if kind == "served":
        return _case(None, "icosphere", log(256, 1280), log(144, 720), rng.choice([4, 16]),
                     rng.randint(4, 8), form="served", count=rng.randint(2, 10))
    scene = rng.choice(["cornell", "textured", "icosphere", "instanced"])
    width = log(64, 1600)
    height = max(36, int(width * rng.uniform(0.5, 1.0)))
    spp = log(1, 16)
    deepest = {"cornell": 6, "textured": 6, "icosphere": 8, "instanced": 12}[scene]
    depth = rng.randint(2, deepest)
    hero = rng.random() < 0.25
    roulette = 3 if rng.random() < 0.25 else 0
    if kind == "share":
        first = rng.randint(0, spp - 1)
        return _case(None, scene, width, height, spp, depth, form="share", hero=hero,
                     roulette=roulette, first=first, count=rng.randint(1, spp - first))
    return _case(None, scene, width, height, spp, depth, frames=rng.choice(["ab", "abb"]), hero=hero,
                 roulette=roulette)


def _pose(scene, rng):
    """A camera that looks at the scene."""
    if scene in ("cornell", "textured"):  # in front of the open side of the room
        return ((rng.uniform(-0.25, 0.25), rng.uniform(-3.6, -3.2), rng.uniform(0.8, 1.2)),
                (rng.uniform(-0.07, 0.07), 1.0, rng.uniform(-0.05, 0.05)))
    if scene == "icosphere":  # around the mesh, a little above the ground
        a, r, z = rng.uniform(0, 2 * math.pi), rng.uniform(3.8, 4.6), rng.uniform(0.3, 1.2)
        d = (-r * math.cos(a), -r * math.sin(a), -z)
        n = math.sqrt(sum(x * x for x in d))
        return (r * math.cos(a), r * math.sin(a), z), tuple(x / n for x in d)
    g = np.random.default_rng(rng.randrange(1 << 30))
    p, d = scenes.sphere_pose(g)
    return tuple(map(float, p)), tuple(map(float, d))


def _film(width, height):
    return torch.empty((height, width, 3), dtype=torch.float32, pin_memory=True).numpy()


def prepare(case, seed):
    rng = random.Random(seed * 1000003 + 17)
    _environment(case)
    names = [case["scene"]] + (["instanced2048"] if case["form"] == "served" else [])
    loaded = [B.LoadScene(_description(n)) for n in names]
    state = dict(case=case, scenes=loaded, seed=rng.randrange(1 << 31))
    if case["form"] in ("view", "share"):
        frames = case["frames"] if case["form"] == "view" else "a"
        viewport = scenes.camera_viewport(case["width"], case["height"], 0.45)
        poses = {k: B.Camera(*_pose(case["scene"], rng), viewport) for k in sorted(set(frames))}
        state["cameras"] = [poses[k] for k in frames]
        state["films"] = [_film(case["width"], case["height"]) for _ in frames]
        return state
    items = []  # (scene, position, direction, width, height, spp, seed)
    sizes = random.Random(case["count"])  # the mix of sizes is the case's, the views are the seed's
    for k in range(case["count"]):
        which = sizes.randrange(len(names))
        # sides spread over the logarithm up to the case's, the first one the largest
        part = math.exp(sizes.uniform(math.log(0.14), 0.0)) if k else 1.0
        spp = sizes.choice([s for s in (1, 4, 16) if s <= case["spp"]]) if k else case["spp"]
        items.append((which, *_pose(names[which], rng), max(16, int(case["width"] * part)),
                      max(16, int(case["height"] * part)), spp, rng.randrange(1 << 31)))
    if case["form"] == "batch":
        state["views"] = B.make_views([i[1:] for i in items])
    else:
        state["server"] = B.Server(loaded, 64 << 30)
        state["requests"] = [(*i, None, _film(i[3], i[4])) for i in items]
    return state


def run(state):
    case = state["case"]
    _environment(case)
    if case["form"] == "view":
        B.SetSeed(state["seed"])
        for camera, film in zip(state["cameras"], state["films"]):
            B.View(state["scenes"][0], camera)
            B.ReadFilm(_abi.CG_FILM_XYZ32F, film)
        return state["films"]
    if case["form"] == "share":
        B.SetSeed(state["seed"])
        B.ViewSamples(state["scenes"][0], state["cameras"][0], case["first"], case["count"])
        return B.ReadFilm(_abi.CG_FILM_XYZ32F, state["films"][0])
    if case["form"] == "batch":
        return B.batch_render(state["scenes"][0], state["views"])
    ids = [state["server"].submit(*r) for r in state["requests"]]
    return [state["server"].wait(i)[0] for i in ids]


def work(case):
    """Bytes: the scene read once and the films written once.  Flops: one walk
    per camera sample and bounce that cannot be left out (a third of the depth),
    each down to one leaf of a balanced four-wide tree (16 flops a box, 40 a
    triangle), and 200 flops of shading."""
    per = case["count"] * 0.3 if case["form"] in ("batch", "served") else 1
    frames = len(case["frames"]) if case["form"] == "view" else per
    spp = case["count"] if case["form"] == "share" else case["spp"]
    pixels = case["width"] * case["height"] * frames
    walk = 64 * math.ceil(math.log(SCENES[case["scene"]]["tris"], 4)) + 40 + 200
    lanes = 4 if case["hero"] else 1
    return {"bytes": SCENES[case["scene"]]["bytes"] + 12 * pixels,
            "flops": pixels * spp * max(1, case["depth"] / 3) * (walk + 200 * (lanes - 1))}


def exact(case, seed):
    """None: a film is a Monte Carlo estimate of its own sample streams, which
    no formula in 64 bits gives."""
    return None
