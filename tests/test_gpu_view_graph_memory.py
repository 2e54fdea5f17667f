"""The graphs kept for View() are bounded by their size as well as their number:
scenes whose frames take thousands of launches do not add up."""
import pytest
import torch

from crystalgraphics_b200 import backend as B
from crystalgraphics_b200 import scenes

pytestmark = pytest.mark.gpu

KIB = 1 << 10


def used():
    free, total = torch.cuda.mem_get_info()
    return total - free


def test_large_graphs_do_not_add_up():
    s = scenes.textured_cornell()
    B.EnvInit(B.PathTraceConf(render_width=1280, render_height=720, sample_count=1, trace_depth=8))
    B.SetTuning(queue_capacity=1 << 14)  # hundreds of chunks
    cam = B.Camera.from_c(s.camera)
    loaded, after = [], []
    for _ in range(4):
        loaded.append(B.LoadScene(s))
        for _ in range(3):  # direct, captured, replayed
            B.View(loaded[-1], cam)
        after.append(used())
    launches = B.LastStats().kernel_launches
    assert launches > 20000
    # a graph takes about 2.6 KB of device memory a launch: three more scenes add
    # their own few MB, and not a graph each
    assert after[-1] - after[0] < 1.5 * 2.6 * KIB * launches
    for g in loaded:
        g.close()
    B.EnvTerm()
