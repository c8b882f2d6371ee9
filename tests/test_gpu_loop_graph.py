"""The regenerating loop's captured graph is kept while only the number of passes of a launch changes."""
import statistics
import time

import pytest
import torch

from helpers import sb
from spectral_b200 import configs

pytestmark = pytest.mark.gpu


def host_ms(r, launches):
    """median host time of the launches, each on an idle device"""
    times = []
    for settings, passes in launches:
        if settings:
            r.set_launch_config(**settings)
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        r.cast_rays_bundle(0, passes, pass_idx=0)
        times.append((time.perf_counter() - t0) * 1e3)
    torch.cuda.synchronize()
    return statistics.median(times[2:])


# 300 x 300: 25 and 7 passes get a ray per lane; 2 passes (180,000 paths) and 1 a group of lanes
@pytest.mark.parametrize("a,b", [(25, 7), (25, 2), (2, 1)])
def test_changing_the_number_of_passes_builds_no_graph(a, b):
    s, c, ex = configs.box_scene(width=300, height=300, depth=2, sphere_slices=8, sphere_stacks=9)
    cfg = sb.RenderConfig(**{**c.__dict__, "kernel": "wavefront", "queue_capacity": 25 * 300 * 300})
    with sb.Renderer(s, cfg, eems=ex["eems"], cmf=ex["cmf"]) as r:
        built = host_ms(r, [({"block_size": (128, 256)[k % 2]}, a) for k in range(12)])
        kept = host_ms(r, [(None, (a, b)[k % 2]) for k in range(24)])
        assert r.check_device() == 0
    # a launch is two calls; a build captures, instantiates and uploads a graph besides
    assert kept < 0.5 * built, (kept, built)
