"""Paths of no vertex: the wavefront kernel deposits nothing, whatever runs its passes."""
import pytest

from helpers import sb
from spectral_b200 import configs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("settings", [{}, {"sort_keys": 1}, {"queue_capacity": 100}, {"defer_passes": True}])
@pytest.mark.parametrize("width,height", [(1, 1), (40, 31), (592, 385)])
def test_wavefront_pass_without_vertices_leaves_the_film(width, height, settings):
    s, c, ex = configs.box_scene(width=width, height=height, depth=0, sphere_slices=8, sphere_stacks=9)
    cfg = sb.RenderConfig(**{**c.__dict__, "kernel": "wavefront", **settings})
    with sb.Renderer(s, cfg, eems=ex["eems"], cmf=ex["cmf"]) as r:
        r.block_film.fill_(0.25)
        for p in range(3):
            r.cast_rays(p, pass_idx=p)
        assert r.check_device() == 0
        assert bool((r.block_film == 0.25).all())
