"""The trace stages by themselves: sorted queues keep a small pass on the stages, a queue capacity puts it on the loop.
All ways to run a stage (a group of lanes per ray, a ray per lane at its own pace, a warp's rays together) and their
lists of ties give the megakernel's film."""
import numpy as np
import pytest
import torch

from helpers import sb
from spectral_b200 import batch as sbatch
from spectral_b200 import configs

pytestmark = pytest.mark.gpu

LAYOUTS = [(2, False), (4, False), (8, False), (4, True), (8, True)]


def renderer(scene, cfg, ex, width, quantize=False, **settings):
    return sb.Renderer(scene, sb.RenderConfig(**{**cfg.__dict__, **settings}), eems=ex["eems"], cmf=ex["cmf"],
                       bvh_params={"width": width, "quantize": quantize})


def film(r, passes, bundle=False):
    r.clear_pixel_space()
    if bundle:  # of more passes than path slots: they are filled again
        r.cast_rays_bundle(0, passes, pass_idx=0)
    else:
        for p in range(passes):
            r.cast_rays(p, pass_idx=p)
    assert r.check_device() == 0
    return r.block_film.clone()


def doubled(scene):
    """Every triangle twice, the copy with another material: each hit lies at exactly the distance of its copy."""
    copies = [dict(m, material_id=m["material_id"] % 6 + 1) for m in scene["meshes"]]
    return dict(scene, meshes=scene["meshes"] + copies)


# FP64 film sums in another order: equal to a few last bits.  Paths on either side of what selects the way: 56,832 and
# 227,328 slots that are filled again, 113,664 and 378,880 paths of a pass
@pytest.mark.parametrize("width,height", [(1, 1), (33, 3), (296, 192), (297, 192), (592, 192), (593, 192), (592, 384),
                                          (592, 385), (640, 592), (640, 593)])
@pytest.mark.parametrize("node_width,quantize", LAYOUTS)
def test_stages_and_loop_give_the_megakernel_film(width, height, node_width, quantize):
    s, c, ex = configs.volume_scene(width=width, height=height, depth=6, medium_slices=20, medium_stacks=21)
    with renderer(s, c, ex, node_width, quantize, kernel="mega") as r:
        a = film(r, 2)
        assert float(a.sum()) > 0
        for settings in ({"sort_keys": 1}, {"sort_keys": 7}, {"queue_capacity": width * height}):
            r.set_launch_config(**{"kernel": "wavefront", "sort_keys": 0, "queue_capacity": 0, **settings})
            assert torch.allclose(a, film(r, 2), rtol=1e-12, atol=0), settings
            if "queue_capacity" in settings:
                assert r.wave_loop_iterations() > 0
                assert torch.allclose(a, film(r, 2, bundle=True), rtol=1e-12, atol=0), settings


# a tree of more than 32,768 triangles: 1,060,864 slots that are filled again; passes at their own pace, above 227,328
# pixels with two children
@pytest.mark.parametrize("width,height", [(592, 384), (592, 385), (1024, 1036), (1024, 1037)])
@pytest.mark.parametrize("node_width,quantize", LAYOUTS[:2] + LAYOUTS[4:])
def test_large_tree(width, height, node_width, quantize):
    s, c, ex = configs.terrain_scene(width=width, height=height, depth=3, grid=140, sphere_slices=20, sphere_stacks=21)
    with renderer(s, c, ex, node_width, quantize, kernel="mega") as r:
        assert r.scene_info()["num_tris"] > 32768
        a = film(r, 2)
        assert float(a.sum()) > 0
        for settings in ({"sort_keys": 1}, {"queue_capacity": width * height}):
            r.set_launch_config(**{"kernel": "wavefront", "sort_keys": 0, "queue_capacity": 0, **settings})
            bundle = "queue_capacity" in settings
            assert torch.allclose(a, film(r, 2, bundle), rtol=1e-12, atol=0), settings


# 1,600 paths: groups, which decide their ties at once; 60,000 and 240,000: slots that are filled again at their own pace
# and together, a pass in groups and at its own pace, whose ties go to lists
@pytest.mark.parametrize("width,height", [(40, 40), (300, 200), (600, 400)])
@pytest.mark.parametrize("node_width", [2, 4, 8])
def test_ties_in_stages_and_loop(width, height, node_width):
    s, c, ex = configs.box_scene(width=width, height=height, depth=5, sphere_slices=12, sphere_stacks=13)
    with renderer(doubled(s), c, ex, node_width, kernel="mega") as r:
        a = film(r, 2)
        assert float(a.sum()) > 0
        for settings in ({"sort_keys": 1}, {"sort_keys": 7}, {}, {"queue_capacity": width * height}):
            r.set_launch_config(**{"kernel": "wavefront", "sort_keys": 0, "queue_capacity": 0, **settings})
            assert torch.allclose(a, film(r, 2), rtol=1e-12, atol=0), settings
            if "queue_capacity" in settings:
                assert torch.allclose(a, film(r, 2, bundle=True), rtol=1e-12, atol=0), settings


# all paths of a step in their slots, 62,000 and 372,000 (own pace), 620,000 (together); 230,000 slots filled again
# (together)
@pytest.mark.parametrize("width,slots", [(40, 0), (240, 0), (400, 0), (310, 230000)])
@pytest.mark.parametrize("use_graph", [True, False])
@pytest.mark.parametrize("node_width", [2, 4, 8])
def test_ties_in_a_wavefront_batch(node_width, use_graph, width, slots):
    rs = []
    for k in range(2):
        s, c, ex = configs.box_scene(seed=k, width=width, height=31, depth=5, sphere_slices=12, sphere_stacks=13)
        rs.append(renderer(doubled(s), c, ex, node_width, kernel="mega"))
    films = []
    for kernel in ("mega", "wavefront"):
        with sbatch.Batch(rs, kernel=kernel, use_graph=use_graph,
                          queue_capacity=slots if kernel == "wavefront" else 0) as b:
            b.reset(0)
            b.step()
            assert b.check() == 0
            films.append([r.mean_film.clone() for r in rs])
    for x, y in zip(*films):
        assert torch.allclose(x, y, rtol=1e-12, atol=0) and float(x.sum()) > 0
    for r in rs:
        r.close()


# more rays than get a group of lanes each (75,776, or 113,664 with two children), against queries of fewer: the same
# triangle of each coincident pair
@pytest.mark.parametrize("rays_in_query", [75777, 113665])
@pytest.mark.parametrize("node_width,quantize", LAYOUTS)
def test_ties_of_a_large_query(node_width, quantize, rays_in_query):
    s, c, ex = configs.box_scene(sphere_slices=24, sphere_stacks=25)
    g = torch.Generator(device="cuda").manual_seed(11)
    d = torch.randn(rays_in_query, 3, device="cuda", generator=g)
    o = torch.rand(rays_in_query, 3, device="cuda", generator=g) * 0.9 - 0.45
    rays = torch.cat([o, d / d.norm(dim=1, keepdim=True)], 1).contiguous()
    with renderer(doubled(s), c, ex, node_width, quantize) as r:
        large = r.trace(rays)
        part = min(50001, len(rays) // 2)
        parts = [r.trace(rays[k:k + part]) for k in range(0, len(rays), part)]
        ref = r.trace(rays, mode="reference_order")
        assert r.check_device() == 0
    for k in range(4):
        assert torch.equal(large[k], torch.cat([p[k] for p in parts])), k
    assert float((large[1] == ref[1]).float().mean()) > 0.999  # distances: but for near ties
    n = sum(len(m["faces"]) for m in s["meshes"])
    hit = large[0] >= 0
    assert float(hit.float().mean()) > 0.9
    same = large[1] == ref[1]
    assert bool(((large[0] % n) == (ref[0] % n))[same & hit].float().mean() > 0.99)
