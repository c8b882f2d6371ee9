"""The wavefront trace stage: a ray per lane and a group of lanes per ray give the megakernel's films,
on either side of the frame size that selects them, and where every hit is a tie."""
import numpy as np
import pytest
import torch

from helpers import sb
from spectral_b200 import configs

pytestmark = pytest.mark.gpu


def films(scene, cfg, ex, node_width, passes, kernels=("mega", "wavefront"), capacity=0):
    out = []
    for kern in kernels:
        c = sb.RenderConfig(**{**cfg.__dict__, "kernel": kern, "queue_capacity": capacity if kern != "mega" else 0})
        with sb.Renderer(scene, c, eems=ex["eems"], cmf=ex["cmf"], bvh_params={"width": node_width}) as r:
            for p in range(passes):
                r.cast_rays(p, pass_idx=p)
            assert r.check_device() == 0
            out.append(r.block_film.clone())
    return out


# 227,328 path slots: the most that get a group of lanes per ray
@pytest.mark.parametrize("width,height", [(1, 1), (33, 3), (592, 384), (592, 385)])
@pytest.mark.parametrize("node_width", [2, 4, 8])
def test_lanes_and_groups_give_the_megakernel_film(width, height, node_width):
    s, c, ex = configs.volume_scene(width=width, height=height, depth=6, medium_slices=20, medium_stacks=21)
    a, b = films(s, c, ex, node_width, 2)
    assert torch.allclose(a, b, rtol=1e-12, atol=0) and float(a.sum()) > 0


@pytest.mark.parametrize("capacity", [0, 300000])
@pytest.mark.parametrize("node_width", [2, 4, 8])
def test_ties_are_decided_alike(node_width, capacity):
    # every triangle twice, the copy with another material: each hit lies at exactly the distance of its copy
    s, c, ex = configs.box_scene(width=40, height=40, depth=5, sphere_slices=12, sphere_stacks=13)
    copies = [dict(m, material_id=m["material_id"] % 6 + 1) for m in s["meshes"]]
    s = dict(s, meshes=s["meshes"] + copies)
    a, b = films(s, c, ex, node_width, 3, capacity=capacity)
    assert torch.allclose(a, b, rtol=1e-12, atol=0) and float(a.sum()) > 0


@pytest.mark.parametrize("node_width", [2, 4, 8])
def test_axis_parallel_rays(node_width):
    # two components of every direction are zero, origins on the planes of boxes among them
    s, c, ex = configs.box_scene(sphere_slices=16, sphere_stacks=17)
    ax = np.linspace(-0.5, 0.5, 21)
    o = np.stack(np.meshgrid(ax, ax, [0.0], indexing="ij"), -1).reshape(-1, 3)
    rays = np.concatenate([np.concatenate([np.roll(o, k, 1), np.tile(np.roll([0.0, 0.0, sg], k), (len(o), 1))], 1)
                           for k in range(3) for sg in (-1.0, 1.0)]).astype(np.float32)
    with sb.Renderer(s, c, eems=ex["eems"], cmf=ex["cmf"], bvh_params={"width": node_width}) as r:
        tri, t, _, _ = r.trace(torch.from_numpy(rays).cuda())
        ref, tr, _, _ = r.trace(torch.from_numpy(rays).cuda(), mode="reference_order")
    assert torch.equal(t, tr) and torch.equal(tri < 0, ref < 0)
