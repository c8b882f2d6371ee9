"""Adopted trees whose leaves hold more triangles than a device leaf: which of two coincident triangles wins."""
import numpy as np
import pytest
import torch

from helpers import sb
from spectral_b200 import configs

pytestmark = pytest.mark.gpu


def big_leaf_scene(root_is_leaf):
    """A leaf of 36 triangles, split in halves of 18 and those in nines.  Triangles 3 and 21 coincide in the plane
    z = 0; triangle 30, beside the ray, lies at z = 1 and so brings the box of the second half nearer."""
    far = lambda z: [[5.0, 5.0, z], [6.0, 5.0, z], [5.0, 6.0, z]]
    tris = np.array([far(0.0)] * 36)
    tris[3] = tris[21] = [[-1.0, -1.0, 0.0], [3.0, -1.0, 0.0], [-1.0, 3.0, 0.0]]
    tris[30] = [[-9.0, -9.0, 1.0], [9.0, -9.0, 1.0], [9.0, -8.0, 1.0]]
    s, c, ex = configs.box_scene(width=16, height=16, sphere_slices=8, sphere_stacks=9)
    verts = tris.reshape(-1, 3)
    meshes = [{"vertices": verts, "faces": np.arange(len(verts)).reshape(-1, 3), "material_id": 1}]
    n = 36
    if not root_is_leaf:  # a second leaf of one triangle behind the others
        meshes.append({"vertices": np.array([[-1.0, -1.0, -2.0], [3.0, -1.0, -2.0], [-1.0, 3.0, -2.0]]),
                       "faces": np.array([[0, 1, 2]]), "material_id": 1})
        n = 37
    big = ([-9.1, -9.1, -0.1], [9.1, 9.1, 1.1])
    small = ([-1.1, -1.1, -2.1], [3.1, 3.1, -1.9])
    if root_is_leaf:
        boxes, left, right, cnt, start = [big], [-1], [-1], [36], [0]
    else:
        boxes = [([-9.1, -9.1, -2.1], [9.1, 9.1, 1.1]), big, small]
        left, right, cnt, start = [1, -1, -1], [2, -1, -1], [0, 36, 1], [0, 0, 36]
    bvh = {"node_min": np.array([b[0] for b in boxes]), "node_max": np.array([b[1] for b in boxes]),
           "node_left": left, "node_right": right, "node_num_tris": cnt, "node_tri_start": start,
           "tri_perm": np.arange(n)}
    return dict(s, meshes=meshes), c, ex, bvh


# groups of lanes per ray, and more rays than get them
@pytest.mark.parametrize("rays", [1, 70, 200000])
@pytest.mark.parametrize("root_is_leaf", [True, False])
@pytest.mark.parametrize("node_width", [2, 4, 8])
def test_tie_between_the_halves_of_a_big_leaf(node_width, root_is_leaf, rays):
    s, c, ex, bvh = big_leaf_scene(root_is_leaf)
    q = torch.tensor([[0.25, 0.25, 5.0, 0.0, 0.0, -1.0]], device="cuda").repeat(rays, 1)
    with sb.Renderer(s, c, eems=ex["eems"], cmf=ex["cmf"], bvh=bvh, bvh_params={"width": node_width}) as r:
        assert r.scene_info()["num_ref_nodes"] == len(bvh["node_left"])
        tri, t, _, _ = r.trace(q)
        ref, tr, _, _ = r.trace(q, mode="reference_order")
        assert r.check_device() == 0
    assert bool((t == 5.0).all()) and bool((tr == 5.0).all())
    assert bool((tri == 21).all())  # the second half is entered first
    assert bool((ref == 3).all())   # the reference takes a leaf's triangles in order


def chain_scene(depth):
    """A tree that is one chain: node k has triangle k, at height k, and the rest above it.  A ray from above enters
    every box, the rest's first, and leaves a triangle waiting at each level."""
    n = depth + 1
    tris = np.array([[[-1.0, -1.0, float(k)], [3.0, -1.0, float(k)], [-1.0, 3.0, float(k)]] for k in range(n)])
    s, c, ex = configs.box_scene(width=16, height=16, sphere_slices=8, sphere_stacks=9)
    meshes = [{"vertices": tris.reshape(-1, 3), "faces": np.arange(3 * n).reshape(-1, 3), "material_id": 1}]
    lo, hi, left, right, cnt, start = [], [], [], [], [], []
    for k in range(depth):  # inner node 2k, its leaf 2k + 1; the last inner node's second child is the leaf 2 * depth
        lo += [[-1.1, -1.1, k - 0.1], [-1.1, -1.1, k - 0.1]]
        hi += [[3.1, 3.1, depth + 0.1], [3.1, 3.1, k + 0.1]]
        left += [2 * k + 1, -1]
        right += [2 * k + 2, -1]
        cnt += [0, 1]
        start += [0, k]
    lo, hi = lo + [[-1.1, -1.1, depth - 0.1]], hi + [[3.1, 3.1, depth + 0.1]]
    left, right, cnt, start = left + [-1], right + [-1], cnt + [1], start + [depth]
    bvh = {"node_min": np.array(lo), "node_max": np.array(hi), "node_left": left, "node_right": right,
           "node_num_tris": cnt, "node_tri_start": start, "tri_perm": np.arange(n)}
    return dict(s, meshes=meshes), c, ex, bvh


# more waiting boxes than a group of lanes has room for (32); from below the nearest triangle comes first
@pytest.mark.parametrize("rays", [1, 70, 200000])
@pytest.mark.parametrize("depth", [1, 20, 60])
@pytest.mark.parametrize("node_width,quantize", [(2, False), (4, False), (8, False), (4, True), (8, True)])
def test_deep_chain(node_width, quantize, depth, rays):
    s, c, ex, bvh = chain_scene(depth)
    down = torch.tensor([[0.25, 0.25, 100.0, 0.0, 0.0, -1.0]], device="cuda").repeat(rays, 1)
    up = torch.tensor([[0.25, 0.25, -100.0, 0.0, 0.0, 1.0]], device="cuda").repeat(rays, 1)
    with sb.Renderer(s, c, eems=ex["eems"], cmf=ex["cmf"], bvh=bvh,
                     bvh_params={"width": node_width, "quantize": quantize}) as r:
        for mode in ("fast", "reference_order"):
            tri, t, _, _ = r.trace(down, mode=mode)
            assert bool((tri == depth).all()) and bool((t == 100.0 - depth).all()), mode
            tri, t, _, _ = r.trace(up, mode=mode)
            assert bool((tri == 0).all()) and bool((t == 100.0).all()), mode
        assert r.check_device() == 0


@pytest.mark.parametrize("rays", [1, 200000])
@pytest.mark.parametrize("node_width,quantize", [(2, False), (4, False), (8, False), (4, True), (8, True)])
def test_single_triangle(node_width, quantize, rays):
    s, c, ex = configs.box_scene(width=16, height=16, depth=3, sphere_slices=8, sphere_stacks=9)
    tri = {"vertices": np.array([[-1.0, -1.0, 0.0], [3.0, -1.0, 0.0], [-1.0, 3.0, 0.0]]), "faces": np.array([[0, 1, 2]]),
           "material_id": 1}
    q = torch.tensor([[0.25, 0.25, 5.0, 0.0, 0.0, -1.0], [0.25, 0.25, 5.0, 0.0, 0.0, 1.0]], device="cuda").repeat(rays, 1)
    with sb.Renderer(dict(s, meshes=[tri]), c, eems=ex["eems"], cmf=ex["cmf"],
                     bvh_params={"width": node_width, "quantize": quantize}) as r:
        hit, t, _, _ = r.trace(q)
        assert bool((hit[0::2] == 0).all()) and bool((t[0::2] == 5.0).all()) and bool((hit[1::2] == -1).all())
        r.cast_rays(0)
        assert r.check_device() == 0
