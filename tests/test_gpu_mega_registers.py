"""The register budget that the megakernel takes by itself, on either side of the number of paths that selects it."""
import pytest
import torch

from helpers import sb
from spectral_b200 import configs

pytestmark = pytest.mark.gpu


# 2^19 = 524,288 paths: 64 registers from there on.  Film sums are FP64 in path order: equal to a few last bits
@pytest.mark.parametrize("width,height,passes", [(31, 5, 1), (169, 126, 24), (169, 126, 25), (8192, 64, 1), (8191, 64, 1)])
def test_budget_by_paths_gives_the_film_of_both_budgets(width, height, passes):
    s, c, ex = configs.box_scene(width=width, height=height, depth=4, sphere_slices=12, sphere_stacks=13)
    films = []
    with sb.Renderer(s, sb.RenderConfig(**{**c.__dict__, "kernel": "mega"}), eems=ex["eems"], cmf=ex["cmf"]) as r:
        for occupancy in (0, 5, 8):
            r.set_launch_config(occupancy=occupancy)
            r.clear_pixel_space()
            if passes == 1:
                r.cast_rays(0, pass_idx=0)
            else:
                r.cast_rays_bundle(0, passes, pass_idx=0)
            assert r.check_device() == 0
            films.append(r.block_film.clone())
    for f in films[1:]:
        assert torch.allclose(films[0], f, rtol=1e-12, atol=0) and float(f.sum()) > 0
