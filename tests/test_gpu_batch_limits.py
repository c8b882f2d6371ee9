"""Batches of different sizes side by side: creating one changes nothing for another."""
import pytest
import torch

from helpers import sb
from spectral_b200 import batch as sbatch
from spectral_b200 import configs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("use_graph", [False, True])
def test_small_batch_made_after_a_large_one(use_graph):
    s, c, ex = configs.box_scene(width=16, height=16, depth=3, sphere_slices=8, sphere_stacks=9)
    owner = sb.Renderer(s, c, eems=ex["eems"], cmf=ex["cmf"])
    views = [owner.view() for _ in range(128)]
    with sbatch.Batch(views, use_graph=use_graph) as large:
        large.reset(0)
        with sbatch.Batch([owner], use_graph=use_graph) as small:
            small.reset(0)
            small.step()
            large.step()
            assert small.check() == 0 and large.check() == 0
        want = owner.mean_film.clone()
        assert float(want.sum()) > 0
        for v in views[::31]:
            assert torch.allclose(v.mean_film, want, rtol=1e-12, atol=0)
    for r in views + [owner]:
        r.close()
