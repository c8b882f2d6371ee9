"""color_rays calls of one renderer on several streams, or captured, do not touch one another's image."""
import pytest
import torch

from helpers import sb
from spectral_b200 import configs

pytestmark = pytest.mark.gpu


def bits(image):
    """The image's words: out-of-gamut pixels are NaN, which equals nothing."""
    return image.view(torch.int32)


@pytest.mark.parametrize("frame,image", [((700, 500), (1400, 1000)), ((700, 500), (300, 1800)), ((700, 500), (700, 500)),
                                         ((300, 260), (300, 260))])
def test_exposures_on_two_streams(frame, image):
    s, c, ex = configs.box_scene(width=frame[0], height=frame[1], sphere_slices=8, sphere_stacks=9)
    c.image_width, c.image_height = image
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    with sb.Renderer(s, c, eems=ex["eems"], cmf=ex["cmf"]) as r:
        g = torch.Generator(device="cuda").manual_seed(5)
        r.block_film.copy_(torch.rand(c.bands, frame[1], frame[0], dtype=torch.float64, device="cuda", generator=g))
        r.average_and_reset_block(1)
        alone = []
        for exposure in (0.5, 4.0):
            r.config.exposure = exposure
            alone.append(bits(r.color_rays()).clone())
        torch.cuda.synchronize()
        images = []
        for k in range(40):
            r.config.exposure = (0.5, 4.0)[k % 2]
            with torch.cuda.stream(streams[k % 2]):
                images.append(bits(r.color_rays()))
        torch.cuda.synchronize()
    assert not torch.equal(alone[0], alone[1])
    for k, im in enumerate(images):
        assert torch.equal(im, alone[k % 2]), k


def test_captured_image_beside_another_stream():
    s, c, ex = configs.box_scene(width=700, height=500, sphere_slices=8, sphere_stacks=9)
    c.image_width, c.image_height = 1400, 1000
    with sb.Renderer(s, c, eems=ex["eems"], cmf=ex["cmf"]) as r:
        r.block_film.copy_(torch.rand(c.bands, 500, 700, dtype=torch.float64, device="cuda"))
        r.average_and_reset_block(1)
        r.config.exposure = 4.0
        other = bits(r.color_rays()).clone()
        r.config.exposure = 0.5
        image = torch.empty_like(r.color_rays())
        xyz = r.resolve_xyz().cpu()
        want = bits(r.color_rays()).clone()
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            r.color_rays(out=image)
        r.config.exposure = 4.0
        side = torch.cuda.Stream()
        for _ in range(10):
            image.fill_(0)
            side.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(side):
                beside = bits(r.color_rays())
            graph.replay()
            host = torch.from_numpy(r.resolve_xyz_host())
            torch.cuda.synchronize()
            assert torch.equal(bits(image), want) and torch.equal(beside, other)
            assert torch.equal(host, xyz)
        del graph
