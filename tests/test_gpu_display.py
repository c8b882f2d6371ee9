"""color_rays for images above, at and below the frame's size, against its formula in 64 bits."""
import numpy as np
import pytest
import torch

from helpers import sb
from spectral_b200 import configs, spectral_data

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("frame,image", [((1, 1), (1, 1)), ((33, 17), (33, 17)), ((33, 17), (66, 34)),
                                         ((33, 17), (101, 40)), ((50, 20), (1003, 1)), ((64, 48), (31, 23)),
                                         ((257, 255), (300, 511)), ((257, 255), (600, 511))])
def test_color_rays_of_any_image_size(frame, image):
    s, c, ex = configs.box_scene(width=frame[0], height=frame[1], sphere_slices=8, sphere_stacks=9)
    c.image_width, c.image_height = image
    rng = np.random.default_rng(3)
    film = rng.uniform(0.2, 1.0, (c.bands, frame[1], frame[0])) * rng.uniform(0.5, 2.0, (1, frame[1], frame[0]))
    with sb.Renderer(s, c, eems=ex["eems"], cmf=ex["cmf"]) as r:
        r.block_film.copy_(torch.from_numpy(film))
        r.average_and_reset_block(1)
        rgb = r.color_rays().cpu().numpy()
        xyz = r.resolve_xyz().cpu().numpy()
        scale, cmf = r.cmf_scale, np.asarray(r.compiled.cmf, np.float64)
    f = np.float32
    xyz64 = np.einsum("bhw,bc->hwc", film, cmf) * scale
    assert np.all(np.abs(xyz - xyz64) <= 2.0 ** -23 * np.abs(xyz64))  # one rounding to float32
    ri = (np.arange(image[0]).astype(f) / f(image[0]) * f(frame[0])).astype(int)
    rj = (np.arange(image[1]).astype(f) / f(image[1]) * f(frame[1])).astype(int)
    big = xyz64[rj][:, ri]
    M = np.asarray(spectral_data.srgb_xyz_to_rgb(), f).astype(np.float64).reshape(3, 3)
    e = c.exposure * (big @ M.T)
    ref = (e / (e + 1.0)) ** (1.0 / c.gamma)
    # h: three products and two sums of rounded factors, 5 roundings of at most sum |M| |x|; then the
    # quotient (2) and the power (2 units in the last place, its argument's error halved)
    mag = big @ np.abs(M).T
    tol = (5.0 * mag / np.abs(e) + 8.0) * 2.0 ** -23
    ok = np.isfinite(ref)
    assert np.array_equal(np.isnan(rgb), np.isnan(ref))
    assert np.all(np.abs(rgb - ref)[ok] <= (tol * np.abs(ref))[ok])
