"""Performance cases of the renderer: the work a user's program has it do, through its public calls.

Each case names one kind of call with its sizes:

  pass      an interactive viewer after a camera move: the film cleared and one sample pass cast
  block     the reference's cadence on a default Renderer: one cast_rays per band, the block averaged, the image resolved
  bundle    offline rendering: a whole spectral block in one launch, averaged and resolved to XYZ
  gradient  one step of inverse rendering: the film of one block and the gradient of an image loss
  batch     one step of a batch of scenes (a spectral block of each)
  rays      closest-hit queries of a ray array
  display   the block average and the image of a film that is already rendered

Scenes are the package's own workload generators (box, terrain, volume).  The seed draws the scene's materials (box and
volume), the camera's position, the random stream, the rays or the film.  The terrain's mesh and its tree, which a
program loads once, are kept from one preparation to the next.
"""
import functools
import math

import numpy as np
import torch

import spectral_b200 as sb
from spectral_b200 import autodiff, configs
from spectral_b200.batch import Batch

BANDS = configs.BANDS
MAX_SLOTS = 1 << 25  # path slots of a wavefront loop (RenderConfig.queue_capacity)


def listed():
    return [
        # the smallest call: a thumbnail preview, one pass of few paths, where launches and latency are everything
        {"name": "preview_box_64", "kind": "pass", "scene": "box", "tris": 2062, "width": 64, "height": 64, "depth": 8,
         "kernel": "wavefront"},
        # a preview of a mid-size mesh in an odd window size with the one-kernel renderer
        {"name": "preview_terrain_333x217", "kind": "pass", "scene": "terrain", "tris": 100000, "width": 333,
         "height": 217, "depth": 12, "kernel": "mega"},
        # the reference's render loop as it stands in its application, default settings, the box workload's frame
        {"name": "block_box_256", "kind": "block", "scene": "box", "tris": 2062, "width": 256, "height": 256,
         "depth": 8, "kernel": "wavefront"},
        # the same loop on a large mesh and a frame that no tile divides
        {"name": "block_terrain_401x299", "kind": "block", "scene": "terrain", "tris": 647258, "width": 401,
         "height": 299, "depth": 12, "kernel": "wavefront"},
        # offline rendering of the box workload with tuned settings: all 25 passes of a block in flight
        {"name": "bundle_box_256", "kind": "bundle", "scene": "box", "tris": 2062, "width": 256, "height": 256,
         "depth": 8, "kernel": "wavefront", "node_width": 4, "budget": 8, "slots": BANDS * 256 * 256},
        # the benchmark's workload: 2.59M triangles, 1024^2, depth 12, tuned settings
        {"name": "bundle_terrain_1024", "kind": "bundle", "scene": "terrain", "tris": 2593074, "width": 1024,
         "height": 1024, "depth": 12, "kernel": "wavefront", "node_width": 4, "budget": 16,
         "slots": BANDS * 1024 * 1024},
        # the volume and fluorescence workload: paths up to 32 vertices, tuned settings
        {"name": "bundle_volume_512", "kind": "bundle", "scene": "volume", "tris": 20014, "width": 512, "height": 512,
         "depth": 32, "kernel": "wavefront", "node_width": 4, "budget": 8, "slots": BANDS * 512 * 512},
        # inverse rendering at its workload's frame: forward block and adjoint, material and EEM gradients
        {"name": "gradient_volume_256", "kind": "gradient", "scene": "volume", "tris": 20014, "width": 256,
         "height": 256, "depth": 32, "kernel": "mega"},
        # the same at a small odd frame of a surface-only scene, the size of a unit of a larger optimisation
        {"name": "gradient_box_75x53", "kind": "gradient", "scene": "box", "tris": 2062, "width": 75, "height": 53,
         "depth": 8, "kernel": "mega"},
        # many small uneven scenes at once, the batch's default engine
        {"name": "batch_12_scenes", "kind": "batch", "scenes": 12, "tris": 8000, "width": 128, "height": 128,
         "depth": 16, "kernel": "mega"},
        # geometry queries on the large mesh, a count that no block divides
        {"name": "rays_terrain_1m", "kind": "rays", "scene": "terrain", "tris": 2593074, "rays": 1000003},
        # the end of every block at the benchmark's frame: average, display image, XYZ
        {"name": "display_1024", "kind": "display", "scene": "box", "tris": 2062, "width": 1024, "height": 1024,
         "image_width": 1600, "image_height": 1600},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["pass", "block", "bundle", "bundle", "gradient", "batch", "rays", "display"])
    scene = rng.choice(["box", "terrain", "volume"])
    if kind == "rays":
        return {"kind": kind, "scene": scene, "tris": _log(rng, 2000, 650000), "rays": _log(rng, 1000, 2000000)}
    if kind == "display":
        w, h = _log(rng, 48, 1024), _log(rng, 48, 1024)
        up = rng.choice([1, 2])
        return {"kind": kind, "scene": "box", "tris": 2062, "width": w, "height": h, "image_width": up * w,
                "image_height": up * h}
    if kind == "batch":
        side = _log(rng, 32, 160)
        return {"kind": kind, "scenes": rng.randint(2, 12), "tris": _log(rng, 1000, 20000), "width": side,
                "height": max(16, side - rng.randint(0, 9)), "depth": rng.randint(4, 16),
                "kernel": rng.choice(["mega", "wavefront"])}
    w = _log(rng, 48, 160 if kind == "gradient" else 512)
    h = max(32, int(w * rng.uniform(0.5, 1.0)))
    depth = rng.randint(4, 12) if scene != "volume" else rng.randint(8, 32)
    case = {"kind": kind, "scene": scene, "tris": _log(rng, 1000, 20000 if scene == "volume" else 650000), "width": w,
            "height": h, "depth": depth, "kernel": rng.choice(["mega", "wavefront"])}
    if kind == "bundle":
        passes = rng.choice([1, 2, 4, BANDS])  # frames' worth of paths in flight
        case.update(node_width=rng.choice([2, 4, 8]), budget=rng.choice([8, 16]), slots=passes * w * h)
    if kind == "gradient":
        case["kernel"] = "mega"
    return case


# ------------------------------------------------------------------------------------------------ preparation
@functools.lru_cache(maxsize=2)
def _terrain(tris):
    grid = max(8, int(round(math.sqrt(0.807 * tris / 2))) + 1)
    n = max(8, int(round(math.sqrt(0.193 * tris / 2))))
    scene, cfg, extras = configs.terrain_scene(grid=grid, sphere_slices=n, sphere_stacks=n + 1)
    tri = sb.compile_scene(scene, cfg.bands).tris
    return scene, cfg, extras, sb._lib.build_bvh_host(tri["v0"], tri["v1"], tri["v2"])


def _scene(kind, tris, seed):
    """(scene, config, extras, tree): the generator's scene at about `tris` triangles."""
    n = max(8, int(round(math.sqrt(tris / 2))))
    if kind == "terrain":
        scene, cfg, extras, tree = _terrain(tris)
    elif kind == "volume":
        (scene, cfg, extras), tree = configs.volume_scene(seed=seed, medium_slices=n, medium_stacks=n + 1,
                                                          fluorescent_medium=seed % 2 == 0), None
    else:
        (scene, cfg, extras), tree = configs.box_scene(seed=seed, sphere_slices=n, sphere_stacks=n + 1), None
    rng = np.random.default_rng(seed)
    camera = dict(scene["camera"])
    camera["origin"] = (np.asarray(camera["origin"]) * (1.0 - 0.03 * rng.uniform(0, 1, 3))).tolist()
    return dict(scene, camera=camera), cfg, extras, tree


def _renderer(case, seed, scene=None, depth=None):
    scene, cfg, extras, tree = scene or _scene(case["scene"], case["tris"], seed)
    c = sb.RenderConfig(width=case.get("width", 64), height=case.get("height", 64), bands=BANDS,
                        lambda_min=cfg.lambda_min, lambda_max=cfg.lambda_max,
                        max_path_length=depth or case.get("depth", 8), fov_scale=cfg.fov_scale,
                        image_width=case.get("image_width", case.get("width", 64)),
                        image_height=case.get("image_height", case.get("height", 64)), seed=seed,
                        kernel=case.get("kernel", "wavefront"))
    if case["kind"] == "bundle":
        c.queue_capacity, c.trace_budget, c.block_size = min(case["slots"], MAX_SLOTS), case["budget"], 256
    return sb.Renderer(scene, c, eems=extras["eems"], cmf=extras["cmf"], bvh=tree,
                       bvh_params={"width": case.get("node_width", 0)})


def _rays(case, seed):
    """Origins in the scene's air and directions over the sphere, most of them towards the geometry."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    n = case["rays"]
    d = torch.randn(n, 3, device="cuda", generator=g)
    u = torch.rand(n, 3, device="cuda", generator=g) * 2 - 1
    if case["scene"] == "terrain":
        o = u * torch.tensor([11.0, 2.0, 11.0], device="cuda") + torch.tensor([0.0, 5.0, 0.0], device="cuda")
        d[:, 1] = -d[:, 1].abs()
    else:
        o = u * 0.49
    return torch.cat([o, d / d.norm(dim=1, keepdim=True)], 1).contiguous()


def _film(case, seed):
    """A block's film as rendering leaves it: smooth spectra with per-cell noise, [B, H, W] float64."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    H, W = case["height"], case["width"]
    lum = torch.rand(1, H, W, dtype=torch.float64, device="cuda", generator=g) ** 2 + 0.02
    noise = torch.rand(BANDS, H, W, dtype=torch.float64, device="cuda", generator=g)
    band = torch.linspace(0.8, 1.2, BANDS, dtype=torch.float64, device="cuda")[:, None, None]
    return lum * band * (0.75 + 0.5 * noise)


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind}
    if kind == "batch":
        s["renderers"] = []
        for j in range(case["scenes"]):
            own = dict(case, scene=("box", "terrain", "volume")[j % 3], tris=max(1000, case["tris"] >> (j % 4)),
                       width=case["width"] >> (j % 2), height=case["height"] >> (j % 2))
            depth = max(4, case["depth"] - 2 * j)
            s["renderers"].append(_renderer(own, 64 * seed + j, depth=depth))
        s["batch"] = Batch(s["renderers"], kernel=case["kernel"])
        s["batch"].reset(0)
        return s
    s["renderer"] = r = _renderer(case, seed)
    s["first"] = seed % 1000 * BANDS
    if kind == "gradient":
        s["mat"] = autodiff.material_table(r).requires_grad_(True)
        s["eem"] = autodiff.eem_table(r).requires_grad_(True) if case["scene"] == "volume" else None
        g = torch.Generator(device="cuda").manual_seed(seed)
        s["target"] = torch.rand(case["height"], case["width"], 3, dtype=torch.float64, device="cuda", generator=g)
    if kind == "rays":
        s["rays"] = _rays(case, seed)
    if kind == "display":
        r.block_film.copy_(_film(case, seed))
    return s


# ------------------------------------------------------------------------------------------------ one pass
def _view(film, s):
    """A film view together with the state that owns its memory: it is valid while its renderer is."""
    film.owner = s
    return film


def run(s):
    kind = s["kind"]
    if kind == "batch":
        s["batch"].step()
        return [_view(r.mean_film, s) for r in s["renderers"]]
    r = s["renderer"]
    if kind == "pass":
        r.clear_pixel_space()
        r.cast_rays(s["first"] % BANDS, pass_idx=s["first"])
        return _view(r.block_film, s)
    if kind == "block":
        for band in range(BANDS):
            r.cast_rays(band, pass_idx=s["first"] + band)
        r.average_and_reset_block(1)
        return {"film": _view(r.mean_film, s), "rgb": r.color_rays()}
    if kind == "bundle":
        r.cast_rays_bundle(0, BANDS, pass_idx=s["first"])
        r.average_and_reset_block(1)
        return {"film": _view(r.mean_film, s), "xyz": r.resolve_xyz()}
    if kind == "gradient":
        s["mat"].grad = None
        if s["eem"] is not None:
            s["eem"].grad = None
        film = autodiff.render_film(r, s["mat"], s["eem"], first_pass=s["first"], num_blocks=1)
        xyz = autodiff.film_to_xyz(film, r.compiled.cmf, r.cmf_scale)
        loss = ((xyz - s["target"]) ** 2).sum()
        loss.backward()
        return {"film": film.detach(), "loss": loss.detach(), "mat_grad": s["mat"].grad,
                "eem_grad": None if s["eem"] is None else s["eem"].grad}
    if kind == "rays":
        return r.trace(s["rays"])
    r.average_and_reset_block(1)
    return {"film": _view(r.mean_film, s), "m2": _view(r.m2_film, s), "rgb": r.color_rays(), "xyz": r.resolve_xyz()}


# ------------------------------------------------------------------------------------------------ what it cannot do without
VERTICES = {"box": 6.0, "terrain": 2.0, "volume": 14.0}  # mean vertices of a path of the generators' scenes


def _path_work(scene, tris, npix, depth, passes):
    """A path vertex casts an extension and a shadow ray; a ray meets about 4 boxes of each level of a four-child tree
    (12 operations a box) and 4 triangles (45 each); a vertex's events take about 500 operations."""
    paths = npix * passes
    verts = paths * min(VERTICES[scene], depth)
    ray = 4 * 12 * math.log(max(tris, 4), 4) + 4 * 45
    film = 2 * 8 * paths
    return film + 96 * tris, verts * (2 * ray + 500)


def work(case):
    kind = case["kind"]
    if kind == "batch":
        total = np.zeros(2)
        for j in range(case["scenes"]):
            npix = (case["width"] >> (j % 2)) * (case["height"] >> (j % 2))
            total += _path_work(("box", "terrain", "volume")[j % 3], max(1000, case["tris"] >> (j % 4)), npix,
                                max(4, case["depth"] - 2 * j), BANDS)
            total[0] += 5 * 8 * BANDS * npix
        return {"bytes": float(total[0]), "flops": float(total[1])}
    if kind == "rays":
        ray = 4 * 12 * math.log(max(case["tris"], 4), 4) + 4 * 45
        return {"bytes": 40.0 * case["rays"] + 48.0 * case["tris"], "flops": ray * case["rays"]}
    npix = case["width"] * case["height"]
    if kind == "display":
        image = case["image_width"] * case["image_height"]
        return {"bytes": 5.0 * 8 * BANDS * npix + 12.0 * image + 12.0 * npix,
                "flops": 6.0 * BANDS * (npix + image) + 6.0 * BANDS * npix}
    passes = 1 if kind == "pass" else BANDS
    b, f = _path_work(case["scene"], case["tris"], npix, case["depth"], passes)
    if kind == "gradient":  # forward, then each path once more with its derivatives
        return {"bytes": 2.0 * b + 16.0 * BANDS * npix, "flops": 3.0 * f}
    return {"bytes": b + (3.0 if kind == "pass" else 5.0) * 8 * BANDS * npix, "flops": f}


# ------------------------------------------------------------------------------------------------ in 64 bits
def exact(case, seed):
    """The display path's values.  Rendered films have none: a path in 64 bits takes other random branches than one in
    32 bits (the tests hold them to the oracle's streams instead), and the closest hits of a large mesh take too long."""
    if case["kind"] != "display":
        return None
    _, cfg, extras, _ = _scene(case["scene"], case["tris"], seed)
    film = _film(case, seed)
    cmf64 = torch.as_tensor(np.asarray(extras["cmf"], np.float32).astype(np.float64), device="cuda")
    step = (cfg.lambda_max - cfg.lambda_min) / (BANDS - 1)
    scale = step / (float(cmf64[:, 1].sum()) * step)
    xyz = torch.einsum("bhw,bc->hwc", film, cmf64) * scale
    W, H, iw, ih = case["width"], case["height"], case["image_width"], case["image_height"]
    f = np.float32
    ri = (np.arange(iw).astype(f) / f(iw) * f(W)).astype(np.int64)  # the nearest source pixel of each image pixel
    rj = (np.arange(ih).astype(f) / f(ih) * f(H)).astype(np.int64)
    big = xyz[torch.from_numpy(rj).cuda()][:, torch.from_numpy(ri).cuda()]
    m = torch.as_tensor(np.asarray(sb.spectral_data.srgb_xyz_to_rgb(), np.float32).astype(np.float64), device="cuda")
    e = big @ m.reshape(3, 3).T
    return {"film": film, "m2": film * film, "rgb": (e / (e + 1.0)) ** 0.5, "xyz": xyz}
