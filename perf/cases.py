"""What a user has this framework do, as cases whose speed can be followed.

Every case goes through a public entry point: a training iteration, the autograd function on its own, an accumulation
step, the viewer's frames, an evaluation over test cameras, RGB + alpha + depth for one camera, and the neighbour
distances that size the first Gaussians of a cloud.  Scenes are those of ``raygaussx_b200.scenes`` (an object seen from
a hemisphere, an unbounded scene seen from a ring, a stress scene of needles), drawn on the GPU.  With other counts than
the ones those are defined for, the Gaussians grow or shrink with the spacing between them, as they do in a scene that
is being densified.
"""
import math
from types import SimpleNamespace

import torch

from raygaussx_b200 import dist, inference, training
from raygaussx_b200 import render_optix as ro
from raygaussx_b200.scenes import SimpleCamera
from simple_knn._C import distCUDA2

DEVICE = "cuda"

#: Per scene: the count it is defined for, field of view (degrees), march parameters, and per ray of the full-size image
#: the hits, (sample, Gaussian) pairs inside the truncation ellipsoids and slabs with hits, from the work counters.
SCENES = {
    "object": dict(n=300_000, fov=40.0, dt=0.0025, dynamic=False, cap=2048, white=True, eps=1e-3, hits=88.0, pairs=1104.0, slabs=15.4),
    "unbounded": dict(n=3_000_000, fov=60.0, dt=0.005, dynamic=True, cap=512, white=False, eps=1e-3, hits=191.0, pairs=1098.0, slabs=4.2),
    "stress": dict(n=7_000_000, fov=50.0, dt=0.005, dynamic=True, cap=512, white=False, eps=1e-4, hits=159.0, pairs=1562.0, slabs=3.3),
}


def listed():
    return [
        # a small scene and a thumbnail, one optimizer step per view: the overhead of an iteration
        dict(name="iterate-object-4k", kind="iterate", scene="object", n=4096, width=64, height=64, degree=3, lobes=0, views=1),
        # early in a training run, before densification; odd sizes, degree 1, spherical-Gaussian lobes
        dict(name="iterate-unbounded-30k", kind="iterate", scene="unbounded", n=30_011, width=399, height=301, degree=1, lobes=3, views=1),
        # a whole iteration late in a training run on an unbounded scene
        dict(name="iterate-unbounded-3m", kind="iterate", scene="unbounded", n=3_000_000, width=1256, height=828, degree=3, lobes=0, views=1),
        # forward and backward of the autograd function on its own: an object, then degree 2 with seven lobes
        dict(name="view-object-300k", kind="view", scene="object", n=300_000, width=800, height=800, degree=3, lobes=0, views=1),
        dict(name="view-unbounded-1m-lobes", kind="view", scene="unbounded", n=1_000_003, width=628, height=414, degree=2, lobes=7, views=1),
        # gradients of several views accumulated before an optimizer step (late training, multi-GPU training)
        dict(name="window-unbounded-3m", kind="window", scene="unbounded", n=3_000_000, width=1256, height=828, degree=3, lobes=0, views=4),
        # the viewer: one frame of an object; a camera path through a scene of seven million needles
        dict(name="frames-object-300k", kind="frames", scene="object", n=300_000, width=800, height=800, degree=3, lobes=0, views=1),
        dict(name="frames-stress-7m", kind="frames", scene="stress", n=7_000_000, width=1920, height=1080, degree=3, lobes=0, views=3),
        # evaluation over test cameras with 2x2 rays per pixel, images and PSNR on the host
        dict(name="evaluate-object-300k", kind="evaluate", scene="object", n=300_000, width=400, height=400, degree=3, lobes=0, views=6),
        # RGB, alpha and depth of one camera
        dict(name="full-unbounded-1m", kind="full", scene="unbounded", n=1_000_000, width=640, height=360, degree=3, lobes=0, views=1),
        # neighbour distances of an initial cloud: points on surfaces (structure from motion), and a large scene's
        dict(name="knn-surface-100k", kind="knn", scene="surface", n=100_003, width=0, height=0, degree=0, lobes=0, views=0),
        dict(name="knn-unbounded-3m", kind="knn", scene="unbounded", n=3_000_000, width=0, height=0, degree=0, lobes=0, views=0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["iterate"] * 4 + ["view"] * 3 + ["window", "frames", "frames", "evaluate", "full", "knn", "knn"])
    if kind == "knn":
        return dict(kind=kind, scene=rng.choice(["surface", "unbounded", "object"]), n=_log_int(rng, 4096, 3_000_000), width=0,
                    height=0, degree=0, lobes=0, views=0)
    scene = rng.choice(["object", "unbounded"]) if kind != "frames" else rng.choice(["object", "unbounded", "stress"])
    most = {"object": 600_000, "unbounded": 3_000_000, "stress": 7_000_000}[scene]
    pixels = math.exp(rng.uniform(math.log(64 * 64), math.log(800 * 800 if kind != "evaluate" else 400 * 400)))
    aspect = rng.uniform(0.75, 1.8)
    views = {"window": rng.randint(2, 4), "frames": rng.randint(1, 3), "evaluate": rng.randint(2, 6)}.get(kind, 1)
    return dict(kind=kind, scene=scene, n=_log_int(rng, 4096, most), width=max(16, int(math.sqrt(pixels * aspect))),
                height=max(16, int(math.sqrt(pixels / aspect))), degree=rng.choice([0, 1, 2, 3, 3]),
                lobes=0 if kind == "window" else rng.choice([0, 0, 0, 1, 3, 7]), views=views)


# ----------------------------------------------------------------------------- inputs
def _cloud(scene, n, g):
    """Positions and linear scales."""
    randn = lambda *s: torch.randn(*s, generator=g, device=DEVICE)
    rand = lambda *s: torch.rand(*s, generator=g, device=DEVICE)
    if scene == "surface":                      # noisy points on spheres of several sizes
        k = 24
        centres, radii = randn(k, 3) * 2.0, 0.1 + rand(k, 1)
        which = torch.randint(0, k, (n,), generator=g, device=DEVICE)
        d = randn(n, 3)
        return centres[which] + d / d.norm(dim=1, keepdim=True) * radii[which] + 0.002 * randn(n, 3), None
    grow = (SCENES[scene]["n"] / n) ** (1.0 / 3.0)
    if scene == "object":
        return (randn(n, 3) * 0.5).clamp(-1.5, 1.5), torch.exp(randn(n, 3) * 0.5 - 4.5) * grow
    if scene == "unbounded":
        core = rand(n, 1) < 0.8
        d = randn(n, 3)
        shell = d / d.norm(dim=1, keepdim=True) * (rand(n, 1) * 45.0 + 5.0)
        ratio = torch.exp(rand(n, 3) * math.log(10.0))
        shell_scale = torch.exp(randn(n, 1) * 0.5 - 1.0) * ratio.min(dim=1, keepdim=True).values / ratio
        return torch.where(core, randn(n, 3), shell), torch.where(core, torch.exp(randn(n, 3) * 0.6 - 4.0), shell_scale) * grow
    centres = rand(64, 3) * 6 - 3
    which = torch.randint(0, 64, (n,), generator=g, device=DEVICE)
    pos = torch.where(rand(n, 1) < 6.0 / 7.0, rand(n, 3) * 6 - 3, centres[which] + randn(n, 3) * 0.05)
    ratio = torch.exp(rand(n, 3) * math.log(100.0))
    return pos, torch.exp(randn(n, 1) * 0.5 - 5.0) * ratio / ratio.min(dim=1, keepdim=True).values * grow


def _gaussians(case, g):
    """The eight tensors of the operator."""
    n, k, lobes = case["n"], (case["degree"] + 1) ** 2, case["lobes"]
    randn = lambda *s: torch.randn(*s, generator=g, device=DEVICE)
    pos, scales = _cloud(case["scene"], n, g)
    quats = randn(n, 4)
    quats = quats / quats.norm(dim=1, keepdim=True)
    gain, shift = {"object": (20.0, 0.0), "unbounded": (10.0, 0.0), "stress": (30.0, 1.0)}[case["scene"]]
    dens = gain * torch.nn.functional.softplus(randn(n) + shift)
    sh = randn(n, 3, k) * 0.05
    sh[:, :, 0] = randn(n, 3) * 0.2 + 0.5
    feats = randn(n, 3, lobes) * 0.1
    sharp = torch.nn.functional.softplus(randn(n, lobes)) * 4.0 + 0.5
    axis = randn(n, lobes, 3)
    return [pos, scales, quats, dens, sh, feats, sharp, axis / axis.norm(dim=2, keepdim=True)]


def _cameras(case, seed):
    """Cameras of the scene's own arrangement, at places that the seed chooses."""
    w, h = case["width"], case["height"]
    tan = math.tan(math.radians(SCENES[case["scene"]]["fov"]) / 2)
    fovx, fovy = 2 * math.atan(tan), 2 * math.atan(tan * h / w)
    r = torch.rand(max(1, case["views"]), 2, generator=torch.Generator().manual_seed(seed)).tolist()
    cams = []
    for u, v in r:
        a = 2 * math.pi * u
        if case["scene"] == "object":
            s = math.sqrt(max(0.0, 1 - v * v))
            eye = (4 * s * math.cos(a), 4 * s * math.sin(a), 4 * v)
        elif case["scene"] == "unbounded":
            eye = (3 * math.cos(a), 3 * math.sin(a), 0.5)
        else:
            s = math.sqrt(max(0.0, 1 - (2 * v - 1) ** 2))
            eye = (6 * s * math.cos(a), 6 * s * math.sin(a), 6 * (2 * v - 1))
        cams.append(SimpleCamera(eye, fovx=fovx, fovy=fovy, width=w, height=h).to(DEVICE))
    return cams


def _photo(case, g):
    """[3, H, W]: smooth shapes and some noise, in [0, 1]."""
    h, w = case["height"], case["width"]
    coarse = torch.rand(1, 3, max(2, h // 16), max(2, w // 16), generator=g, device=DEVICE)
    img = torch.nn.functional.interpolate(coarse, size=(h, w), mode="bilinear", align_corners=False)[0]
    return (img + 0.03 * torch.randn(3, h, w, generator=g, device=DEVICE)).clamp(0, 1)


def _settings(case, cam, supersampling=(1, 1)):
    m = SCENES[case["scene"]]
    return ro.RenderOptixSettings(None, False, None, None, None, None, None, m["dt"], m["dynamic"], cam, m["cap"], case["lobes"],
                                  supersampling=supersampling, white_background=m["white"], transmittance_eps=m["eps"])


#: Learning rates at the end of their schedules, so that a scene stays what it is however often it is stepped.
LATE_LRS = dict(positions=1.6e-6, scales=5e-5, quaternions=1e-5, densities=5e-4, rgb=2.5e-5, spherical_harmonics=1.25e-6,
                sph_gauss_features=2.5e-5, bandwidth_sharpness=1e-5, lobe_axis=1e-5)


def prepare(case, seed):
    g = torch.Generator(device=DEVICE).manual_seed(seed)
    kind = case["kind"]
    st = SimpleNamespace(case=case, kind=kind)
    if kind == "knn":
        st.points = _cloud(case["scene"], case["n"], g)[0].contiguous()
        return st
    tensors = [t.contiguous() for t in _gaussians(case, g)]
    st.cams = _cameras(case, seed)
    m = SCENES[case["scene"]]
    rays = case["width"] * case["height"]
    if kind == "iterate":
        st.cloud = training.SimplePointCloud(*tensors, lrs=LATE_LRS)
        st.cams[0].original_image = _photo(case, g)
        st.config = training.default_config(dt=m["dt"], dynamic_sampling=m["dynamic"], white_background=m["white"],
                                            max_prim_slice=m["cap"])
        st.schedule = training.AccumulationSchedule()
    elif kind == "view":
        st.leaves = [t.requires_grad_(t.numel() > 0) for t in tensors]
        st.settings = _settings(case, st.cams[0])
        st.dl = torch.sign(torch.randn(rays, 3, generator=g, device=DEVICE)) / (3 * rays)       # of an L1 loss
    elif kind == "window":
        st.tensors = tensors
        st.structs = [ro.camera_struct(c) for c in st.cams]
        st.targets = [torch.rand(rays, 3, generator=g, device=DEVICE) for _ in st.cams]
        st.grads = dist.GradBuffer(case["n"], tensors[4].shape[2], DEVICE)
        st.march_of = lambda cam, rows, flags: ro.Renderer._march(m["dt"], m["dynamic"], m["cap"], m["white"], m["eps"], rows,
                                                                  cam.height, flags)
    elif kind == "full":
        st.tensors = tensors
        st.settings = _settings(case, st.cams[0])
    else:
        st.cloud = training.SimplePointCloud(*tensors)
        for cam in st.cams if kind == "evaluate" else ():
            cam.original_image = _photo(case, g)
    return st


# ----------------------------------------------------------------------------- one pass
def run(st):
    case = st.case
    m = SCENES.get(case["scene"])
    if st.kind == "knn":
        return distCUDA2(st.points)
    if st.kind == "iterate":
        loss, _ = training.training_iteration(st.cloud, st.cams[0], st.config, 0, st.schedule)
        c = st.cloud
        return [loss, c.positions, c.scales, c.quaternions, c.densities, c.rgb, c.spherical_harmonics, c.sph_gauss_features,
                c.bandwidth_sharpness, c.lobe_axis, c.xyz_gradient_accum_norm, c.num_accum, c.num_accum_gnv]
    if st.kind == "view":
        with torch.no_grad():
            st.leaves[3].mul_(1.0)             # an optimizer has written to the parameters since the last view
        rgb = ro.RenderOptixFunction.apply(*st.leaves, st.settings)
        wanted = [t for t in st.leaves if t.requires_grad]
        return [rgb.detach(), *torch.autograd.grad(rgb, wanted, st.dl)]
    if st.kind == "window":
        dist.accumulation_step(ro.get_renderer(DEVICE), st.tensors, st.structs, st.targets, st.march_of, st.grads)
        return st.grads.flat
    if st.kind == "full":
        return ro.render_full(*st.tensors, st.settings)
    if st.kind == "frames":
        return inference.frames(st.cloud, st.cams, m["cap"], m["dt"], m["dynamic"], transmittance_eps=m["eps"])
    psnr, _, images, _ = inference.inference(None, st.cloud, st.cams, m["cap"], m["dt"], 0, (2, 2), m["white"], m["dynamic"])
    return [psnr, images]


# ----------------------------------------------------------------------------- what a pass cannot do without
def work(case):
    n, kind = case["n"], case["kind"]
    if kind == "knn":                           # points in, distances out; each point against the 32 of one leaf
        return {"bytes": 16.0 * n, "flops": 8.0 * 32 * n}
    m = SCENES[case["scene"]]
    per_gaussian = 4.0 * (11 + 3 * (case["degree"] + 1) ** 2 + 7 * case["lobes"])
    pixels = float(case["width"] * case["height"] * case["views"])
    rays = pixels * (4 if kind == "evaluate" else 1)
    # operations per hit, per pair inside and per slab with hits; hits along a ray grow with the cube root of the count
    more = (n / m["n"]) ** (1.0 / 3.0)
    hits, pairs, slabs = rays * m["hits"] * more, rays * m["pairs"] * more, rays * m["slabs"]
    flops = 90 * hits + 12 * pairs + 480 * slabs
    if kind in ("iterate", "view", "window"):
        flops += 290 * hits + 22 * pairs + 640 * slabs
    if kind == "iterate":                       # parameters and the two moments of Adam in and out, statistics, target image
        data = 6 * per_gaussian * n + 24.0 * n + 12 * pixels
    elif kind in ("view", "window"):            # parameters in, gradients out; the loss's gradient or the target in, colours out
        data = 2 * per_gaussian * n + 24 * pixels
    elif kind == "full":
        data = per_gaussian * n + 20 * pixels
    else:
        data = per_gaussian * n + (8 if kind == "frames" else 24) * pixels
    return {"bytes": data, "flops": flops}


def tolerance(case):
    kind = case["kind"]
    if kind == "knn":
        return {"rel": 1e-6, "max": 1e-5}
    if kind in ("iterate", "view", "window"):
        # sums of up to a million fp32 terms per Gaussian, added in no fixed order; single entries in which they cancel
        return {"rel": 1e-4, "max": 2e-2}
    # a few hundred fp32 terms per ray; a sample at the rim of a Gaussian may fall on either side of the cut-off.  Bytes of
    # a frame may differ where a colour lies at the edge between two of them.
    return {"rel": 1e-5, "max": 2e-3, "differ": 2e-3}
