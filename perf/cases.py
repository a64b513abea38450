"""What a user has this renderer do, as cases that can be timed and whose outputs can be compared.

Every case is one call (or one optimisation step) through the public entry points on a seeded
synthetic scene. The scenes are the benchmark configurations' (dtrt_gb300.scenes: a fog sphere, a
cloud in a dielectric cube, a displaced mesh, a free cloud, uneven batch scenes) and the tank scene
of the reference's glass example, over image sides 24 to 512, 1 to 128 samples per pixel, 2 to 16
bounces, 1, 3, 4 and 8 derivative images, meshes of 320 to 20480 triangles and grids of 16^3 to
128^3. Sizes are odd as often as round: crops, previews and pyramid levels are.

A case's seed changes its grid or mesh, its image gradient and its random numbers.
"""
import functools
import math

import numpy as np
import torch

from dtrt_gb300 import dtrt, native, pydtrt, scenes

# ----------------------------------------------------------------------------- the cases


def listed():
    return [
        # a preview while a scene is set up: few samples of a small image, where launches and waits count
        dict(name="forward_preview", kind="forward", scene="sphere", width=48, height=32, spp=4, depth=5, nder=1,
             sppse=4, sppe=16, subdiv=3),
        # forward-mode images of a moving homogeneous sphere: edge, interface and primary-edge terms (C0)
        dict(name="forward_sphere", kind="forward", scene="sphere", width=256, height=256, spp=32, depth=5, nder=1,
             sppse=10, sppe=1024, subdiv=3),
        # material derivatives of a cloud in a glass cube (C1, the headline)
        dict(name="forward_glass_cloud", kind="forward", scene="glass", width=512, height=512, spp=64, depth=10,
             nder=3, sppse=10, sppe=1024, res=64),
        # eight vertex directions of a 20480-triangle mesh: silhouette edges carry the work (C2)
        dict(name="forward_mesh", kind="forward", scene="mesh", width=256, height=256, spp=64, depth=4, nder=8,
             sppse=10, sppe=1024, subdiv=5),
        # eight parameters of a 128^3 cloud, the longest paths (C3)
        dict(name="forward_cloud", kind="forward", scene="cloud", width=512, height=512, spp=128, depth=16, nder=8,
             sppse=10, sppe=1024, res=128),
        # image and gradient of all voxels of that cloud in one replay, dL/dI and results on the device
        dict(name="density_adjoint", kind="density_adjoint", scene="cloud", width=512, height=512, spp=64, depth=16,
             nder=1, sppe=0, res=128),
        # one optimisation step on a smaller cloud: image, L2 loss and backward through torch.autograd
        dict(name="density_step", kind="density_step", scene="cloud", width=200, height=150, spp=16, depth=12, nder=1,
             sppe=0, res=48),
        # image and gradient of all vertex positions of a mesh
        dict(name="vertex_adjoint", kind="vertex_adjoint", scene="mesh", width=256, height=256, spp=16, depth=4,
             nder=1, sppse=10, sppe=256, subdiv=5),
        # a plain image of a cloud, without derivatives
        dict(name="primal_glass_cloud", kind="primal", scene="glass", width=512, height=512, spp=64, depth=10, nder=1,
             res=64),
        # a plain image of a mesh at an odd size
        dict(name="primal_mesh", kind="primal", scene="mesh", width=333, height=217, spp=50, depth=6, nder=1,
             subdiv=5),
        # the reference's own call: description in, scene built, rendered, images back on the host
        dict(name="render_scene", kind="render_scene", width=160, height=120, spp=16, depth=8, sppse=4, sppe=128,
             subdiv=3),
        # a batch of uneven scenes, image and density gradient of each
        dict(name="batch", kind="batch", items=12, side=160, spp=12, depth=8),
    ]


_COST = dict(sphere=1.0, glass=0.35, mesh=1.4, cloud=0.35)


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _image(rng, budget, lo=24, hi=512):
    """Image sides and samples per pixel with at most `budget` camera paths."""
    w, h = _log(rng, lo, hi), _log(rng, lo, hi)
    spp = min(_log(rng, 1, 128), max(1, int(budget / (w * h))))
    return dict(width=w, height=h, spp=spp)


def draw(rng):
    kind = rng.choice(["forward"] * 5 + ["density_adjoint", "density_step", "vertex_adjoint", "primal", "primal",
                                         "render_scene", "batch"])
    if kind == "batch":
        return dict(kind=kind, items=rng.randint(3, 16), side=_log(rng, 40, 200), spp=_log(rng, 2, 24),
                    depth=rng.randint(4, 12))
    if kind == "render_scene":
        return dict(kind=kind, **_image(rng, 1.0e6, hi=256), depth=rng.randint(3, 10), sppse=rng.randint(1, 8),
                    sppe=_log(rng, 16, 256), subdiv=rng.randint(2, 4))
    scene = {"density_adjoint": ["cloud", "glass"], "density_step": ["cloud", "glass"],
             "vertex_adjoint": ["mesh"]}.get(kind, ["sphere", "glass", "mesh", "cloud"])
    c = dict(kind=kind, scene=rng.choice(scene))
    c["nder"] = rng.choice([1, 3, 4, 8]) if kind == "forward" else 1
    if c["nder"] < 3 and c["scene"] == "glass" and kind == "forward":
        c["nder"] = 3  # its three parameters
    heavy = kind in ("forward", "vertex_adjoint")
    c.update(_image(rng, (3.0e6 if heavy else 8.0e6) / _COST[c["scene"]] / (2 if kind == "vertex_adjoint" else 1)))
    c["depth"] = rng.randint(2, 8) if c["scene"] in ("sphere", "mesh") else rng.randint(3, 16)
    if heavy:
        c["sppse"] = rng.randint(1, 10)
    if kind != "primal":
        c["sppe"] = _log(rng, 16, 1024) if heavy else 0
    if c["scene"] in ("sphere", "mesh"):
        c["subdiv"] = rng.randint(2, 5)
    else:
        c["res"] = _log(rng, 16, 128)
    return c


# ----------------------------------------------------------------------------- scenes


@functools.lru_cache(maxsize=8)
def _sphere(subdiv):
    v, f = scenes.icosphere(subdiv, 0.7)
    return v, f, scenes.vertex_normals(v, f)


def _blobs(res, nblobs, rng):
    """The density of scenes.blob_grid from separable factors (quick to make)."""
    x = np.linspace(0.0, 1.0, res)
    c, s, a = rng.uniform(0.2, 0.8, (nblobs, 3)), rng.uniform(0.05, 0.15, nblobs), rng.uniform(0.5, 1.0, nblobs)
    g = np.exp(-(x[None, :, None] - c[:, None, :]) ** 2 / (2 * s[:, None, None] ** 2))  # [blob, x, axis]
    zy = (a[:, None, None] * g[:, :, None, 2] * g[:, None, :, 1]).reshape(nblobs, -1)
    return (zy.T @ g[:, :, 0]).reshape(res, res, res).astype(np.float32)


def _spec(case, rng):
    w, h, nder = case["width"], case["height"], case["nder"]
    if case["scene"] == "sphere":
        spec = scenes.config0(w, h, subdiv=case["subdiv"], nder=nder)
        spec.media[0].sigma_t = float(rng.uniform(0.8, 1.5))
        return spec
    if case["scene"] == "mesh":
        spec = scenes.config2(w, h, subdiv=0, nder=nder)
        v, f, n = _sphere(case["subdiv"])
        s = spec.shapes[0]
        s.vertices = (v + n * rng.normal(0.0, 0.003, (v.shape[0], 1))).astype(np.float32)
        s.indices = f
        d = rng.normal(size=(nder, v.size))
        s.velocities = (d / np.linalg.norm(d, axis=1, keepdims=True)).reshape(-1, 3).astype(np.float32)
        return spec
    if case["scene"] == "glass":
        spec = scenes.config1(w, h, res=2, nder=nder)
        spec.media[0].density = _blobs(case["res"], 8, rng)
        return spec
    spec = scenes.config3(w, h, res=2, nder=nder, param_slots=case["kind"] == "forward", nblobs=1)
    spec.media[0].density = _blobs(case["res"], 32, rng)
    return spec


def _tank(case, rng):
    """The tank of the reference's glass example from pydtrt objects: a Phong body in a
    rough-dielectric tank of fog over a diffuse floor under an area light; three
    translations of the body and the roughness vary. Returns a SceneManager's arguments."""
    v, f, n = _sphere(case["subdiv"])
    v = (0.5 * v + n * rng.normal(0.0, 0.002, (v.shape[0], 1))).astype(np.float32)
    bv, bf = scenes.box((-0.8, -0.7, -0.8), (0.8, 0.7, 0.8))
    gv, gf = scenes.quad((0.0, -1.0, 0.0), 2.0, 2.0, 1.0)
    lv, lf = scenes.quad((0.0, 2.0, 0.0), 0.5, 0.5, -1.0)
    T = lambda a: torch.from_numpy(np.ascontiguousarray(a))
    shapes = [pydtrt.Shape(T(v), T(f), None, None, 0, 0, -1), pydtrt.Shape(T(bv), T(bf), None, None, 1, -1, 0),
              pydtrt.Shape(T(gv), T(gf), None, None, 2, -1, -1), pydtrt.Shape(T(lv), T(lf), None, None, 3, -1, -1)]
    bsdfs = [pydtrt.BSDF_Phong(torch.tensor([0.3, 0.4, 0.2]), torch.tensor([0.3, 0.3, 0.3]), torch.tensor([20.0])),
             pydtrt.BSDF_roughdielectric(torch.tensor([0.05]), torch.tensor([1.33]), torch.tensor([1.0])),
             pydtrt.BSDF_diffuse(torch.tensor([0.5, 0.5, 0.5])), pydtrt.BSDF_diffuse(torch.zeros(3))]
    cam = pydtrt.Camera(torch.tensor([0.0, 0.3, 4.0]), torch.zeros(3), torch.tensor([0.0, 1.0, 0.0]),
                        torch.tensor([45.0]), 0.01, (case["width"], case["height"]))
    media = [pydtrt.Homogeneous(torch.tensor([float(rng.uniform(0.4, 0.8))]), torch.tensor([0.8, 0.8, 0.8]), 0)]
    scene = pydtrt.Scene(cam, shapes, bsdfs, media, [pydtrt.HG(torch.tensor([0.3]))],
                         [pydtrt.AreaLight(3, torch.tensor([10.0, 10.0, 10.0]))])
    R = pydtrt.SceneTransform
    moves = [[R("SHAPE_TRANSLATE", torch.eye(3)[k], 0)] for k in range(3)] + [[R("BSDF_VARY", "roughdielectric", 1, 0.1, 0.0)]]
    return pydtrt.SceneManager(pydtrt.serialize_scene(scene), moves).args


def _uneven(case, seed, rng):
    """The batch's scenes: displaced spheres of 320 to 5120 triangles, half of them in a cloud,
    image sides, samples and depths as uneven as scenes.config4's."""
    shape = np.random.default_rng([7, case["items"], case["side"]])  # sizes belong to the case, not to the seed
    out = []
    for i in range(case["items"]):
        side = int(case["side"] * shape.uniform(0.35, 1.0))
        c = dict(kind="batch", scene="mesh", width=side, height=side, nder=1, subdiv=int(shape.integers(2, 5)))
        spec = _spec(c, rng)
        if i % 2:
            cv, cf = scenes.box((-0.9, -0.9, -0.9), (0.9, 0.9, 0.9))
            from dtrt_gb300 import _abi
            spec.bsdfs.append(scenes.BsdfSpec(_abi.BSDF_NULL))
            spec.shapes.append(scenes.ShapeSpec(cv, cf, bsdf_id=len(spec.bsdfs) - 1, med_int_id=0))
            spec.phases.append(scenes.PhaseSpec(_abi.PHASE_HG, g=0.3))
            spec.media.append(scenes.MediumSpec(
                _abi.MEDIUM_HETEROGENEOUS, phase_id=0, albedo=(0.9,) * 3, density_scale=2.0,
                density=_blobs(int(shape.choice([32, 48, 64])), 8, rng), vol_min=(-0.9,) * 3, vol_max=(0.9,) * 3))
        opts = dict(seed=seed * 64 + i, spp=max(1, int(case["spp"] * shape.uniform(0.3, 1.0))),
                    max_bounces=int(shape.integers(3, case["depth"] + 1)), sppe=0)
        out.append((spec, opts))
    return out


# ----------------------------------------------------------------------------- one pass


def _options(case, seed):
    return native.NativeScene.options(seed=seed, spp=case["spp"], max_bounces=case["depth"], sppe=case.get("sppe", 0),
                                      sppse=case.get("sppse", 0))


def _stream():
    return torch.cuda.current_stream().cuda_stream


def prepare(case, seed):
    rng = np.random.default_rng([seed, 11])
    gen = torch.Generator("cuda").manual_seed(seed)
    kind = case["kind"]
    st = dict(case=case, kind=kind)
    if kind == "render_scene":
        st["args"] = _tank(case, rng)
        st["options"] = dtrt.RenderOptions(seed, case["spp"], case["depth"], case["sppe"], case["sppse"], True)
        st["integrator"] = dtrt.VolPathTracerAD()
        return st
    if kind == "batch":
        items, st["out"] = [], []
        for spec, kw in _uneven(case, seed, rng):
            sc = native.NativeScene(spec)
            n = sc.gradient_sizes()[0]
            dimg = torch.randn((spec.height, spec.width, 3), device="cuda", generator=gen)
            img, grad = torch.zeros_like(dimg), torch.zeros(max(n, 1), device="cuda")
            st["out"] += [img, grad] if n else [img]
            items.append((sc, sc.options(**kw), dimg.data_ptr(), img.data_ptr(), grad.data_ptr() if n else 0))
            st.setdefault("keep", []).append(dimg)
        st["batch"] = native.Batch(items, stream=_stream())
        return st
    spec = _spec(case, rng)
    st["scene"] = native.NativeScene(spec)
    st["options"] = _options(case, seed)
    shape = (case["height"], case["width"], 3)
    if kind == "forward":
        st["out"] = torch.zeros((case["nder"] + 1,) + shape, device="cuda")
    else:
        st["out"] = torch.zeros(shape, device="cuda")
        st["dimg"] = torch.randn(shape, device="cuda", generator=gen)
    voxels, vertices = st["scene"].gradient_sizes()
    if kind == "density_adjoint":
        st["grad"] = torch.zeros(voxels, device="cuda")
    elif kind == "vertex_adjoint":
        st["grad"] = torch.zeros((vertices, 3), device="cuda")
    elif kind == "density_step":
        st["density"] = torch.from_numpy(spec.media[0].density).cuda().requires_grad_()
        st["target"] = torch.rand(shape, device="cuda", generator=gen)
    return st


def run(st):
    kind, sc = st["kind"], st.get("scene")
    if kind == "forward":
        sc.render(out=st["out"].data_ptr(), stream=_stream(), options=st["options"])
        return st["out"]
    if kind == "primal":
        sc.render_primal(out=st["out"].data_ptr(), stream=_stream(), options=st["options"])
        return st["out"]
    if kind == "density_adjoint":
        sc.render_adjoint(st["dimg"].data_ptr(), image=st["out"].data_ptr(), density_grad=st["grad"].data_ptr(),
                          stream=_stream(), device=True, options=st["options"])
        return st["out"], st["grad"]
    if kind == "vertex_adjoint":
        sc.render_vertex_adjoint(st["dimg"].data_ptr(), image=st["out"].data_ptr(), vertex_grad=st["grad"].data_ptr(),
                                 stream=_stream(), device=True, options=st["options"])
        return st["out"], st["grad"]
    if kind == "density_step":
        x = st["density"]
        x.grad = None
        img = pydtrt.DensityRenderFunc.apply(x, sc, 0, st["options"])
        ((img - st["target"]) ** 2).mean().backward()
        return img.detach(), x.grad
    if kind == "render_scene":
        return pydtrt.render_scene(st["integrator"], st["options"], *st["args"])
    st["batch"].launch(stream=_stream())
    return st["out"]


# ----------------------------------------------------------------------------- what a pass cannot do without


def _triangles(case):
    return 20 * 4 ** case["subdiv"] + 4 if "subdiv" in case else 16


def work(case):
    """Bytes: the scene (36 B of vertices and indices per triangle, the grid) and a given image
    gradient read once, each image and gradient written once. Operations: each camera path's
    first ray (one box test of 24 operations per tree level, one triangle test of 45), and for each
    edge sample its two sub-paths' rays; the bounces after them are random and not counted."""
    if case["kind"] == "batch":
        shape = np.random.default_rng([7, case["items"], case["side"]])
        b = f = 0.0
        for i in range(case["items"]):
            side, sub = int(case["side"] * shape.uniform(0.35, 1.0)), int(shape.integers(2, 5))
            res = int(shape.choice([32, 48, 64])) if i % 2 else 0
            spp = max(1, int(case["spp"] * shape.uniform(0.3, 1.0)))
            shape.integers(3, case["depth"] + 1)
            w = work(dict(kind="density_adjoint", width=side, height=side, spp=spp, subdiv=sub))
            b, f = b + w["bytes"] + 8.0 * res ** 3, f + w["flops"]
        return {"bytes": b, "flops": f}
    kind, pix, tri = case["kind"], case["width"] * case["height"], _triangles(case)
    nder = 4 if kind == "render_scene" else case.get("nder", 1)
    voxels = case.get("res", 0) ** 3
    b = 36.0 * tri + 4.0 * voxels + 12.0 * pix * (nder + 1 if kind in ("forward", "render_scene") else 1)
    if kind in ("density_adjoint", "density_step"):
        b += 12.0 * pix + 4.0 * voxels
    if kind == "vertex_adjoint":
        b += 12.0 * pix + 6.0 * tri
    ray = 24.0 * math.log2(tri) + 45.0
    rays = float(pix) * case["spp"]
    if kind in ("forward", "vertex_adjoint", "render_scene") and case.get("scene", "mesh") in ("mesh", "sphere"):
        rays += 2.0 * pix * case["spp"] * case["sppse"]
    return {"bytes": b, "flops": rays * ray}


def exact(case, seed):
    """None: a render is a Monte Carlo estimate whose value is set by its random decisions; there
    is no 64-bit value of the estimate apart from the estimator itself."""
    return None
