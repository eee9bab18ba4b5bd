"""The workloads that a user of the renderer runs, as timed cases.

A case is a dict of plain values; its "kind" says which entry point it goes
through:

  cast     Context.raycast_device / occluded_device on rays that are already on
           the GPU (picking, visibility and ambient-occlusion queries of a host
           application), exact mode
  frame    Context.render_frame: one image of one resident scene, with the
           preset's post passes, read back as the call does
  batch    Context.render_batch: many small views over a resident scene set
  adjoint  Context.forward + Context.backward: one step of inverse rendering
  post     bc_post_process_noalloc on device images (real-time loop)
  build    bc_build_sah: the BVH of a new mesh, host arrays in and out

Scenes: "soup" (seeded random triangles in the unit cube), "field" (a grid of
displaced geodesic spheres over a ground quad with emissive quads, half of the
spheres rough metal), "beads" (a grid of a few hundred analytic spheres on a
ground sphere), and the built-in "cornell", "room" and "showcase".
"""
import ctypes as C
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "beamcast-gx-v1.0-beta-_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import bcgx  # noqa: E402
from bcgx import scenes  # noqa: E402
from bcgx.scene import MAT_DIFFUSE, MAT_EMISSIVE, MAT_METAL, Material  # noqa: E402
from bcgx.settings import Camera, quality  # noqa: E402

DEV = "cuda"


def listed():
    return [
        # a cursor pick or a few probe rays: the launches are the cost
        dict(name="pick", kind="cast", scene="soup", prims=20_000, rays=1_000, pattern="random", query="closest"),
        # one visibility image (pixel-ordered camera rays) over analytic spheres
        dict(name="beads_visibility", kind="cast", scene="beads", prims=822, rays=200_003, pattern="camera",
             query="closest"),
        # the ray-cast benchmark's sizes: incoherent rays, a scene larger than any cache level but L2
        dict(name="cast_large", kind="cast", scene="soup", prims=1_000_000, rays=4_194_304, pattern="random",
             query="closest"),
        # ambient occlusion baked on a mesh: short hemisphere rays, any hit, a ragged count
        dict(name="occlusion_bake", kind="cast", scene="field", prims=200_000, rays=1_048_583, pattern="hemisphere",
             query="any"),
        # the Cornell-box workload: a frame of under a millisecond, post passes off
        dict(name="cornell_frame", kind="frame", scene="cornell", prims=36, width=320, height=240, spp=16, bounces=5,
             preset="Draft", integrator="path", post=False, guides=False, adaptive=False, photons=0),
        # the Preview preset as it comes: sphere lights, adaptive stop, denoise, bloom, guides
        dict(name="preview_frame", kind="frame", scene="room", prims=9, width=960, height=540, spp=8, bounces=6,
             preset="Preview", integrator="path", post=True, guides=True, adaptive=True, photons=0),
        # the Ultra-shaped frame (2560 x 1440, 16 bounces, 2M triangles) at a quarter of its samples
        dict(name="ultra_frame", kind="frame", scene="field", prims=2_048_000, width=2560, height=1440, spp=64,
             bounces=16, preset="Ultra Realism", integrator="path", post=True, guides=False, adaptive=False,
             photons=0),
        # photon mapping at the Balanced preset's size
        dict(name="photon_frame", kind="frame", scene="room", prims=9, width=1280, height=720, spp=16, bounces=8,
             preset="Balanced", integrator="photon", post=False, guides=False, adaptive=False, photons=3),
        # dataset generation: views of many sizes over four scenes in one call
        dict(name="batch_views", kind="batch", views=16, side=960, spp_lo=4, spp_hi=32, bounces=8, prims=500_000),
        # one iteration of material recovery: 256 albedos, 8 emitters
        dict(name="adjoint_step", kind="adjoint", prims=200_000, width=512, height=512, spp=64, bounces=8, slots=256),
        # one 720p frame of a real-time loop: denoise, bloom, tone map
        dict(name="post_720p", kind="post", width=1280, height=720, denoise=True, taa=1, bloom=1, hdr=3),
        # a million-triangle mesh arrives: build its tree
        dict(name="build_1m", kind="build", prims=1_000_000, bins=32, leaf=4),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["cast", "cast", "cast", "frame", "frame", "frame", "batch", "adjoint", "post", "build"])
    if kind == "cast":
        scene = rng.choice(["soup", "soup", "field", "beads"])
        query = rng.choice(["closest", "closest", "any"])
        prims = _log(rng, 100, 2_000) if scene == "beads" else _log(rng, 1_000, 1_000_000)
        rays = _log(rng, 200, 1_000_000 if scene == "beads" else 4_000_000)
        patterns = ["random", "camera"] if scene != "field" else ["camera", "hemisphere"]
        return dict(kind=kind, scene=scene, prims=prims, rays=rays, pattern=rng.choice(patterns), query=query)
    if kind == "frame":
        scene = rng.choice(["cornell", "room", "showcase", "field"])
        post = rng.random() < 0.5
        integrator = rng.choice(["path", "path", "path", "recursive", "photon"])
        if scene in ("cornell", "field"):
            integrator = "path"
        return dict(kind=kind, scene=scene, prims=_log(rng, 5_000, 500_000) if scene == "field" else 9,
                    width=_log(rng, 120, 1920), height=_log(rng, 90, 1080), spp=_log(rng, 1, 32),
                    bounces=rng.randint(2, 16), preset=rng.choice(["Draft", "Preview", "Ultra Realism"]),
                    integrator=integrator, post=post, guides=rng.random() < 0.3, adaptive=rng.random() < 0.3,
                    photons=rng.randint(1, 4) if integrator == "photon" else 0)
    if kind == "batch":
        return dict(kind=kind, views=rng.randint(2, 24), side=_log(rng, 200, 960), spp_lo=rng.randint(1, 4),
                    spp_hi=rng.randint(5, 32), bounces=rng.randint(2, 12), prims=_log(rng, 20_000, 500_000))
    if kind == "adjoint":
        return dict(kind=kind, prims=_log(rng, 5_000, 200_000), width=_log(rng, 64, 512), height=_log(rng, 64, 512),
                    spp=_log(rng, 4, 64), bounces=rng.randint(2, 8), slots=_log(rng, 4, 256))
    if kind == "post":
        w = _log(rng, 64, 1280)
        return dict(kind=kind, width=w, height=_log(rng, 64, 720), denoise=rng.random() < 0.8, taa=rng.randint(0, 3),
                    bloom=rng.randint(0, 3), hdr=rng.randint(0, 3))
    return dict(kind=kind, prims=_log(rng, 1_000, 1_000_000), bins=rng.choice([16, 32]), leaf=rng.choice([2, 4, 8]))


# ---- scenes ---------------------------------------------------------------------
def _field_side(prims):
    return max(2, int(round(math.sqrt(prims / 500.0))))


def _field(prims, seed):
    """n x n displaced geodesic spheres of 500 triangles, spacing 1, radius 0.4."""
    n = _field_side(prims)
    rng = np.random.default_rng(seed)
    base = scenes.geodesic_sphere(5)
    uniq, inv = np.unique(np.round(base.reshape(-1, 3), 12), axis=0, return_inverse=True)
    inv = inv.reshape(-1)
    sp = scenes.SceneSpec(name="field", bvh_mode="SAH", bvh_bins=32, bvh_leaf=4)
    ground = sp.material(Material(MAT_DIFFUSE, (0.45, 0.45, 0.45)))
    ext = float(n)
    sp.triangles(scenes.quad((-1, 0, -1), (-1, 0, ext + 1), (ext + 1, 0, ext + 1), (ext + 1, 0, -1)), ground)
    mats = np.empty(n * n, np.int32)
    for k in range(n * n):
        if rng.random() < 0.5:
            mats[k] = sp.material(Material(MAT_DIFFUSE, tuple(rng.uniform(0.2, 0.8, 3))))
        else:
            mats[k] = sp.material(Material(MAT_METAL, tuple(rng.uniform(0.5, 0.95, 3)),
                                           roughness=float(rng.uniform(0.05, 1.0))))
    k = np.arange(n * n)
    center = np.stack([k % n + 0.5, np.full(n * n, 0.45), k // n + 0.5], axis=1)
    disp = np.zeros((n * n, len(uniq)))
    for _ in range(4):
        wave = rng.normal(size=(n * n, 3)) * 3.0
        disp += np.sin(wave @ uniq.T + rng.uniform(0, 2 * np.pi, (n * n, 1)))
    verts = center[:, None, :] + uniq[None] * (0.4 + 0.0125 * disp)[:, :, None]
    sp.triangles(verts[:, inv].reshape(-1, 9), np.repeat(mats, len(base)))
    for _ in range(n):
        lum = rng.lognormal(1.0, 1.0)
        e = sp.material(Material(MAT_EMISSIVE, emission=tuple(rng.uniform(0.6, 1.0, 3) * lum)))
        x, z = rng.uniform(0, ext, 2)
        s, y = rng.uniform(0.5, 1.5), rng.uniform(2.5, 4.0)
        sp.triangles(scenes.quad((x, y, z), (x + s, y, z), (x + s, y, z + s), (x, y, z + s)), e)
    a = rng.uniform(-0.1, 0.1, 2) * ext
    cam = Camera((ext * 0.5 + a[0], ext * 0.35 + 1.0, -ext * 0.25 + a[1]), (ext * 0.5, 0.0, ext * 0.45), (0, 1, 0),
                 50.0)
    return sp, cam


def _beads(prims, seed):
    """A grid of spheres on a ground sphere, jittered, with one light."""
    rng = np.random.default_rng(seed)
    sp = scenes.SceneSpec(name="beads", bvh_mode="SAH", bvh_bins=16, bvh_leaf=4)
    ground = sp.material(Material(MAT_DIFFUSE, (.45, .48, .52)))
    blue = sp.material(Material(MAT_METAL, (.25, .52, .92), roughness=.12))
    light = sp.material(Material(MAT_EMISSIVE, emission=(25, 22, 18)))
    sp.sphere((0, -1001, -10), 1000, ground)
    cols = max(1, int(round(math.sqrt(2.0 * max(1, prims - 2)))))
    for k in range(max(1, prims - 2)):
        x, z = k % cols - cols / 2, k // cols
        j = rng.uniform(-0.1, 0.1, 3)
        sp.sphere((x * .58 + j[0], -.65 + j[1], -3 - z * .58 + j[2]), .22, blue)
    sp.sphere((0, 8, -8), 1.2, light)
    return sp, Camera((9, 5, 8), (0, -.5, -8), (0, 1, 0), 42.0)


def _soup(prims, seed):
    sp = scenes.random_triangles(prims, seed)
    az = np.random.default_rng(seed + 7).uniform(0, 2 * np.pi)
    return sp, Camera((0.5 + 2 * math.cos(az), 0.9, 0.5 + 2 * math.sin(az)), (0.5, 0.5, 0.5), (0, 1, 0), 45.0)


def _scene(name, prims, seed):
    if name == "soup":
        return _soup(prims, seed)
    if name == "field":
        return _field(prims, seed)
    if name == "beads":
        return _beads(prims, seed)
    if name == "cornell":
        sp, cam, _ = scenes.cornell_box(seed)
        return sp, cam
    sp, cam = scenes.cornell_reference_scene() if name == "room" else scenes.showcase_scene()
    d = np.random.default_rng(seed).uniform(-0.3, 0.3, 3)
    cam.position = tuple(float(p + q) for p, q in zip(cam.position, d))
    return sp, cam


def _resident(spec):
    """A context with the scene built and uploaded, as an application holds it."""
    ctx = bcgx.Context(0)
    sc = scenes.to_scene(spec, build=False)
    if spec.n_triangles() > 10_000:
        sc.build_device(ctx)
    else:
        sc.build()
    ctx.upload(sc)
    return ctx, sc


# ---- rays -----------------------------------------------------------------------
def _unit(v):
    return v / v.norm(dim=1, keepdim=True).clamp_min(1e-20)


def _rays(case, spec, cam, seed):
    """(n, 8) float32 on the GPU: origin, tmin, direction, tmax."""
    n = case["rays"]
    g = torch.Generator(device=DEV).manual_seed(seed)
    r = torch.empty((n, 8), dtype=torch.float32, device=DEV)
    r[:, 3] = 1e-4
    r[:, 7] = 1e30
    if case["pattern"] == "random":
        lo, hi = (0.0, 1.0) if case["scene"] == "soup" else (-8.0, 8.0)
        r[:, 0:3] = torch.rand((n, 3), generator=g, device=DEV) * (hi - lo) + lo
        r[:, 4:7] = _unit(torch.randn((n, 3), generator=g, device=DEV))
    elif case["pattern"] == "camera":
        w = max(1, int(math.sqrt(n * 1.5)))
        h = (n + w - 1) // w
        i = torch.arange(n, device=DEV)
        jit = torch.rand((n, 2), generator=g, device=DEV)
        u = ((i % w) + jit[:, 0]) / w - 0.5
        v = 0.5 - ((i // w) + jit[:, 1]) / h
        p, t = torch.tensor(cam.position, device=DEV), torch.tensor(cam.target, device=DEV)
        fwd = _unit((t - p).float()[None])[0]
        right = _unit(torch.linalg.cross(fwd, torch.tensor([0.0, 1.0, 0.0], device=DEV))[None])[0]
        up = torch.linalg.cross(right, fwd)
        s = 2 * math.tan(math.radians(cam.fov) / 2)
        r[:, 0:3] = p.float()
        r[:, 4:7] = _unit(fwd + (u * s * w / h)[:, None] * right + (v * s)[:, None] * up)
    else:  # hemisphere rays off the triangles
        tri = torch.from_numpy(np.concatenate(spec.tri_verts)).to(DEV).float()
        k = torch.randint(0, len(tri), (n,), generator=g, device=DEV)
        k = k.sort().values  # a bake walks its texels in surface order
        a, b, c = tri[k, 0:3], tri[k, 3:6], tri[k, 6:9]
        q = torch.rand((n, 2), generator=g, device=DEV)
        q = torch.where((q.sum(1, keepdim=True) > 1), 1 - q, q)
        nrm = _unit(torch.linalg.cross(b - a, c - a))
        d = _unit(torch.randn((n, 3), generator=g, device=DEV))
        d = torch.where((d * nrm).sum(1, keepdim=True) < 0, -d, d)
        r[:, 0:3] = a + q[:, :1] * (b - a) + q[:, 1:] * (c - a) + nrm * 1e-3
        r[:, 4:7] = d
        r[:, 7] = torch.rand((n,), generator=g, device=DEV) * 0.9 + 0.1
    return r


# ---- prepare --------------------------------------------------------------------
def _settings(case, seed):
    st = quality(case["preset"])
    st.width, st.height, st.spp, st.bounces = case["width"], case["height"], case["spp"], case["bounces"]
    st.msaa, st.tsaa = 1, 0
    st.adaptive_sampling = case["adaptive"]
    if not case["post"]:
        st.denoise, st.bloom = False, 0
    st.integrator = {"path": bcgx.INTEGRATOR_PATH, "recursive": bcgx.INTEGRATOR_RECURSIVE,
                     "photon": bcgx.INTEGRATOR_PHOTON}[case["integrator"]]
    st.photon_mapping = case["photons"]
    st.seed = seed
    return st


def _post_images(case, seed):
    """A noisy HDR image and its first-hit guides: shaded patches, planes in depth, some sky."""
    W, H = case["width"], case["height"]
    g = torch.Generator(device=DEV).manual_seed(seed)

    def smooth(ch, cells):
        x = torch.rand((1, ch, cells, cells), generator=g, device=DEV)
        return torch.nn.functional.interpolate(x, size=(H, W), mode="bilinear", align_corners=True)[0]

    def patches(ch, cells):
        x = torch.rand((1, ch, cells, cells), generator=g, device=DEV)
        return torch.nn.functional.interpolate(x, size=(H, W), mode="nearest")[0]

    shade = smooth(3, 9) * patches(3, 13) * 2.0
    noise = -torch.log(torch.rand((3, H, W), generator=g, device=DEV).clamp_min(1e-6))
    bright = (torch.rand((1, H, W), generator=g, device=DEV) < 0.01).float() * 6.0
    img = (shade * (0.6 + 0.4 * noise) + bright).permute(1, 2, 0).contiguous()
    nrm = patches(3, 13) - 0.5 + 0.1 * (smooth(3, 17) - 0.5)
    nrm = nrm / nrm.norm(dim=0, keepdim=True).clamp_min(1e-6)
    depth = 1.0 + 8.0 * patches(1, 13) + smooth(1, 5)
    depth = torch.where(patches(1, 7) < 0.08, torch.full_like(depth, -1.0), depth)
    guide = torch.cat([nrm, depth]).permute(1, 2, 0).contiguous()
    return img, guide


def _batch_views(case, seed):
    """Views of log-uniform sizes, 128 x 128 up to side x 9/16 side, over scenes 0..3 in turn:
    sizes and samples belong to the case, cameras and sample streams to the seed."""
    shape, rng = np.random.default_rng(case["views"] * 10_000 + case["side"]), np.random.default_rng(seed)
    side = max(128, case["side"])
    views = []
    for v in range(case["views"]):
        t = shape.uniform()
        st = quality("Draft")
        st.width, st.height = (int(round(128 * (m / 128) ** t)) for m in (side, max(128, side * 9 // 16)))
        st.spp, st.bounces = int(shape.integers(case["spp_lo"], case["spp_hi"] + 1)), case["bounces"]
        st.msaa, st.tsaa = 1, 0
        st.firefly_clamp, st.rr_depth, st.adaptive_sampling = 0.0, 4, False
        st.denoise, st.bloom = False, 0
        st.seed = seed + v
        az, el, dist = rng.uniform(0, 2 * np.pi), rng.uniform(0.1, 0.6), rng.uniform(1.8, 2.6)
        pos = [0.5 + dist * math.cos(el) * math.cos(az), 0.5 + dist * math.sin(el),
               0.5 + dist * math.cos(el) * math.sin(az)]
        views.append((v % 4, Camera(tuple(pos), (0.5, 0.5, 0.5), (0, 1, 0), 45.0), st))
    return views


def prepare(case, seed):
    kind = case["kind"]
    if kind == "cast":
        spec, cam = _scene(case["scene"], case["prims"], seed)
        ctx, sc = _resident(spec)
        n = case["rays"]
        rays = _rays(case, spec, cam, seed)
        s = dict(kind=kind, query=case["query"], ctx=ctx, scene=sc, n=n, rays=rays, stream=torch.cuda.Stream())
        if case["query"] == "any":
            s["hit"] = torch.zeros(n, dtype=torch.uint8, device=DEV)
        else:
            s["t"] = torch.zeros(n, dtype=torch.float32, device=DEV)
            s["prim"] = torch.zeros(n, dtype=torch.int32, device=DEV)
        return s
    if kind == "frame":
        spec, cam = _scene(case["scene"], case["prims"], seed)
        ctx, sc = _resident(spec)
        return dict(kind=kind, ctx=ctx, scene=sc, cam=cam, st=_settings(case, seed), guides=case["guides"])
    if kind == "batch":
        sizes = [max(1_000, int(case["prims"] * f)) for f in (0.02, 0.1, 0.4, 1.0)]
        specs = [scenes.batch_scene(n, seed + 1 + k) for k, n in enumerate(sizes)]
        views = _batch_views(case, seed)
        ctx = bcgx.Context(0)
        scs = [scenes.to_scene(sp, build=False) for sp in specs]
        for sc in scs:
            sc.build_device(ctx)
        ctx.upload_set(scs)
        return dict(kind=kind, ctx=ctx, scenes=scs, views=views)
    if kind == "adjoint":
        pb = scenes.diff_scene(seed=seed, n_tris=case["prims"], n_slots=case["slots"], width=case["width"],
                               height=case["height"], spp=case["spp"], bounces=case["bounces"])
        ctx, sc = _resident(pb.spec)
        ctx.diff_configure(pb.cam, pb.settings, pb.albedo_materials, pb.emission_materials)
        target, _ = ctx.forward(pb.true_params, seed + 1, want_loss=False)
        ctx.diff_set_target(target)
        return dict(kind=kind, ctx=ctx, scene=sc, params=pb.init_params, seed=seed + 2)
    if kind == "post":
        img, guide = _post_images(case, seed)
        st = quality("Ultra Realism")
        st.denoise, st.taa, st.txaa, st.bloom, st.hdr = case["denoise"], case["taa"], 0, case["bloom"], case["hdr"]
        return dict(kind=kind, W=case["width"], H=case["height"], st=st.c(), img=img, guide=guide,
                    out=torch.zeros_like(img), rgba=torch.zeros(img.shape[:2], dtype=torch.int32, device=DEV))
    v = scenes.random_triangle_verts(case["prims"], seed).reshape(-1, 3, 3)
    box = np.concatenate([v.min(axis=1) - 1e-6, v.max(axis=1) + 1e-6], axis=1)  # the builder's padded boxes
    cent = ((v[:, 0] + v[:, 1]) + v[:, 2]) * (1.0 / 3.0)
    n = len(v)
    cap = 2 * n - 1
    return dict(kind=kind, ctx=bcgx.Context(0), n=n, bins=case["bins"], leaf=case["leaf"],
                box=np.ascontiguousarray(box), cent=np.ascontiguousarray(cent),
                out=[np.zeros((cap, 6)), np.zeros(cap, np.int32), np.zeros(cap, np.int32), np.zeros(cap, np.int32),
                     np.zeros(cap, np.int32), np.zeros(n, np.int32)])


# ---- run ------------------------------------------------------------------------
def _p(a, t):
    return a.ctypes.data_as(C.POINTER(t))


def run(s):
    kind = s["kind"]
    if kind == "cast":
        if s["query"] == "any":
            s["ctx"].occluded_device(s["rays"].data_ptr(), s["n"], s["hit"].data_ptr(), s["stream"].cuda_stream)
            return s["hit"]
        s["ctx"].raycast_device(s["rays"].data_ptr(), s["n"], s["t"].data_ptr(), s["prim"].data_ptr(),
                                s["stream"].cuda_stream)
        return {"t": s["t"], "prim": s["prim"]}
    if kind == "frame":
        return s["ctx"].render_frame(s["cam"], s["st"], want_guides=s["guides"])
    if kind == "batch":
        images, rays = s["ctx"].render_batch(s["views"])
        return {"images": images, "rays": rays}
    if kind == "adjoint":
        image, loss = s["ctx"].forward(s["params"], s["seed"])
        d_albedo, d_emission = s["ctx"].backward()
        return {"image": image, "loss": loss, "d_albedo": d_albedo, "d_emission": d_emission}
    if kind == "post":
        rc = bcgx.lib().bc_post_process_noalloc(s["W"], s["H"], s["img"].data_ptr(), s["guide"].data_ptr(),
                                                C.byref(s["st"]), s["out"].data_ptr(), s["rgba"].data_ptr(), None)
        if rc:
            raise RuntimeError("bc_post_process_noalloc: status %d" % rc)
        return {"linear": s["out"], "rgba": s["rgba"]}
    nn = C.c_int32(0)
    box, left, right, start, count, order = s["out"]
    rc = bcgx.lib().bc_build_sah(s["ctx"].handle, s["n"], _p(s["box"], C.c_double), _p(s["cent"], C.c_double),
                                 s["bins"], s["leaf"], C.byref(nn), _p(box, C.c_double), _p(left, C.c_int32),
                                 _p(right, C.c_int32), _p(start, C.c_int32), _p(count, C.c_int32),
                                 _p(order, C.c_int32))
    if rc:
        raise RuntimeError("bc_build_sah: status %d" % rc)
    return {"nodes": nn.value, "box": box, "left": left, "right": right, "start": start, "count": count,
            "order": order}


# ---- work -----------------------------------------------------------------------
# A query on a tree of N primitives tests about 3.3 log2 N boxes (18 operations)
# and 8 primitives (45 operations): the counts that the CPU renderer makes on a
# binary tree (70 and 8 on the 2M-triangle field).
def _query_flops(prims):
    return 18 * 3.3 * math.log2(max(2, prims)) + 45 * 8


def _scene_bytes(prims):
    return 64.0 * prims + 40.0 * prims


def work(case):
    kind = case["kind"]
    if kind == "cast":
        out = 1 if case["query"] == "any" else 8
        return {"bytes": case["rays"] * (32.0 + out) + _scene_bytes(case["prims"]),
                "flops": case["rays"] * _query_flops(case["prims"])}
    if kind == "frame":
        px = case["width"] * case["height"]
        paths = px * case["spp"]
        per = min(case["bounces"], 5)
        out = 16 + (12 if case["guides"] else 0)
        return {"bytes": px * float(out) + _scene_bytes(case["prims"]),
                "flops": paths * per * (_query_flops(case["prims"]) + 150.0)}
    if kind == "batch":
        px = case["views"] * case["side"] * case["side"] * 9 / 16 / 4
        paths = px * (case["spp_lo"] + case["spp_hi"]) / 2
        return {"bytes": px * 12.0 + 1.5 * _scene_bytes(case["prims"]),
                "flops": paths * 1.3 * (_query_flops(case["prims"]) + 150.0)}
    if kind == "adjoint":
        px = case["width"] * case["height"]
        return {"bytes": px * 24.0 + 2 * _scene_bytes(case["prims"]),
                "flops": 2.0 * px * case["spp"] * min(case["bounces"], 2) * (_query_flops(case["prims"]) + 200.0)}
    if kind == "post":
        px = case["width"] * case["height"]
        passes = 2 + min(3, case["taa"]) if case["denoise"] else 0
        return {"bytes": px * (12.0 + (16.0 if passes else 0.0) + 16.0),
                "flops": px * (passes * 9 * 50.0 + case["bloom"] * 30.0 + 60.0)}
    n = case["prims"]
    return {"bytes": n * (72.0 + 2 * 64.0 + 4.0), "flops": n * math.log2(max(2, n)) * 40.0}


# ---- exact ----------------------------------------------------------------------
def _exact_cast(case, seed):
    """Nearest distance of every ray by testing every primitive in 64 bits."""
    spec, cam = _scene(case["scene"], case["prims"], seed)
    r = _rays(case, spec, cam, seed).double()
    n = len(r)
    o, tmin, d, tmax = r[:, 0:3], r[:, 3:4], r[:, 4:7], r[:, 7:8]
    best = torch.full((n,), math.inf, dtype=torch.float64, device=DEV)
    if spec.spheres:
        c = torch.tensor([s[0] for s in spec.spheres], dtype=torch.float64, device=DEV)
        rad = torch.tensor([s[1] for s in spec.spheres], dtype=torch.float64, device=DEV)
        step = max(1, 40_000_000 // len(c))
        for a in range(0, n, step):
            oo, dd, lo, hi = o[a:a + step], d[a:a + step], tmin[a:a + step], tmax[a:a + step]
            oc = oo[:, None, :] - c[None]
            dl2 = (dd * dd).sum(1, keepdim=True)
            hb = (oc * dd[:, None, :]).sum(2)
            disc = hb * hb - dl2 * ((oc * oc).sum(2) - rad * rad)
            sq = disc.clamp_min(0).sqrt()
            for root in ((-hb + sq) / dl2, (-hb - sq) / dl2):
                ok = (disc >= 0) & (root >= lo) & (root <= hi)
                best[a:a + step] = torch.minimum(best[a:a + step], torch.where(ok, root, math.inf).min(1).values)
    if spec.tri_verts:
        v = torch.from_numpy(np.concatenate(spec.tri_verts)).to(DEV)
        step = max(1, 20_000_000 // len(v))
        p0, e1, e2 = v[:, 0:3], v[:, 3:6] - v[:, 0:3], v[:, 6:9] - v[:, 0:3]

        def dot(a, b):
            return a[0] * b[0] + a[1] * b[1] + a[2] * b[2]

        def cross(a, b):
            return (a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0])

        p0, e1, e2 = ([x[None, :, k] for k in range(3)] for x in (p0, e1, e2))
        for a in range(0, n, step):
            dd = [d[a:a + step, k, None] for k in range(3)]
            s = [o[a:a + step, k, None] - p0[k] for k in range(3)]
            h = cross(dd, e2)
            det = dot(e1, h)
            u = dot(s, h) / det
            q = cross(s, e1)
            w = dot(dd, q) / det
            t = dot(e2, q) / det
            ok = (det.abs() >= 1e-10) & (u >= 0) & (w >= 0) & (u + w <= 1) & (t >= tmin[a:a + step]) & (
                t <= tmax[a:a + step])
            best[a:a + step] = torch.minimum(best[a:a + step], torch.where(ok, t, math.inf).min(1).values)
    return torch.where(torch.isinf(best), -1.0, best)


def _exact_post(case, seed):
    """The denoise and bloom passes in 64 bits."""
    img, guide = _post_images(case, seed)
    x, gd = img.double(), guide.double()
    H, W = x.shape[:2]
    lum = torch.tensor([0.2126, 0.7152, 0.0722], dtype=torch.float64, device=DEV)

    def span(k, size):
        """Target and source ranges of a shift by k along an axis."""
        return (slice(max(0, -k), min(size, size - k)), slice(max(0, k), min(size, size + k)))

    passes = 2 + min(3, case["taa"]) if case["denoise"] else 0
    for it in range(passes):
        step = 1 << it
        num, den = torch.zeros_like(x), torch.zeros((H, W), dtype=torch.float64, device=DEV)
        for oy in (-1, 0, 1):
            for ox in (-1, 0, 1):
                if abs(oy) * step >= H or abs(ox) * step >= W:
                    continue
                (ty, sy), (tx, sx) = span(oy * step, H), span(ox * step, W)
                g0, g1, c0, c1 = gd[ty, tx], gd[sy, sx], x[ty, tx], x[sy, sx]
                v0, v1 = g0[..., 3] >= 0, g1[..., 3] >= 0
                w = torch.exp(-((c0 @ lum) - (c1 @ lum)).abs() * 3.5)
                nd = (g0[..., :3] * g1[..., :3]).sum(-1).clamp(-1, 1)
                scale = (0.04 * g0[..., 3].clamp_min(1.0)).clamp_min(0.15)
                geo = torch.exp((nd - 1) * 48) * torch.exp(-(g0[..., 3] - g1[..., 3]).abs() / scale)
                w = w * torch.where(v0, geo, torch.ones_like(geo)) * (v0 == v1)
                if oy == 0 and ox == 0:
                    w = w * 1.5
                num[ty, tx] += c1 * w[..., None]
                den[ty, tx] += w
        x = torch.where((den > 1e-12)[..., None], num / den.clamp_min(1e-300)[..., None], x)
    if case["bloom"] > 0:
        radius, thr, strength = 1 + case["bloom"], 1.25 - 0.2 * case["bloom"], 0.08 + 0.09 * case["bloom"]
        l = (x @ lum)[..., None]
        b = torch.where(l > thr, x * (l - thr) / l.clamp_min(1e-6), torch.zeros_like(x))
        for axis in (1, 0):
            size = b.shape[axis]
            acc, cnt = torch.zeros_like(b), torch.zeros_like(b)
            for k in range(-radius, radius + 1):
                if abs(k) >= size:
                    continue
                t, s = span(k, size)
                at = (slice(None), t) if axis == 1 else (t,)
                src = (slice(None), s) if axis == 1 else (s,)
                acc[at] += b[src]
                cnt[at] += 1
            b = acc / cnt
        x = x + b * strength
    return x


def exact(case, seed):
    """In 64 bits, where plain arithmetic gives it: the distances of a ray cast
    (every primitive tested) and the post passes. Path-traced images have none
    but a second renderer."""
    if case["kind"] == "cast" and case["query"] == "closest" and case["rays"] * case["prims"] <= 2e10:
        return {"t": _exact_cast(case, seed), "prim": None}
    if case["kind"] == "post":
        return {"linear": _exact_post(case, seed), "rgba": None}
    return None
