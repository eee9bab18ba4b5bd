"""Batched multi-view rendering (bc_scene_set_upload + bc_render_batch).

Every (pixel, sample) path draws from its own seeded stream and each pixel
adds its samples in sample order, so a view rendered inside a batch must be
bit-identical to the same view rendered alone, whatever the other views, the
wave capacity or the launch form (captured graph or plain stream launches).
The single-view renderer is checked against the fp64 oracle in
test_render_gpu.py; these tests tie the batch engine to it exactly.
"""
import numpy as np
import pytest

import bcgx
from bcgx import scenes

pytestmark = pytest.mark.gpu


def _settings(W, H, spp, bounces, seed, sampler="Halton", power=True, clamp=0.0):
    st = bcgx.quality("Draft")
    st.width, st.height, st.spp, st.bounces = W, H, spp, bounces
    st.msaa, st.tsaa = 1, 0
    st.sampler, st.mis, st.power_light_sampling = sampler, True, power
    st.firefly_clamp, st.rr_depth, st.adaptive_sampling = clamp, 3, False
    st.denoise, st.bloom = False, 0
    st.seed = seed
    return st


def _scene_mix():
    """Three scenes with different material tables and lights: sphere lights
    (NEE, power-weighted light choice) in two of them, so light, material and
    primitive offsets of the set are all exercised."""
    a, cam_a = scenes.cornell_reference_scene()
    b, cam_b, _ = scenes.cornell_box()
    c, cam_c = scenes.showcase_scene()
    return [a, b, c], [cam_a, cam_b, cam_c]


def _alone(ctx, spec, cam, st):
    ctx.upload(scenes.to_scene(spec))
    return ctx.render_frame(cam, st, want_guides=False, want_rgba=False)


def test_batch_equals_single_views(gpu_ctx):
    specs, cams = _scene_mix()
    built = [scenes.to_scene(s) for s in specs]
    views = [
        (0, cams[0], _settings(96, 64, 8, 6, 11)),
        (1, cams[1], _settings(80, 60, 12, 5, 12, sampler="R2")),
        (2, cams[2], _settings(120, 72, 5, 7, 13, sampler="Random", power=False, clamp=9.0)),
        (0, cams[0], _settings(33, 17, 3, 2, 14)),
        (2, cams[2], _settings(64, 64, 16, 4, 15)),
    ]
    alone = []
    for k, cam, st in views:
        gpu_ctx.upload(built[k])
        r = gpu_ctx.render_frame(cam, st, want_guides=False, want_rgba=False)
        alone.append((r["linear"], r["rays"]))
    gpu_ctx.upload_set(built)
    outs, rays = gpu_ctx.render_batch(views)
    for v, (o, (ref, _)) in enumerate(zip(outs, alone)):
        assert o.shape == ref.shape
        assert np.array_equal(o, ref), f"view {v}: batch differs from the view rendered alone"
    assert rays == sum(r for _, r in alone)


@pytest.mark.parametrize("cap,graph", [(4096, 1), (4096, 0), (50_000, 1)])
def test_batch_independent_of_wave_split(gpu_ctx, cap, graph):
    specs, cams = _scene_mix()
    built = [scenes.to_scene(s) for s in specs]
    views = [(k % 3, cams[k % 3], _settings(40 + 8 * k, 30 + 4 * k, 4 + k, 5, 100 + k)) for k in range(7)]
    gpu_ctx.upload_set(built)
    ref, rays_ref = gpu_ctx.render_batch(views)
    old_cap, old_graph = gpu_ctx.get_option("render_wave_cap"), gpu_ctx.get_option("render_graph")
    try:
        gpu_ctx.set_option("render_wave_cap", cap)
        gpu_ctx.set_option("render_graph", graph)
        outs, rays = gpu_ctx.render_batch(views)
    finally:
        gpu_ctx.set_option("render_wave_cap", old_cap)
        gpu_ctx.set_option("render_graph", old_graph)
    assert rays == rays_ref
    for v in range(len(views)):
        assert np.array_equal(outs[v], ref[v]), f"view {v} depends on the wave split"


def test_wave_graph_reuse_across_batch_shapes(gpu_ctx):
    """A captured wave is replayed by later calls: calls that differ in view
    count, sample-table size and frame size must still match plain launches."""
    specs, cams = _scene_mix()
    gpu_ctx.upload_set([scenes.to_scene(s) for s in specs])
    calls = [
        [(k % 3, cams[k % 3], _settings(48 + 4 * k, 40, 6 + 2 * k, 5, 300 + k)) for k in range(6)],
        [(1, cams[1], _settings(90, 70, 9, 5, 400))],
        [(2, cams[2], _settings(64, 48, 17, 5, 401)), (0, cams[0], _settings(30, 20, 2, 5, 402))],
        [(0, cams[0], _settings(100, 80, 5, 5, 403, sampler="Random"))],
    ]
    old_cap, old_graph = gpu_ctx.get_option("render_wave_cap"), gpu_ctx.get_option("render_graph")
    try:
        gpu_ctx.set_option("render_wave_cap", 4096)
        got = []
        gpu_ctx.set_option("render_graph", 1)
        for views in calls:
            got.append(gpu_ctx.render_batch(views))
        gpu_ctx.set_option("render_graph", 0)
        for c, views in enumerate(calls):
            ref, rays = gpu_ctx.render_batch(views)
            assert got[c][1] == rays, f"call {c}: ray count differs under graph replay"
            for v in range(len(views)):
                assert np.array_equal(got[c][0][v], ref[v]), f"call {c} view {v} differs under graph replay"
    finally:
        gpu_ctx.set_option("render_wave_cap", old_cap)
        gpu_ctx.set_option("render_graph", old_graph)


def test_single_frame_independent_of_wave_split(gpu_ctx):
    spec, cam, st = scenes.cornell_box()
    st = st.copy()
    st.width, st.height, st.spp = 160, 120, 24
    st.denoise, st.bloom = False, 0
    gpu_ctx.upload(scenes.to_scene(spec))
    ref = gpu_ctx.render_frame(cam, st, want_guides=False, want_rgba=False)
    old = gpu_ctx.get_option("render_wave_cap")
    try:
        gpu_ctx.set_option("render_wave_cap", 7000)  # not a multiple of the frame: waves split samples
        out = gpu_ctx.render_frame(cam, st, want_guides=False, want_rgba=False)
    finally:
        gpu_ctx.set_option("render_wave_cap", old)
    assert np.array_equal(out["linear"], ref["linear"])
    assert out["rays"] == ref["rays"]


def test_batch_small_workload_matches_single(gpu_ctx):
    """A scaled-down batching workload (4 scenes, 8 views) through both forms."""
    specs, views = scenes.batch_views(n_views=8, sizes=(2000, 4000, 8000, 16000), max_side=(192, 108),
                                      spp_range=(2, 6))
    built = [scenes.to_scene(s) for s in specs]
    gpu_ctx.upload_set(built)
    batch, rays_b = gpu_ctx.render_batch(views)
    plain_rays = 0
    for v, view in enumerate(views):
        out, r = gpu_ctx.render_batch([view])
        plain_rays += r
        assert np.array_equal(out[0], batch[v])
    assert plain_rays == rays_b
    for o in batch:
        assert np.isfinite(o).all() and o.mean() > 0


def test_batch_argument_errors(gpu_ctx):
    specs, cams = _scene_mix()
    gpu_ctx.upload_set([scenes.to_scene(s) for s in specs[:2]])
    with pytest.raises(bcgx.BCError, match="INVALID_ARG"):
        gpu_ctx.render_batch([(2, cams[0], _settings(16, 16, 1, 1, 1))])
    with pytest.raises(bcgx.BCError, match="INVALID_ARG"):
        gpu_ctx.render_batch([(0, cams[0], _settings(0, 16, 1, 1, 1))])
    with pytest.raises(bcgx.BCError, match="INVALID_ARG"):
        gpu_ctx.set_option("render_wave_cap", 100)
    # single-view calls see scene 0 of the set
    st = _settings(48, 32, 4, 3, 5)
    a = gpu_ctx.render_frame(cams[0], st, want_guides=False, want_rgba=False)["linear"]
    b, _ = gpu_ctx.render_batch([(0, cams[0], st)])
    assert np.array_equal(a, b[0])


def _soup(n_tris, n_spheres, seed):
    r = np.random.default_rng(seed)
    sp = scenes.SceneSpec(name="soup")
    mats = [sp.material(bcgx.Material(kind=k, color=(0.8, 0.7, 0.6), roughness=0.1, ior=1.5)) for k in (0, 1, 2)]
    light = sp.material(bcgx.Material(kind=3, emission=(6.0, 5.0, 4.0)))
    if n_tris:
        c = r.random((n_tris, 1, 3))
        v = c + (r.random((n_tris, 3, 3)) - 0.5) * 1.5
        v[::3, :, 1] = np.round(v[::3, :, 1])  # axis-aligned ones: boxes without thickness
        sp.triangles(v.reshape(n_tris, 9), r.integers(0, 3, n_tris))
    for i in range(n_spheres):
        sp.sphere(r.random(3), 0.25, light if i == 0 else mats[i % 3])
    return sp


@pytest.mark.parametrize("n_tris,n_spheres", [(1, 0), (2, 1), (0, 24), (23, 1), (24, 0), (25, 0), (12, 13)])
def test_unwalked_scenes_match_the_walk(gpu_ctx, n_tris, n_spheres):
    """A scene of at most 24 primitives resident alone is rendered without its tree; in a
    set of two it is walked. Same images, bit for bit."""
    sc = scenes.to_scene(_soup(n_tris, n_spheres, 7 * n_tris + n_spheres))
    cams = [bcgx.Camera((0.5, 0.5, 2.8), (0.5, 0.5, 0.5), (0, 1, 0), 50.0),
            bcgx.Camera((0.4, 0.6, 0.5), (0.9, 0.1, 0.2), (0, 1, 0), 90.0)]
    views = [(0, cams[k], _settings(160, 120, 16, 8, 50 + k)) for k in range(2)]
    gpu_ctx.upload_set([sc, sc], set_id=900 + n_tris, revision=1)
    walked, rays_walked = gpu_ctx.render_batch(views)
    gpu_ctx.upload(sc)
    flat, rays_flat = gpu_ctx.render_batch(views)
    assert rays_flat == rays_walked
    for a, b in zip(flat, walked):
        assert np.array_equal(a, b)


def test_unwalked_scene_needs_a_sound_tree(gpu_ctx):
    """A tree that leaves a primitive outside its boxes is walked, as the caller built it,
    also when a geometry update brings such boxes, and no longer when one mends them."""
    sc = scenes.to_scene(_soup(9, 0, 3))
    views = [(0, bcgx.Camera((0.5, 0.5, 2.8), (0.5, 0.5, 0.5), (0, 1, 0), 50.0), _settings(96, 64, 4, 4, 5))]
    good = sc.arrays()
    boxes = good.node_box.copy()
    leaf = int(np.flatnonzero(good.node_count)[0])

    def shrink(a, on):
        a.node_box[:] = boxes
        if on:
            a.node_box.reshape(-1, 6)[leaf, 3:] = a.node_box.reshape(-1, 6)[leaf, :3] + 1e-3

    gpu_ctx.upload(good, scene_id=77, topology_rev=1, geometry_rev=1)
    want, _ = gpu_ctx.render_batch(views)
    shrink(good, True)
    gpu_ctx.upload_set([good, good], set_id=78, revision=1)
    cut, _ = gpu_ctx.render_batch(views)
    assert not np.array_equal(cut[0], want[0])
    gpu_ctx.upload(good, scene_id=79, topology_rev=1, geometry_rev=1)
    assert np.array_equal(gpu_ctx.render_batch(views)[0][0], cut[0])
    shrink(good, False)
    gpu_ctx.upload(good, scene_id=80, topology_rev=1, geometry_rev=1)
    for rev, on in ((2, True), (3, False)):  # updates of the resident scene's geometry
        shrink(good, on)
        gpu_ctx.upload(good, scene_id=80, topology_rev=1, geometry_rev=rev)
        assert np.array_equal(gpu_ctx.render_batch(views)[0][0], cut[0] if on else want[0])


@pytest.mark.parametrize("spheres", [False, True])
@pytest.mark.parametrize("up_along_edge", [False, True])
def test_unwalked_scene_matches_the_walk_at_the_rim_of_a_wide_view(gpu_ctx, spheres, up_along_edge):
    """The edge where two least faces of the scene's boxes meet, seen from outside, forty
    tangent units off the view axis: a camera's rays there are forty units long. The walk
    loses some of the hits within 1e-5 of such an edge, whatever the rays' length."""
    sp = scenes.SceneSpec(name="edge")
    m = sp.material(bcgx.Material(kind=0, color=(0.8, 0.7, 0.6)))
    light = sp.material(bcgx.Material(kind=3, emission=(5.0, 4.0, 3.0)))
    sp.triangles(scenes.quad((0, 0, 0), (0, 1, 0), (0, 1, 1), (0, 0, 1)), m if spheres else light)
    sp.triangles(scenes.quad((1, 0, 0), (1, 1, 0), (1, 1, 1), (1, 0, 1)), m)
    for k in range(4 if spheres else 0):
        sp.sphere((0.1, 0.1, 0.1 + 0.25 * k), 0.1, light)
    sc = scenes.to_scene(sp)
    eye, side, off = np.array([-0.5, 0.2, 0.5]), np.array([0.0, 0.0, 1.0]), 40.0
    d = np.array([0.0, 0.0, 0.5]) - eye
    d /= np.linalg.norm(d)
    n = np.cross(d, side)
    axis = (d + off * n) / np.hypot(1.0, off)
    cam = bcgx.Camera(tuple(eye), tuple(eye + axis), tuple(side if up_along_edge else n),
                      float(2 * np.degrees(np.arctan(1.02 * off + 0.1))))
    views = [(0, cam, _settings(1280, 720, 128, 2, 7))]
    gpu_ctx.upload_set([sc, sc], set_id=950 + 2 * spheres + up_along_edge, revision=1)
    walked, rays_walked = gpu_ctx.render_batch(views)
    gpu_ctx.upload(sc)
    flat, rays_flat = gpu_ctx.render_batch(views)
    assert rays_flat == rays_walked and np.array_equal(flat[0], walked[0])
